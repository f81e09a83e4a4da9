"""Performance cases of the CKKS evaluation core, through its Python binding.

Every case is a call (or the few calls) a program makes on ciphertexts it holds on the GPU,
with its context created and autotuned and its keys uploaded once.  Keys, plaintext diagonals
and ciphertexts are uniform residues, which is how RLWE keys and ciphertexts are distributed.
Results are residues, compared exactly; the slot encoder and decoder compute in FP64.
"""
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "fideslib-fork_b200"))
import fides_b200 as F  # noqa: E402
from fides_b200 import params  # noqa: E402

_contexts, _keys, _boots = {}, {}, {}


def listed():
    return [
        # the smallest call: one rotation on the small ring (multiplicative depth 5) after some
        # levels are used up; launches and host time decide
        dict(name="rotate_n8192_l3", op="rotate", logN=13, nq=6, bits=50, dnum=2, K=0, level=3, rotation=1),
        # one product in a shallow program (N = 2^14, depth 11) midway through its levels
        dict(name="hmult_n16384_l9", op="hmult", logN=14, nq=12, bits=50, dnum=3, K=0, level=9, rescale=True),
        # an ordinary rotation on the middle ring, by an odd step
        dict(name="rotate_n32768_l13", op="rotate", logN=15, nq=18, bits=50, dnum=3, K=0, level=13, rotation=-5),
        # one product at the top level of the large ring: what an interactive program waits for
        dict(name="hmult_n65536_l30", op="hmult", logN=16, nq=30, bits=50, dnum=3, K=4, level=30, rescale=True),
        # 16 rotations of one ciphertext that share their ModUp (matrix-vector products)
        dict(name="hoisted16_n65536_l29", op="hoisted", logN=16, nq=30, bits=50, dnum=3, K=4, level=29, count=16),
        # throughput: 8 products and 8 rotations at the top level in one batch
        dict(name="mixed8_n65536_l30", op="mixed", logN=16, nq=30, bits=50, dnum=3, K=4,
             products="30,30,30,30,30,30,30,30", rotations="30,30,30,30,30,30,30,30"),
        # a server's batch: requests that happen to be waiting, at levels 5 to 30
        dict(name="served_n65536", op="mixed", logN=16, nq=30, bits=50, dnum=3, K=4, products="28,17,9,22,6",
             rotations="30,13,5,24"),
        # forward and inverse transforms of whole polynomials under 60-bit primes (import and
        # export of coefficient-form data)
        dict(name="ntt_n65536_60bit", op="ntt", logN=16, nq=36, bits=60, dnum=1, K=-1, level=36, count=4),
        # weighted sum of ciphertexts with plaintext weights, integer constants and a rescale (one
        # layer of a linear model)
        dict(name="weighted_n32768_l17", op="weighted", logN=15, nq=18, bits=50, dnum=3, K=0, level=17, terms=11),
        # a 16-diagonal linear transform, 4 baby x 4 giant steps, on a chain of 59-bit primes
        dict(name="lintrans_n65536_l15_59bit", op="lintrans", logN=16, nq=24, bits=59, dnum=3, K=0, level=15, baby=4,
             giant=4),
        # a client's side: encode a batch of full-slot vectors, decode another
        dict(name="encdec_n65536_l24", op="encdec", logN=16, nq=24, bits=50, dnum=3, K=0, level=24, count=32),
        # the largest: one bootstrap of 2^15 slots, with sparse-secret encapsulation
        dict(name="bootstrap_n65536", op="bootstrap", logN=16, nq=24, bits=50, dnum=3, K=0, count=1),
    ]


def draw(rng):
    op = rng.choices(["rotate", "hmult", "hoisted", "mixed", "ntt", "weighted", "lintrans", "encdec", "bootstrap"],
                     [3, 3, 2, 3, 2, 2, 2, 2, 1])[0]
    logN = rng.choice([12, 13, 14, 15, 16, 16])
    low, high = {12: (2, 4), 13: (3, 8), 14: (6, 14), 15: (10, 20), 16: (18, 32)}[logN]
    c = dict(op=op, logN=logN, nq=rng.randint(low, high), bits=rng.choice([50, 50, 59]), dnum=rng.randint(2, 3), K=0)
    c["dnum"] = min(c["dnum"], c["nq"])
    top, half = c["nq"], 1 << (logN - 1)
    step = lambda: rng.choice([1, -1]) * min(half - 1, int(2 ** rng.uniform(0, logN - 1)))  # noqa: E731
    if op == "rotate":
        c.update(level=rng.randint(1, top), rotation=step())
    elif op == "hmult":
        c.update(level=rng.randint(2, top), rescale=rng.random() < 0.75)
    elif op == "hoisted":
        c.update(level=rng.randint(1, top), count=rng.randint(2, 16))
    elif op == "mixed":
        some = lambda: ",".join(str(rng.randint(2, top)) for _ in range(rng.randint(1, 8)))  # noqa: E731
        c.update(products=some(), rotations=some())
    elif op == "ntt":
        c.update(level=rng.randint(1, top), count=max(1, int(2 ** rng.uniform(0, 4.5))), K=-1, dnum=1)
    elif op == "weighted":
        c.update(level=rng.randint(2, top), terms=rng.randint(2, 16))
    elif op == "lintrans":
        c.update(level=rng.randint(2, top), baby=rng.randint(2, 8), giant=rng.randint(1, 4))
    elif op == "encdec":
        c.update(level=rng.randint(1, top), count=max(1, int(2 ** rng.uniform(0, 5))))
    else:  # a bootstrap needs the levels of the listed chain; smaller rings run it too
        c.update(logN=rng.randint(12, 15), nq=rng.randint(23, 25), bits=50, dnum=3, count=rng.randint(1, 4))
    return c


# ---- what a program keeps: the context, its keys, plaintext weights, the bootstrapper

def _context(case):
    at = tuple(case[k] for k in ("logN", "nq", "bits", "dnum", "K"))
    if at not in _contexts:
        logN, nq, bits, dnum, K = at
        if K < 0:  # transforms only: distinct primes of one size, no special primes
            ctx = F.Context(logN, params.gen_primes(logN, bits, nq), [], dnum)
        else:
            p = params.chain(logN, 60, bits, nq, dnum, K=K or None)
            ctx = F.Context(p.logN, p.q, p.p, p.dnum)
        ctx.autotune()
        _contexts[at] = ctx
    return _contexts[at]


def _uniform(ctx, primes, lead, gen):
    """[*lead, len(primes), N] residues, uniform modulo each prime."""
    q = torch.tensor(primes, dtype=torch.int64, device="cuda").view(-1, 1)
    x = torch.empty(*lead, len(primes), ctx.N, dtype=torch.int64, device="cuda")
    return x.random_(0, (1 << 63) - 1, generator=gen).remainder_(q).view(torch.uint64)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _key(ctx, which):
    if (ctx, which) not in _keys:
        _keys[ctx, which] = _uniform(ctx, ctx.q + ctx.p, (2, ctx.dnum), _generator(1000 + which % 100003))
    return _keys[ctx, which]


def _rotation_key(ctx, rotation):
    return _key(ctx, 10 + rotation % (ctx.N // 2))


def _ciphertext(ctx, level, gen):
    return F.Ciphertext(_uniform(ctx, ctx.q[:level], (), gen), _uniform(ctx, ctx.q[:level], (), gen))


def _weights(ctx, level, count):
    at = (ctx, "plain", level, count)
    if at not in _keys:
        _keys[at] = list(_uniform(ctx, ctx.q[:level], (count,), _generator(77)))
    return _keys[at]


def _bootstrapper(case):
    ctx = _context(case)
    if ctx not in _boots:
        top = 2.0 ** case["bits"]
        boot = F.NativeBootstrapper(ctx, top_level=ctx.n_q, top_scale=top, msg_scale=top, K=12, prescale_bits=5,
                                    encapsulation=True)
        boot.set_keys(_key(ctx, 0), _key(ctx, 1), _key(ctx, 2), _key(ctx, 3))
        for r in boot.rotations():
            boot.set_rotation_key(r, _rotation_key(ctx, r))
        boot.prepare()
        _boots[ctx] = boot
    return _boots[ctx]


# ---- the hoisted rotations of a matrix-vector product: +-1, +-2, +-4, ...
def _hoisted_steps(ctx, count):
    return [(1 - 2 * (i & 1)) * (1 << (i // 2)) % (ctx.N // 2) for i in range(count)]


def _levels(text):
    return [int(v) for v in text.split(",")]


def _slots(case, count, gen):
    z = torch.rand(count, 1 << (case["logN"] - 1), 2, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    return torch.view_as_complex(z)


SCALE = 2.0 ** 45


def prepare(case, seed):
    gen = _generator(seed)
    s = dict(case=dict(case), ctx=_context(case))
    ctx, op = s["ctx"], case["op"]
    if op == "rotate":
        s.update(ct=_ciphertext(ctx, case["level"], gen), key=_rotation_key(ctx, case["rotation"]))
    elif op == "hmult":
        s.update(a=_ciphertext(ctx, case["level"], gen), b=_ciphertext(ctx, case["level"], gen), key=_key(ctx, 0))
    elif op == "hoisted":
        steps = _hoisted_steps(ctx, case["count"])
        s.update(ct=_ciphertext(ctx, case["level"], gen), steps=steps, keys=[_rotation_key(ctx, r) for r in steps])
    elif op == "mixed":
        s.update(pairs=[(_ciphertext(ctx, l, gen), _ciphertext(ctx, l, gen)) for l in _levels(case["products"])],
                 jobs=[(_ciphertext(ctx, l, gen), _rotation_key(ctx, 1), 1) for l in _levels(case["rotations"])],
                 key=_key(ctx, 0))
    elif op == "ntt":
        s.update(x=_uniform(ctx, ctx.q[:case["level"]], (case["count"],), gen),
                 y=_uniform(ctx, ctx.q[:case["level"]], (case["count"],), gen))
    elif op == "weighted":
        s.update(cts=[_ciphertext(ctx, case["level"], gen) for _ in range(case["terms"])],
                 weights=_weights(ctx, case["level"], case["terms"]),
                 constants=[(-1) ** t * (3 * t + 1) << 20 for t in range(case["terms"])])
    elif op == "lintrans":
        nb, ng = case["baby"], case["giant"]
        d = _weights(ctx, case["level"], nb * ng)
        s.update(ct=_ciphertext(ctx, case["level"], gen), diagonals=[d[i * nb:(i + 1) * nb] for i in range(ng)],
                 steps=list(range(1, nb)), keys=[_rotation_key(ctx, r) for r in range(1, nb)],
                 giant_key=_rotation_key(ctx, nb))
    elif op == "encdec":
        s.update(slots=_slots(case, case["count"], gen),
                 pts=ctx.encode(_slots(case, case["count"], gen), SCALE, case["level"]))
    else:
        s.update(boot=_bootstrapper(case), cts=[_ciphertext(ctx, 1, gen) for _ in range(case["count"])])
    return s


def _whole(ct):
    """A ciphertext's residues as 64-bit integers torch can compare."""
    return [ct.c0.view(torch.int64), ct.c1.view(torch.int64)]


def run(s):
    case, ctx = s["case"], s["ctx"]
    op = case["op"]
    if op == "rotate":
        return _whole(ctx.rotate(s["ct"], s["key"], case["rotation"]))
    if op == "hmult":
        return _whole(ctx.mult(s["a"], s["b"], s["key"], rescale=case["rescale"]))
    if op == "hoisted":
        return [_whole(o) for o in ctx.rotate_hoisted(s["ct"], s["keys"], s["steps"])]
    if op == "mixed":
        products, rotated = ctx.mixed_batch(s["pairs"], s["key"], s["jobs"])
        return [_whole(o) for o in products + rotated]
    if op == "ntt":  # in place: polynomials to transform, others to bring back
        return [ctx.ntt(s["x"]).view(torch.int64), ctx.intt(s["y"]).view(torch.int64)]
    if op == "weighted":
        x = ctx.dot_plain(s["cts"], s["weights"])
        y = ctx.lincomb(s["cts"], s["constants"])
        total = F.Ciphertext(ctx.add_poly(x.c0, y.c0), ctx.add_poly(x.c1, y.c1))
        return _whole(ctx.rescale(total))
    if op == "lintrans":
        babies = [s["ct"]] + ctx.rotate_hoisted(s["ct"], s["keys"], s["steps"])
        sums = ctx.dot_plain_bsgs(babies, s["diagonals"], case["level"])
        acc = sums[-1]
        for part in reversed(sums[:-1]):
            acc = ctx.rotate(acc, s["giant_key"], case["baby"])
            acc = F.Ciphertext(ctx.add_poly(acc.c0, part.c0), ctx.add_poly(acc.c1, part.c1))
        return _whole(ctx.rescale(acc))
    if op == "encdec":
        return [ctx.encode(s["slots"], SCALE, case["level"]).view(torch.int64), ctx.decode(s["pts"], SCALE)]
    if case["count"] == 1:
        return _whole(s["boot"].bootstrap(s["cts"][0]))
    return [_whole(o) for o in s["boot"].bootstrap_batch(s["cts"])]


# ---- compulsory work: bytes of the operands, keys and results, each once; flops as two per
# modular multiplication (a butterfly is one, an inner-product term is one)

def _transforms(case, limbs):
    return limbs * (case["logN"] << (case["logN"] - 1))


def _special(case):
    if case["K"]:
        return max(case["K"], 0)
    bits = [60] + [case["bits"]] * (case["nq"] - 1)
    return params.special_count(bits, case["dnum"], 61)


def _switch(case, level, outs=2):
    """Modular multiplications of one key switch at `level` (ModUp, inner product, ModDown)."""
    N, K, alpha = 1 << case["logN"], _special(case), -(-case["nq"] // case["dnum"])
    beta = -(-level // alpha)
    up, down = level + beta * (level + K) - level, outs * (K + level)
    convert = level * (level + K) + outs * K * level
    return _transforms(case, level + up + down) + N * (convert + 2 * beta * (level + K))


def _key_limbs(case, level):
    alpha = -(-case["nq"] // case["dnum"])
    return 2 * -(-level // alpha) * (level + _special(case))


def work(case):
    op, N = case["op"], 1 << case["logN"]
    l = case.get("level", 0)
    if op == "rotate":
        limbs, mults = 4 * l + _key_limbs(case, l), _switch(case, l)
    elif op == "hmult":
        limbs = 4 * l + 2 * (l - case["rescale"]) + _key_limbs(case, l)
        mults = _switch(case, l) + 4 * N * l
    elif op == "hoisted":
        n = case["count"]
        limbs, mults = 2 * l + n * (2 * l + _key_limbs(case, l)), n * _switch(case, l)
        alpha = -(-case["nq"] // case["dnum"])
        beta = -(-l // alpha)
        mults -= (n - 1) * (_transforms(case, l + beta * (l + _special(case)) - l) + N * l * (l + _special(case)))
    elif op == "mixed":
        hm, ro = _levels(case["products"]), _levels(case["rotations"])
        limbs = sum(6 * v - 2 for v in hm) + sum(4 * v for v in ro) + _key_limbs(case, max(hm)) + \
            _key_limbs(case, max(ro))
        mults = sum(_switch(case, v) + 4 * N * v for v in hm) + sum(_switch(case, v) for v in ro)
    elif op == "ntt":
        limbs, mults = 4 * case["count"] * l, 2 * _transforms(case, case["count"] * l)
    elif op == "weighted":
        t = case["terms"]
        limbs, mults = 3 * t * l + 2 * (l - 1), 4 * t * N * l + _transforms(case, 2 * l)
    elif op == "lintrans":
        nb, ng = case["baby"], case["giant"]
        limbs = 4 * l - 2 + nb * ng * l + nb * _key_limbs(case, l)
        mults = (nb + ng - 2) * _switch(case, l) + 2 * nb * ng * N * l + _transforms(case, 2 * l)
    elif op == "encdec":
        limbs, mults = case["count"] * (l + 1 + 1 + 1), _transforms(case, case["count"] * (l + 3))
    else:
        # keys and diagonals of the linear transforms (about 38 rotations and 6 x 64 diagonals), each
        # read once; about 14000 limb transforms for each ciphertext
        limbs = 38 * _key_limbs(case, case["nq"]) + 6 * 50 * (case["nq"] + _special(case))
        mults = case["count"] * _transforms(case, 14000)
    return {"bytes": 8.0 * N * limbs, "flops": 2.0 * mults}


def tolerance(case):
    if case["op"] == "encdec":
        # residues of rounded coefficients: another order of the FP64 sums may move a rounding tie
        # by one, in every limb (1.1e-4 of the coefficients against an FFT of another order); slots: FP64
        # sums over log N stages (1e-15, largest 3.6e-15)
        return {"rel": 4e-15, "max": 1.5e-14, "differ": 4.3e-4}
    return "exact"


def exact(case, seed):
    """Slots are decoded from plaintexts encoded at a scale whose rounding is far below the slots
    (about 2e-12), so the decoder's exact answer is the slots; residues have no such value."""
    if case["op"] != "encdec":
        return None
    gen = _generator(seed)
    _slots(case, case["count"], gen)
    return [None, _slots(case, case["count"], gen)]
