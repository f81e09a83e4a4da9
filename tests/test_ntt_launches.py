"""GPU tests of how limb lists become NTT launches: small rings on both sides of the 32-limb rule (8 or 16
residues per thread), and lists with more runs (limbs that do not follow one another) than a launch holds."""
import numpy as np
import pytest

import oracle as O
from ckks_host import KeyGen, uniform_limbs, xrng

pytestmark = pytest.mark.gpu


def eq(gpu_t, host):
    import fides_b200 as F
    return np.array_equal(F.to_host(gpu_t), host)


@pytest.mark.parametrize("logN", [12, 13, 14])
@pytest.mark.parametrize("limbs", [1, 32, 33])
def test_small_rings(fides, logN, limbs):
    q = O.gen_primes(logN, 60, 1) + O.gen_primes(logN, 50, 2) + O.gen_primes(logN, 59, 1)
    o, ctx = O.Oracle(logN, q, [], 1), fides.Context(logN, q, [], 1)
    ids = [i % 4 for i in range(limbs)]
    x = uniform_limbs(xrng(logN + limbs), [q[i] for i in ids], o.N)
    d = fides.to_device(x)
    ctx.ntt_limbs([d[i] for i in range(limbs)], ids)
    assert eq(d, o.ntt(x, ids))
    ctx.ntt_limbs([d[i] for i in range(limbs)], ids, inverse=True)
    assert eq(d, x)


@pytest.mark.parametrize("order", ["reversed", "every second", "one prime"])
def test_more_runs_than_a_launch_holds(fides, order):
    logN, n = 12, 230
    q = O.gen_primes(logN, 60, 1) + O.gen_primes(logN, 50, 3)
    o, ctx = O.Oracle(logN, q, [], 1), fides.Context(logN, q, [], 1)
    at = {"reversed": range(n - 1, -1, -1), "every second": range(0, 2 * n, 2), "one prime": range(n)}[order]
    ids = [2] * n if order == "one prime" else [i % 4 for i in range(n)]
    d = fides.to_device(np.zeros((2 * n, o.N), dtype=np.uint64))
    x = uniform_limbs(xrng(7), [q[i] for i in ids], o.N)
    rows = [d[k] for k in at]
    for r, v in zip(rows, x):
        r.copy_(fides.to_device(v))
    ctx.ntt_limbs(rows, ids)
    want = o.ntt(x, ids)
    assert all(eq(r, w) for r, w in zip(rows, want))
    assert not fides.to_host(d)[[k for k in range(2 * n) if k not in set(at)]].any()


@pytest.mark.parametrize("logN,bits", [(13, 50), (14, 59)])
def test_small_ring_products_alone_and_in_a_batch(fides, logN, bits):
    """Products and rotations of a batch (launches beyond 32 limbs) equal the oracle, as single calls do."""
    from fides_b200 import params
    prm = params.chain(logN, 60, bits, 7, 3)
    o, ctx = O.Oracle(logN, prm.q, prm.p, 3), fides.Context(logN, prm.q, prm.p, 3)
    kg = KeyGen(o)
    rk, rot = kg.relin_key(), kg.rotation_key(3)
    rk_d, rot_d = fides.to_device(rk), fides.to_device(rot)
    rng = xrng(logN)
    ct = lambda l: [uniform_limbs(rng, prm.q[:l], o.N) for _ in range(2)]  # noqa: E731
    dev = lambda c: fides.Ciphertext(fides.to_device(c[0]), fides.to_device(c[1]))  # noqa: E731
    levels = [7, 2, 5, 7]
    pairs, cts = [(ct(l), ct(l)) for l in levels], [ct(l) for l in (7, 1, 6)]
    products, rotated = ctx.mixed_batch([(dev(a), dev(b)) for a, b in pairs], rk_d, [(dev(c), rot_d, 3) for c in cts])
    alone = [ctx.mult(dev(a), dev(b), rk_d) for a, b in pairs]
    for (a, b), p, s in zip(pairs, products, alone):
        r0, r1 = o.hmult(*a, *b, rk, rescale=True)
        assert eq(p.c0, r0) and eq(p.c1, r1) and eq(s.c0, r0) and eq(s.c1, r1)
    for c, p in zip(cts, rotated):
        s = ctx.rotate(dev(c), rot_d, 3)
        assert eq(p.c0, fides.to_host(s.c0)) and eq(p.c1, fides.to_host(s.c1))


@pytest.fixture(scope="module")
def small(fides):
    from fides_b200 import params
    prm = params.chain(12, 60, 50, 3, 2)
    return prm, fides.Context(prm.logN, prm.q, prm.p, 2)


@pytest.mark.parametrize("n", [96, 97, 230, 448, 449])
def test_limbs_apart_take_one_launch_pair_per_448(fides, small, n):
    prm, ctx = small
    x = uniform_limbs(xrng(n), [prm.q[1]] * 2 * n, prm.N)
    d = fides.to_device(x)
    before = ctx.launch_count
    ctx.ntt_limbs([d[2 * i] for i in range(n)], [1] * n)
    assert ctx.launch_count - before == 2 * -(-n // 448)
    ctx.ntt_limbs([d[2 * i] for i in range(n)], [1] * n, inverse=True)
    assert eq(d, x)


@pytest.mark.parametrize("call", ["decode", "encode", "rescale", "rotate", "mult"])
def test_batches_of_more_polynomials_than_96(fides, small, call):
    """Every prologue and epilogue on a list of more than 96 runs: one item's launches, its results."""
    import torch
    prm, ctx = small
    n, rng = 100, np.random.default_rng(8)
    ct = lambda l: fides.Ciphertext(*(fides.to_device(uniform_limbs(rng, prm.q[:l], prm.N)) for _ in range(2)))  # noqa: E731
    key = fides.to_device(np.stack([np.stack([uniform_limbs(rng, prm.q + prm.p, prm.N) for _ in range(2)])
                                    for _ in range(2)]))
    polys = lambda cts: [p for c in cts for p in (c.c0, c.c1)]  # noqa: E731
    cts = [ct(2) for _ in range(n)]
    z = torch.from_numpy(rng.uniform(-1, 1, (n, 64, 2))).cuda()
    z = torch.view_as_complex(z)
    do = {"decode": lambda c, s: list(ctx.decode(torch.stack([x.c0.view(torch.int64) for x in c]).view(torch.uint64),
                                                 2.0 ** 30)),
          "encode": lambda c, s: list(ctx.encode(s, 2.0 ** 30, 2)),
          "rescale": lambda c, s: ctx.rescale_many(polys(c)),
          "rotate": lambda c, s: polys(ctx.rotate_batch([(x, key, 3) for x in c])),
          "mult": lambda c, s: polys(ctx.mult_batch([(x, x) for x in c], key))}[call]
    alone = [p for i in range(n) for p in do(cts[i:i + 1], z[i:i + 1])]
    before = ctx.launch_count
    together = do(cts, z)
    launches = ctx.launch_count - before
    assert len(alone) == len(together)
    bits = lambda t: fides.to_host(t) if t.dtype == torch.uint64 else t.cpu().numpy()  # noqa: E731
    for a, b in zip(alone, together):
        assert np.array_equal(bits(a), bits(b))
    before = ctx.launch_count
    do(cts[:1], z[:1])
    single = ctx.launch_count - before
    if call in ("decode", "encode", "rescale"):  # at most 448 limbs in each of their transforms
        assert launches == single
