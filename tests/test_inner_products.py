"""GPU tests of the plaintext inner products and linear combinations (fides_dot_plain, fides_dot_plain_bsgs,
fides_lincomb) against exact integers, at the term counts where the kernels' sums are folded, on primes
below and above 2^50, with residues at their largest among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[50, 59])
def env(request, fides):
    from fides_b200 import params
    p = params.chain(12, 60, request.param, 4, 2)
    ctx = fides.Context(p.logN, p.q, p.p, p.dnum)
    yield fides, ctx
    ctx.close()


def residues(rng, primes, N):
    x = np.stack([rng.integers(0, q, N, dtype=np.uint64) for q in primes])
    for r, q in zip(x, primes):
        r[:64] = q - 1
        r[64:80] = 0
    return x


def check(got, primes, want):
    for i, q in enumerate(primes):
        assert np.array_equal(got[i], np.array([v % q for v in want[i]], dtype=np.uint64))


def products(ws, xs):
    """sum_t ws[t] xs[t] over limbs, as exact integers."""
    return sum(np.asarray(w, dtype=object) * np.asarray(x, dtype=object) for w, x in zip(ws, xs))


@pytest.mark.parametrize("n", [1, 4, 5, 8, 9, 13, 32])
@pytest.mark.parametrize("ext", [False, True])
def test_dot_plain(env, n, ext):
    F, ctx = env
    rng = np.random.default_rng(n)
    level = 3
    primes = ctx.q[:level] + (ctx.p if ext else [])
    c0, c1, w = ([residues(rng, primes, ctx.N) for _ in range(n)] for _ in range(3))
    cts = [F.Ciphertext(F.to_device(a), F.to_device(b)) for a, b in zip(c0, c1)]
    pts = [F.to_device(a) for a in w]
    out = ctx.dot_plain_ext(cts, pts, level) if ext else ctx.dot_plain(cts, pts)
    check(F.to_host(out.c0), primes, products(w, c0))
    check(F.to_host(out.c1), primes, products(w, c1))


@pytest.mark.parametrize("nb,ng", [(1, 1), (7, 3), (8, 4), (9, 2), (16, 5)])
@pytest.mark.parametrize("offset", [0, 1])
def test_dot_plain_bsgs(env, nb, ng, offset):
    """offset: operands off 16-byte alignment, which take one coefficient per thread."""
    F, ctx = env
    rng = np.random.default_rng(10 * nb + ng)
    level = 3
    primes = ctx.q[:level]

    def place(a):
        import torch
        b = torch.zeros(a.size + 2, dtype=torch.int64, device="cuda")[offset:offset + a.size]
        b.copy_(F.to_device(a).view(torch.int64).reshape(-1))
        return b.view(torch.uint64).view(a.shape)
    x0, x1 = ([residues(rng, primes, ctx.N) for _ in range(nb)] for _ in range(2))
    w = [[residues(rng, primes, ctx.N) if (i + k) % 5 or k == 0 else None for k in range(nb)] for i in range(ng)]
    babies = [F.Ciphertext(place(a), place(b)) for a, b in zip(x0, x1)]
    outs = ctx.dot_plain_bsgs(babies, [[None if d is None else place(d) for d in row] for row in w], level)
    for i in range(ng):
        on = [k for k in range(nb) if w[i][k] is not None]
        check(F.to_host(outs[i].c0), primes, products([w[i][k] for k in on], [x0[k] for k in on]))
        check(F.to_host(outs[i].c1), primes, products([w[i][k] for k in on], [x1[k] for k in on]))


@pytest.mark.parametrize("n", [1, 8, 9, 16])
def test_lincomb(env, n):
    F, ctx = env
    rng = np.random.default_rng(n + 50)
    level = 3
    primes = ctx.q[:level]
    c0, c1 = ([residues(rng, primes, ctx.N) for _ in range(n)] for _ in range(2))
    s = [[q - 1 - (t % 3) for q in primes] for t in range(n)]
    add = [q - 1 for q in primes]
    out = ctx.lincomb([F.Ciphertext(F.to_device(a), F.to_device(b)) for a, b in zip(c0, c1)], s, add)
    cols = [np.array(v, dtype=object)[:, None] for v in s]
    check(F.to_host(out.c0), primes, products(cols, c0) + np.array(add, dtype=object)[:, None])
    check(F.to_host(out.c1), primes, products(cols, c1))
