"""Transforms of the residues that bring the butterflies' values to their bounds (all q - 1, 0 and q - 1 in
turn, one or two large coefficients) on primes of every butterfly form, at both counts of residues per thread,
and the slot encoder on primes below 2^33, whose signed coefficients are reduced in integers."""
import numpy as np
import pytest

import oracle as O
from ckks_host import encode, xrng
from test_encode import device_coeffs

pytestmark = pytest.mark.gpu

BITS = [30, 50, 50, 51, 59, 60, 61, 62]


def extremes(q, N, rng):
    """One polynomial of limbs modulo q for each shape."""
    i = np.arange(N)
    sparse = np.isin(i, [1, N - 1])
    return [np.stack([np.where(on, p - 1, 0).astype(np.uint64) for p in q]) for on in
            (i >= 0, i % 2 == 0, i % 2 == 1, i < N // 2, i // (N >> 5) % 2 == 0, i == 0, sparse)] + \
        [np.stack([np.where(rng.integers(0, 2, N) > 0, p - 1, p // 2).astype(np.uint64) for p in q])]


@pytest.mark.parametrize("logN,residues", [(10, 16), (12, 8), (13, 16), (15, 8), (15, 16), (16, 8), (16, 16)])
@pytest.mark.parametrize("inverse", [False, True])
def test_transforms(fides, logN, residues, inverse):
    q = []
    for b in BITS:
        q += O.gen_primes(logN, b, 1, exclude=q)
    o, ctx = O.Oracle(logN, q, [], 1), fides.Context(logN, q, [], 1)
    ids = list(range(len(q)))
    if logN >= 15:
        for inv in (False, True):
            for p in (0, 1):
                for size in range(4):
                    ctx.set_ntt_residues(inv, p, size, residues)
    xs = extremes(q, o.N, xrng(logN))
    together = 1 if residues == 8 else len(xs)  # small rings: 8 residues for up to 32 limbs, 16 beyond
    for k in range(0, len(xs), together):
        x = np.stack(xs[k:k + together])
        d = fides.to_device(x)
        (ctx.intt if inverse else ctx.ntt)(d)
        got = fides.to_host(d)
        for g, v in zip(got, x):
            assert np.array_equal(g, o.ntt(v, ids, inverse=inverse))


def test_encode_on_small_primes(fides):
    import torch
    logN, scale = 12, 2.0 ** 40
    q = O.gen_primes(logN, 60, 1) + O.gen_primes(logN, 30, 1) + O.gen_primes(logN, 33, 1) + O.gen_primes(logN, 34, 1)
    o, ctx = O.Oracle(logN, q, [], 1), fides.Context(logN, q, [], 1)
    N = o.N
    z = xrng(3).uniform(-1, 1, (2, N // 2)) + 1j * xrng(4).uniform(-1, 1, (2, N // 2))
    z[1] *= 2.0 ** 18  # coefficients of both signs about 2^52, whose FP64 errors are some units
    pts = ctx.encode(torch.from_numpy(z), scale, 4)
    for i, units in enumerate([1, 64]):
        m = device_coeffs(fides, ctx, pts[i][:1], q)[0]
        assert np.abs(m - encode(z[i], N, scale).astype(np.int64)).max() <= units
        limbs = np.stack([np.mod(m, p).astype(np.uint64) for p in q])
        assert np.array_equal(fides.to_host(pts[i]), o.ntt(limbs, [0, 1, 2, 3]))
