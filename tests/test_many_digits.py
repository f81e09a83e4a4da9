"""Key switches of up to 14 digits, alone, in batches under one key and hoisted, against the oracle: up to four
digits have kernels of their own, more take the general one."""
import numpy as np
import pytest

import oracle as O
from ckks_host import uniform_limbs, xrng

pytestmark = pytest.mark.gpu


def eq(gpu_t, host):
    import fides_b200 as F
    return np.array_equal(F.to_host(gpu_t), host)


@pytest.mark.parametrize("digits", [1, 2, 3, 4, 5, 8, 9, 10, 11, 12, 13, 14])
def test_key_switches(fides, digits):
    logN = 10
    q, p = (O.gen_primes(logN, 60, 1) + O.gen_primes(logN, 50, 13))[:digits], O.gen_primes(logN, 61, 2)
    o, ctx = O.Oracle(logN, q, p, digits), fides.Context(logN, q, p, digits)
    rng = xrng(digits)
    key = np.stack([np.stack([uniform_limbs(rng, q + p, o.N) for _ in range(digits)]) for _ in range(2)])
    key_d = fides.to_device(key)
    cts = [[uniform_limbs(rng, q, o.N) for _ in range(2)] for _ in range(4)]
    dev = [fides.Ciphertext(fides.to_device(a), fides.to_device(b)) for a, b in cts]
    want_r = [o.rotate(*c, key, 3) for c in cts]
    want_m = o.hmult(*cts[0], *cts[1], key, rescale=False)
    same = lambda g, w: eq(g.c0, w[0]) and eq(g.c1, w[1])  # noqa: E731
    assert same(ctx.rotate(dev[0], key_d, 3), want_r[0])
    assert same(ctx.mult(dev[0], dev[1], key_d, rescale=False), want_m)
    for n in (2, 4):
        assert all(same(g, w) for g, w in zip(ctx.rotate_batch([(c, key_d, 3) for c in dev[:n]]), want_r))
        assert all(same(g, want_m) for g in ctx.mult_batch([(dev[0], dev[1])] * n, key_d, rescale=False))
        h0, h1 = o.rotate_hoisted(*cts[0], [key] * n, list(range(1, n + 1)))
        got = ctx.rotate_hoisted(dev[0], [key_d] * n, list(range(1, n + 1)))
        assert all(same(g, w) for g, w in zip(got, zip(h0, h1)))
