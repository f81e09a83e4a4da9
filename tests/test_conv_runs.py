"""Conversions of many jobs, whose CTAs convert several runs of 128 coefficients (csrc/conv_tc.cu: two from 17
jobs at N = 2^16, four from 33, eight from 65): batches of rescaled products, whose ModDown conversions leave the
dropped limb's coefficients as their last output, and of rotations, with and without the reduced-noise lift.  Each
item equals its own call, which converts one run a CTA, and some the oracle."""
import numpy as np
import pytest

import oracle as O
from ckks_host import uniform_limbs, xrng

pytestmark = pytest.mark.gpu


def eq(gpu_t, host):
    import fides_b200 as F
    return np.array_equal(F.to_host(gpu_t), host)


@pytest.mark.parametrize("lift", [False, True])
@pytest.mark.parametrize("products,rotations", [(9, 0), (0, 17), (24, 0), (33, 15)])
def test_batches(fides, lift, products, rotations):
    from fides_b200 import params
    prm = params.chain(16, 60, 50, 6, 3, K=2)
    o = O.Oracle(prm.logN, prm.q, prm.p, 3, reduced_noise=lift)
    ctx = fides.Context(prm.logN, prm.q, prm.p, 3)
    ctx.set_conv_engine("tensor")
    ctx.set_reduced_noise(lift)
    rng = xrng(10 * products + rotations)
    key = np.stack([np.stack([uniform_limbs(rng, prm.q + prm.p, o.N) for _ in range(3)]) for _ in range(2)])
    key_d = fides.to_device(key)
    pool = {l: [uniform_limbs(rng, prm.q[:l], o.N) for _ in range(5)] for l in (6, 5, 2)}
    dev = {l: [fides.to_device(x) for x in v] for l, v in pool.items()}
    item = lambda i: ((6, 5, 6, 2, 6)[i % 5], i % 3)  # noqa: E731  level, first of its polynomials
    ct = lambda l, k: fides.Ciphertext(dev[l][k], dev[l][k + 1])  # noqa: E731
    pairs = [(ct(*item(i)), ct(item(i)[0], (item(i)[1] + 1) % 3)) for i in range(products)]
    jobs = [(ct(*item(i)), key_d, 5) for i in range(rotations)]
    got, rot = ctx.mixed_batch(pairs, key_d, jobs)
    for i, ((a, b), g) in enumerate(zip(pairs, got)):
        s = ctx.mult(a, b, key_d)
        assert eq(g.c0, fides.to_host(s.c0)) and eq(g.c1, fides.to_host(s.c1)), i
    for i, ((c, _, r), g) in enumerate(zip(jobs, rot)):
        s = ctx.rotate(c, key_d, r)
        assert eq(g.c0, fides.to_host(s.c0)) and eq(g.c1, fides.to_host(s.c1)), i
    for i in {0, 1, products - 1} & set(range(products)):
        (l, k), m = item(i), (item(i)[1] + 1) % 3
        r0, r1 = o.hmult(pool[l][k], pool[l][k + 1], pool[l][m], pool[l][m + 1], key, rescale=True)
        assert eq(got[i].c0, r0) and eq(got[i].c1, r1), i
    for i in {0, rotations - 1} & set(range(rotations)):
        l, k = item(i)
        r0, r1 = o.rotate(pool[l][k], pool[l][k + 1], key, 5)
        assert eq(rot[i].c0, r0) and eq(rot[i].c1, r1), i
