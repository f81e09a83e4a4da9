"""Rescales on primes of each size class of the integer butterflies (csrc/ntt_impl.cuh Lazy4Red; Harvey's form
from 2^61), whose epilogue takes the transform's values unreduced, and on FP64 primes beside them: with 8
residues per thread where most limbs are above 2^50 (N >= 2^15, and few limbs below), with 16 elsewhere."""
import numpy as np
import pytest

import oracle as O
from ckks_host import uniform_limbs, xrng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN,count", [(11, 2), (12, 2), (12, 12), (15, 2)])
@pytest.mark.parametrize("bits", [51, 59, 60, 61, 62])
def test_rescale(fides, logN, count, bits):
    q = O.gen_primes(logN, bits, 3) + O.gen_primes(logN, 50, 1)
    q = [q[0], q[3], q[1], q[2]]  # the limb that goes is a large prime
    o, ctx = O.Oracle(logN, q, [], 1), fides.Context(logN, q, [], 1)
    rng = xrng(100 * bits + logN)
    xs = [uniform_limbs(rng, q, o.N) for _ in range(count)]
    for i, top in enumerate(q):
        xs[0][i] = top - 1
        xs[1][i, ::2] = top - 1
        xs[1][i, 1::2] = 0
    outs = ctx.rescale_many([fides.to_device(x) for x in xs])
    for x, y in zip(xs, outs):
        assert np.array_equal(fides.to_host(y), o.rescale(x))
