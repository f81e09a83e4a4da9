"""Exactness of the floating-point modular arithmetic inside the kernels, checked on the CPU.

The kernels compute integer results with FP64 operations whose exactness rests on rounding
bounds; these tests replay the same operation sequences in Python (IEEE doubles, and an exact
fused multiply-add through rational arithmetic) on random and extreme operands, and compare
with exact integer arithmetic:

* the NTT's prologues and epilogues on FP64 limbs (primes below 2^50, csrc/ntt_impl.cuh): products by
  `f_mulmod`, `f_reduce` (csrc/f64arith.cuh), the signed coefficients of the encoder (`signed_f64`), the
  canonical residue of a result (`f_to_canon`), and the first stage on uncentred inputs in [0, q).  The
  butterflies' bounds and the sums of products are in test_ntt_fp64_bounds.py;
* the tensor-core conversion's fold of eight s32 byte planes with a one-sided quotient
  correction (`tc_fold`, csrc/conv_tc.cu).
"""
import math
import random
from fractions import Fraction

import pytest

RND = 6755399441055744.0  # 1.5 * 2^52
TWO52 = 4503599627370496.0


def fma(a: float, b: float, c: float) -> float:
    """a * b + c with one rounding (float(Fraction) rounds to nearest, ties to even)."""
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def rint(x: float) -> float:
    return (x + RND) - RND


def primes50():
    from fides_b200 import params
    return [q for q in params.config_c(4).q if q < (1 << 50)]


def f_mulmod(y, w, q, qinv):
    p = y * w
    e = fma(y, w, -p)
    k = fma(p, qinv, RND) - RND
    return fma(-k, q, p) + e


def f_reduce(x, q, qinv):
    return fma(-(fma(x, qinv, RND) - RND), q, x)


def centred(w, q):
    return float(w - q if w > q // 2 else w)


def f_to_canon(v, q):
    u = int(Fraction(v + (2.0 * q + TWO52))) & ((1 << 52) - 1)
    u = u - 2 * q if u >= 2 * q else u
    return u - q if u >= q else u


def all_primes():
    from fides_b200 import params
    return primes50()[:5] + params.gen_primes(12, 34, 1) + params.gen_primes(12, 30, 1) + [(1 << 50) - 27, 12289]


def exact(v, ref, q, bound):
    """v is an integer congruent to ref within `bound`."""
    assert v == int(v) and (int(v) - ref) % q == 0 and abs(v) <= bound + 1


def test_prologues():
    """Inputs of a transform's first stage: within 4q forward, within q inverse."""
    rng = random.Random(11)
    for q in all_primes():
        qd, qinv = float(q), 1.0 / q
        pick = lambda: rng.choice([rng.randrange(q), q - 1, 0, q // 2])  # noqa: E731
        for it in range(200):
            a, b = pick(), pick()  # the tensor term a1 b1
            exact(f_mulmod(float(a), float(b), qd, qinv), a * b, q, 0.75 * q)
            # the centred lift of a residue of any other prime below 2^50, and P times it beside the
            # conversion's value
            c = rng.choice([rng.randrange(-(1 << 49), (1 << 49) + 1), 1 << 49, -(1 << 49)])
            exact(f_reduce(float(c), qd, qinv), c, q, q / 2)
            P, x = rng.randrange(q), pick()
            exact(float(x) + f_mulmod(float(c), centred(P, q), qd, qinv), x + c * P, q, 2 * q)
            exact(float(x) + f_mulmod(float(a), centred(P, q), qd, qinv), x + a * P, q, 2 * q)
            if q >= 1 << 33:  # signed_f64: the upper word's part reduced, the lower word as it is
                m = rng.choice([rng.randrange(-(1 << 63), 1 << 63), (1 << 63) - 1, -(1 << 63), -1,
                                rng.randrange(-(1 << 45), 1 << 45)])
                hi = f_reduce(float((m >> 32) << 32), qd, qinv)
                exact(hi + float(m & 0xffffffff), m, q, q)


def test_epilogues():
    """Results of a transform, within 2q, through the epilogues to canonical residues."""
    rng = random.Random(12)
    for q in all_primes():
        qd, qinv = float(q), 1.0 / q
        pick = lambda: rng.choice([rng.randrange(q), q - 1, 0])  # noqa: E731
        for it in range(200):
            v = rng.choice([rng.randrange(-2 * q + 1, 2 * q), 2 * q - 1, -2 * q + 1, 0])
            assert f_to_canon(float(v), qd) == v % q
            e0, e1, w, m = pick(), pick(), pick(), pick()
            down = f_mulmod(float(e0) - float(v), centred(w, q), qd, qinv)  # ModDown, and with a rescale
            exact(down, (e0 - v) * w, q, 0.875 * q)
            assert f_to_canon(down, qd) == (e0 - v) * w % q
            assert f_to_canon(down + float(e1), qd) == ((e0 - v) * w + e1) % q
            scaled = f_mulmod(float(e0), centred(w, q), qd, qinv) + f_mulmod(float(v), centred(m, q), qd, qinv)
            exact(scaled, e0 * w + v * m, q, 1.5 * q)
            assert f_to_canon(scaled, qd) == (e0 * w + v * m) % q


def test_first_stage_on_uncentred_inputs():
    """The first pass converts canonical residues in [0, q) without centring them: the forward first stage
    reduces its x operand and multiplies y < q; the inverse first stage adds (< 2q) and multiplies the
    difference (|d| < q).  Both stay exact within the bounds the later stages assume."""
    rng = random.Random(13)
    for q in all_primes():
        qd, qinv = float(q), 1.0 / q
        for it in range(300):
            w = rng.randrange(-(q // 2), q // 2 + 1)
            x, y = rng.randrange(0, q), rng.randrange(0, q)
            if it % 50 == 0:
                x, y = q - 1, q - 1
            a, r = f_reduce(float(x), qd, qinv), f_mulmod(float(y), float(w), qd, qinv)
            exact(a + r, x + y * w, q, 1.125 * q)
            exact(a - r, x - y * w, q, 1.125 * q)
            exact(f_mulmod(float(x) - float(y), float(w), qd, qinv), (x - y) * w, q, 0.625 * q)


def tc_fold(d, q, qinv):
    a0, a1 = d[0] + (d[1] << 8), d[2] + (d[3] << 8)
    a2, a3 = d[4] + (d[5] << 8), d[6] + (d[7] << 8)
    assert max(a0, a1, a2, a3) < 1 << 32
    x, y = a0 + (a1 << 16), a2 + (a3 << 16)
    vd = fma(float(y), 4294967296.0, float(x))
    t = fma(vd, qinv, 2.0 ** -17)
    qh = math.floor(t)
    assert 0 <= qh < 1 << 32
    m = (1 << 64) - 1
    r = (x + (y << 32) - qh * q) & m
    if r >> 63:
        r = (r + q) & m
    return r


@pytest.mark.parametrize("bits", [49, 50, 55, 60, 61])
def test_conversion_fold_one_sided_correction(bits):
    rng = random.Random(bits)
    dmax = 128 * 255 * 255  # K = 128 bytes of u8 x u8 products
    for _ in range(40):
        q = rng.randrange(1 << (bits - 1), 1 << bits) | 1
        if q <= 1 << 48:
            continue
        qinv = 1.0 / q
        for it in range(60):
            if it % 3 == 0:  # next to a multiple of q
                k = rng.randrange((dmax << 56) // q)
                v = k * q + rng.randrange(-32, 33)
                v = max(v, 0)
                d = [(v >> (8 * c)) & 255 for c in range(7)] + [v >> 56]
            else:
                d = [rng.randrange(dmax + 1) for _ in range(8)]
                if it % 11 == 1:
                    d = [dmax] * 8
            v = sum(dc << (8 * c) for c, dc in enumerate(d))
            assert tc_fold(d, q, qinv) == v % q
