"""Exactness and bounds of the NTT's FP64 butterflies (primes below 2^50, csrc/ntt_impl.cuh).

The quotient of a product is taken from the rounded product itself (`f_mulmod`) and most stages
leave their sums unreduced; these tests replay the product on operands at the largest magnitudes a
stage meets, and the bound recurrence of every chunk of every ring dimension, on the CPU.
"""
import random
from fractions import Fraction

import pytest

RND = 6755399441055744.0  # 1.5 * 2^52


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def f_mulmod(y, w, q, qinv):
    p = y * w
    e = fma(y, w, -p)
    k = fma(p, qinv, RND) - RND
    return fma(-k, q, p) + e


def primes():
    from fides_b200 import params
    return params.gen_primes(16, 50, 4) + params.gen_primes(10, 50, 2) + params.gen_primes(12, 30, 1) + [12289]


def test_product_is_exact_up_to_four_q():
    rng = random.Random(5)
    for q in primes():
        qd, qinv = float(q), 1.0 / q
        for it in range(500):
            w = rng.randrange(-(q // 2), q // 2 + 1) if it % 5 else rng.choice([-1, 1]) * (q // 2)
            y = rng.randrange(-4 * q, 4 * q + 1) if it % 3 else rng.choice([-1, 1]) * (4 * q - rng.randrange(3))
            if w and it % 7 == 0:  # next to a half-integer quotient, where k could fall either way
                y = (rng.randrange(-2 * q, 2 * q) * q + q // 2) // w
                if abs(y) > 4 * q:
                    continue
            r = f_mulmod(float(y), float(w), qd, qinv)
            assert r == int(r) and (int(r) - y * w) % q == 0
            assert abs(r) <= q / 2 + abs(y) / 8 + 1


@pytest.mark.parametrize("logp", [5, 6, 7, 8, 9])
@pytest.mark.parametrize("le", [3, 4])
def test_stage_bounds(logp, le):
    """Bounds in units of q: every product operand within 4, every value within 8 (2^53), every
    transform result within 2 (f_to_canon)."""
    chunks = -(-logp // le)
    # forward: the column pass from canonical input, then the row pass; a row pass follows any column
    bound = 1.0
    for row in (False, True):
        for c in range(chunks):
            n = min(le, logp - c * le)
            last = row and c == chunks - 1
            for k in range(n):
                red = k == 0 or (last and n >= 2 and k == (n - 2 if n > 2 else 1))
                assert bound <= 4
                product = 0.5 + bound / 8
                bound = (0.5 if red else bound) + product
                assert bound < 4
    assert bound < 2
    # inverse: the row pass from canonical input, then the column pass and its last multiplications
    bound = 1.0
    for row in (True, False):
        for b in range(logp):
            assert 2 * bound <= 4
            if not row and b == logp - 1:
                bound = 0.5 + 2 * bound / 8
                continue
            red = bool(b & 1) or (row and b == logp - 1)
            bound = max(0.5 if red else 2 * bound, 0.5 + 2 * bound / 8)
    assert bound < 2


def test_lazy4_product_range():
    """shoup_lazy4 (csrc/modarith.cuh): y w mod q plus 0 to 3 q, for any 64-bit y and q < 2^61."""
    from fides_b200 import params
    rng = random.Random(9)
    for q in (params.gen_primes(16, 61, 2) + params.gen_primes(16, 60, 2) + params.gen_primes(16, 59, 1) +
              params.gen_primes(16, 51, 1)):
        for it in range(3000):
            w = rng.choice([rng.randrange(q), q - 1 - rng.randrange(3), rng.randrange(3)])
            y = rng.choice([rng.randrange(1 << 64), (1 << 64) - 1 - rng.randrange(1 << 33), rng.randrange(1 << 33),
                            rng.randrange(1 << 32) << 32, (rng.randrange(1 << 32) << 32) | 0xffffffff])
            ws = (w << 64) // q
            y0, y1, s0, s1 = y & 0xffffffff, y >> 32, ws & 0xffffffff, ws >> 32
            k = y1 * s1 + (y1 * s0 >> 32) + (y0 * s1 >> 32)
            assert k < 1 << 64 and 0 <= y * w - k * q < 4 * q


@pytest.mark.parametrize("bits", [51, 58, 59, 60, 61])
def test_lazy4_forward_bounds(bits):
    """Forward values with the chunk-wise subtractions of Lazy4Red stay below 2^64; x is below 2 cm
    where it is subtracted."""
    q = (1 << bits) - 1  # any value of this size
    cm = 16 * q if q < 1 << 59 else 8 * q if q < 1 << 60 else 4 * q
    third, odd = q >= 1 << 59, q >= 1 << 60
    for le in (3, 4):
        for logp in (5, 6, 7, 8, 9):
            bound = q
            for _ in range(2):  # the column pass, then the row pass
                for c in range(-(-logp // le)):
                    for k in range(min(le, logp - c * le)):
                        if k == 0 or (third if k == 2 else odd):
                            assert bound <= 2 * cm
                            bound = max(cm, bound - cm)
                        bound += 4 * q
                        assert bound <= 1 << 64


class Acc:
    """F64Acc (csrc/f64arith.cuh)."""
    H0 = 1.25 * 2.0 ** 103

    def __init__(self):
        self.h, self.l = self.H0, 0.0

    def mac(self, a, b):
        n = fma(a, b, self.h)
        self.l += fma(a, b, -(n - self.h))
        self.h = n

    def fold(self, q, qinv):
        w51 = pow(2, 51, q)
        w51 = float(w51 - q if w51 > q // 2 else w51)
        return f_mulmod((self.h - self.H0) * 2.0 ** -51, w51, float(q), qinv) + self.l


def canon(s, q, qinv):
    r = fma(-(fma(s, qinv, RND) - RND), q, s)
    return int(r + q if r < 0 else r)


def test_inner_product_is_exact():
    """The key-switch inner product's extreme cases: four digits, the own one a product of two
    residues, and the tensor terms with P b0, P b1."""
    rng = random.Random(3)
    for q in primes():
        qd, qinv = float(q), 1.0 / q
        pick = lambda: rng.choice([rng.randrange(q), q - 1, q - 1 - rng.randrange(2), 0])  # noqa: E731
        for it in range(300):
            acc, want = Acc(), 0
            for d in range(4):
                x = float(pick())
                if d == it % 5:
                    y = pick()
                    x, x0 = f_mulmod(x, float(y), qd, qinv), int(x) * y
                    assert (int(x) - x0) % q == 0 and abs(x) <= 0.75 * q + 1
                k = pick()
                acc.mac(x, float(k))
                want += int(x) * k
            P = rng.randrange(-(q // 2), q // 2 + 1)
            for _ in range(2):
                p = f_mulmod(float(pick()), float(P), qd, qinv)
                assert abs(p) <= 0.625 * q + 1
                a = pick()
                acc.mac(float(a), p)
                want += a * int(p)
            s = acc.fold(q, qinv)
            assert abs(s) < 2.0 ** 53 and canon(s, qd, qinv) == want % q


class Sum(Acc):
    """F64Sum over F64AccPos (csrc/f64arith.cuh)."""
    H0 = 2.0 ** 103

    def fold(self, q, qinv):
        l, self.l = self.l, 0.0
        r = super().fold(q, qinv) + f_reduce(l, float(q), qinv)
        self.l = l
        return r

    def flush(self, q, qinv):
        self.l, self.h = f_reduce(self.fold(q, qinv), float(q), qinv), self.H0


def f_reduce(x, q, qinv):
    return fma(-(fma(x, qinv, RND) - RND), q, x)


@pytest.mark.parametrize("block", [4, 7])
def test_long_sums_are_exact(block):
    """Sums of residue products folded after the first eight terms and then after every `block` (4 in
    dot_plain and lincomb, 7 in the BSGS sums), at the largest residues and at products whose low parts
    lie half an ulp of h from it, all on one side."""
    rng = random.Random(block)
    for q in primes()[:6] + [(1 << 50) - 27]:
        qd, qinv = float(q), 1.0 / q
        for it in range(60):
            acc, want, rest = Sum(), 0, 8
            for t in range(40):
                if not rest:
                    acc.flush(q, qinv)
                    assert abs(acc.l) <= 2.0 ** 49 + 1
                    rest = block
                a, b = rng.choice([(q - 1, q - 1), (rng.randrange(q), rng.randrange(q)), (0, q - 1)])
                if it % 2 and q > 1 << 49:  # ab = 2^50 - r modulo 2^51, r small
                    a = rng.randrange(q // 2, q - 1) | 1
                    b = min(((1 << 50) - rng.randrange(3)) * pow(a, -1, 1 << 51) % (1 << 51), q - 1)
                acc.mac(float(a), float(b))
                assert abs(acc.l) <= 2.0 ** 53
                want += a * b
                rest -= 1
            s = acc.fold(q, qinv)
            assert abs(s) < 2.0 ** 53 and canon(s, qd, qinv) == want % q
