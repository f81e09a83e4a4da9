// Exact modular arithmetic on integers held in doubles, for primes q < 2^50.  On B200 the FP64 pipe
// carries these products at a higher rate than the FMA-heavy pipe carries 64-bit integer ones.
#pragma once
#include <cstdint>

namespace fides {

constexpr double F64_RND = 6755399441055744.0;  // 1.5 * 2^52
constexpr double F64_TWO52 = 4503599627370496.0;

// y w mod q within q / 2 + |y w / q| 2^-52 q, exact for |y w / q| < 2^51 and products below 2^102:
// y w = p + e exactly; k = rint(p (1/q)) from one fma with the rounding constant; p - k q is an
// integer below 2^53 in magnitude, so the last fma is exact, and so is adding e.
__device__ __forceinline__ double f_mulmod(double y, double w, double q, double qinv) {
  const double p = __dmul_rn(y, w);
  const double e = __fma_rn(y, w, -p);
  const double k = __dadd_rn(__fma_rn(p, qinv, F64_RND), -F64_RND);
  return __dadd_rn(__fma_rn(-k, q, p), e);
}
// x - rint(x / q) q
__device__ __forceinline__ double f_reduce(double x, double q, double qinv) {
  const double k = __dadd_rn(__fma_rn(x, qinv, F64_RND), -F64_RND);
  return __fma_rn(-k, q, x);
}
// u64 < 2^52 -> double (exact)
__device__ __forceinline__ double f_from_u64(uint64_t v) {
  return __dadd_rn(__longlong_as_double((long long)(0x4330000000000000ull | v)), -F64_TWO52);
}
// the canonical residue of an integer |s| < 2^53
__device__ __forceinline__ uint64_t f_canon(double s, double q, double qinv) {
  double r = f_reduce(s, q, qinv);  // |r| <= q / 2 + 1
  if (r < 0) r = __dadd_rn(r, q);
  return (uint64_t)__double_as_longlong(__dadd_rn(r, F64_TWO52)) & ((1ull << 52) - 1);
}

// An inner product sum a_i b_i of residues, exact, reduced once.  h starts at h0 and takes the
// products by fma, which rounds to its ulp of 2^51 while it stays in [2^103, 2^104); the part of a
// product that h did not take, at most 2^50 in magnitude, is found exactly and summed in l, exact up
// to 2^53.  Four operations a term, against seven for a reduced product each.
// F64Acc: h0 = 1.25 2^103, sums in [-2, 6) 2^100 of at most 7 terms.  F64AccPos: h0 = 2^103, at most 8
// terms of products of two residues.
template <bool POS>
struct F64AccT {
  static constexpr double H0 = POS ? 0x1p103 : 0x1.4p103;
  double h = H0, l = 0.0;
  __device__ __forceinline__ void mac(double a, double b) {
    const double n = __fma_rn(a, b, h);
    l = __dadd_rn(l, __fma_rn(a, b, -__dadd_rn(n, -h)));
    h = n;
  }
  // An integer below 2^53 in magnitude that is congruent to the sum: (h - h0) 2^-51, below 2^52 in
  // magnitude, times 2^51 mod q (w51, centred), plus l (POS: plus its residue, so within 2q).
  __device__ __forceinline__ double fold(double w51, double q, double qinv) const {
    const double r = f_mulmod(__dmul_rn(__dadd_rn(h, -H0), 0x1p-51), w51, q, qinv);
    return __dadd_rn(r, POS ? f_reduce(l, q, qinv) : l);
  }
};
using F64Acc = F64AccT<false>;
using F64AccPos = F64AccT<true>;

// A sum of any number of products of two residues, eight at first and at most seven after each fold: a
// fold leaves its residue, below 2^49 + 1 in magnitude, in l, which is exact up to 2^53.  (A third
// double for the folded part cost eight registers where four sums run, and a CTA an SM.)
struct F64Sum {
  F64AccPos acc;
  __device__ __forceinline__ void mac(double a, double b) { acc.mac(a, b); }
  __device__ __forceinline__ void flush(double w51, double q, double qinv) {
    acc.l = f_reduce(acc.fold(w51, q, qinv), q, qinv);
    acc.h = F64AccPos::H0;
  }
  __device__ __forceinline__ uint64_t residue(double w51, double q, double qinv) const {
    return f_canon(acc.fold(w51, q, qinv), q, qinv);
  }
};

}  // namespace fides
