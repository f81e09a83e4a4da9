// Elementwise RNS kernels, basis conversion and KSK inner product.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "kernels.cuh"
#include "conv_tc.hpp"
#include "f64arith.cuh"
#include "launch.cuh"
#include "ntt.cuh"

namespace fides {

namespace {

// automorph_slot (reference src/Rotation.cuh:14-26): j -> brev(((2 brev(j) + 1) k mod 2N) >> 1)
__device__ __forceinline__ uint32_t auto_slot(int logN, uint32_t k, uint32_t j) {
  uint32_t jr = __brev(j) >> (32 - logN);
  uint32_t r = ((((jr << 1) + 1) * k) & ((2u << logN) - 1)) >> 1;
  return __brev(r) >> (32 - logN);
}

constexpr int MAX_SRC = 64;   // limbs on the source side of one conversion
constexpr int MAX_DST = 128;  // limbs on the destination side

// Basis conversion.  NS (source limbs) is a template parameter so that the pre-scaled
// sources stay in registers; NS = 0 is the generic width.  Each thread converts two
// adjacent coefficients (16-byte accesses); destination primes, output positions and the
// conversion matrix are staged in shared memory (broadcast reads).
template <int NS>
__global__ void __launch_bounds__(EW_THREADS) conv_kernel(const __grid_constant__ ConvJobList L, const DevPrime* primes,
                                                          int logN) {
  const ConvJob& J = L.j[blockIdx.y];
  const ConvTable& T = J.t;
  extern __shared__ uint64_t sm[];
  const int ns = NS ? NS : T.n_src, nd = T.n_dst, lift = T.lift;
  DevPrime* dp = reinterpret_cast<DevPrime*>(sm);             // [nd]
  uint64_t* mat = sm + sizeof(DevPrime) / 8 * nd;             // [ns + lift][nd]
  int* dpos = reinterpret_cast<int*>(mat + (ns + lift) * nd); // [nd]
  for (int i = threadIdx.x; i < (ns + lift) * nd; i += blockDim.x) mat[i] = T.mat[i];
  for (int j = threadIdx.x; j < nd; j += blockDim.x) {
    dp[j] = primes[T.dst_prime[j]];
    dpos[j] = T.dst_pos(j);
  }
  __syncthreads();
  pdl_wait();
  const int N = 1 << logN;
  const int n = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  constexpr int R = NS ? NS : MAX_SRC;
  uint64_t y0[R], y1[R];
  uint64_t lift0 = 0, lift1 = 0;  // reduced-noise lift: sources above q_i / 2
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (NS == 0 && i >= ns) break;
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(J.src + (size_t)(T.src0 + i) * N + n);
    y0[i] = v.x;
    y1[i] = v.y;
    if (lift) {
      const uint64_t half = primes[T.src_prime[i]].q >> 1;
      lift0 += y0[i] > half;
      lift1 += y1[i] > half;
    }
  }
  uint64_t* dst = J.dst + n;
  for (int j = 0; j < nd; ++j) {
    const DevPrime p = dp[j];
    U128 a0{0, 0}, a1{0, 0};
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (NS == 0 && i >= ns) break;
      if (i && (i & 7) == 0) {  // keep the sums below 2^128
        a0 = U128{reduce128(a0, p), 0};
        a1 = U128{reduce128(a1, p), 0};
      }
      const uint64_t m = mat[i * nd + j];
      mac128(a0, y0[i], m);
      mac128(a1, y1[i], m);
    }
    if (lift) {  // count (<= 64) times [-Q_src]_{p_j}: below 2^69, no reduction needed first
      const uint64_t m = mat[ns * nd + j];
      mac128(a0, lift0, m);
      mac128(a1, lift1, m);
    }
    uint64_t r0 = reduce128(a0, p), r1 = reduce128(a1, p);
    if (J.top && j == nd - 1) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(J.top + n);
      r0 = shoup(submod(t.x, r0, p.q), J.top_pinv.w, J.top_pinv.ws, p.q);
      r1 = shoup(submod(t.y, r1, p.q), J.top_pinv.w, J.top_pinv.ws, p.q);
    }
    *reinterpret_cast<ulonglong2*>(dst + (size_t)dpos[j] * N) = make_ulonglong2(r0, r1);
  }
}

// CPT adjacent coefficients per thread (the launches use CPT = 2: 16-byte loads of every
// stream; one coefficient per thread was measured 13 % slower).  MAXB is the largest digit
// count of the launch's jobs (0 = any): with it known at compile time every load of a job --
// all digits, the own-digit and tensor operands -- is issued before its first product.  JG:
// jobs per group (one CTA runs a group; its jobs share the key tile, read once).
template <int CPT>
struct KVec {
  uint64_t c[CPT];
};
template <int CPT>
struct KDbl {
  double c[CPT];
};
template <int CPT>
__device__ __forceinline__ KVec<CPT> kld(const uint64_t* q) {
  KVec<CPT> v;
  if constexpr (CPT == 2) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(q);
    v.c[0] = t.x;
    v.c[1] = t.y;
  } else {
    v.c[0] = *q;
  }
  return v;
}
template <int CPT>
__device__ __forceinline__ KDbl<CPT> kdbl(const KVec<CPT>& v) {
  KDbl<CPT> d;
#pragma unroll
  for (int c = 0; c < CPT; ++c) d.c[c] = f_from_u64(v.c[c]);
  return d;
}

// Three CTAs (24 warps) per SM: 80 registers.
template <int MAXB, int JG>
struct KskMinBlocks {
  static constexpr int value = (JG > 1 || (MAXB >= 1 && MAXB <= 3)) ? 3 : 1;
};

template <int MAXB, int JG, int CPT, int CAP, bool SHARE_DIGITS = false>
__global__ void __launch_bounds__(EW_THREADS, KskMinBlocks<MAXB, JG>::value)
    ksk_kernel(const __grid_constant__ KskJobListT<CAP> L, const DevPrime* primes, const ShoupConst* pmod,
               const F64Prime* f64, int logN, int n_q, int K, int dnum, int alpha) {
  using V = KVec<CPT>;
  using D = KDbl<CPT>;
  const int g0 = L.gstart[blockIdx.z], gn = L.gcount[blockIdx.z];
  const KskJob& J0 = L.j[g0];  // the group's jobs share key, level and extras
  const int l = J0.l, ext = l + K;
  const int i = blockIdx.y;
  if (i >= ext) return;
  const int N = 1 << logN;
  const int n = CPT * (blockIdx.x * blockDim.x + threadIdx.x);
  const int pid = i < l ? i : n_q + (i - l);
  const int beta = (l + alpha - 1) / alpha;
  const int own = i < l ? i / alpha : -1;
  const size_t kstride = (size_t)(n_q + K) * N;
  const size_t off = (size_t)i * N + n, koff = (size_t)pid * N + n;
  const bool tensor = J0.a0 && i < l;
  const uint64_t q = primes[pid].q;
  pdl_wait();

  auto ld_digit = [&](const KskJob& J, int d) {
    return kld<CPT>((d == own && J.x) ? J.x + off : J.digits + ((size_t)d * ext + i) * N + n);
  };
  auto ld_key = [&](const KskJob& J, int side, int d) {
    return kld<CPT>(J.key + (size_t)(side * dnum + d) * kstride + koff);
  };
  auto store = [&](const KskJob& J, const uint64_t (&ra)[CPT], const uint64_t (&rb)[CPT]) {
    uint64_t* oa = J.out_a + (size_t)i * N;
    uint64_t* ob = J.out_b + (size_t)i * N;
    if (J.auto_k) {
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const uint32_t o = auto_slot(logN, J.auto_k, (uint32_t)(n + c));
        oa[o] = ra[c];
        ob[o] = rb[c];
      }
    } else if constexpr (CPT == 2) {
      *reinterpret_cast<ulonglong2*>(oa + n) = make_ulonglong2(ra[0], ra[1]);
      *reinterpret_cast<ulonglong2*>(ob + n) = make_ulonglong2(rb[0], rb[1]);
    } else {
      oa[n] = ra[0];
      ob[n] = rb[0];
    }
  };

  // Limbs of primes below 2^50, at most four digits: both sides as exact FP64 inner products
  // (F64Acc).  Bounds in units of 2^100: the own digit a1 b1 is within 0.75 q (f_mulmod of two
  // residues), P b0 and P b1 within 0.625 q, P within q / 2, so a side sums between -0.75 - 1.25
  // and 4 + 1.25 in at most 6 terms.  Memory bounds this form: 461 us for the 16 jobs of 8 products and
  // 8 rotations at N = 2^16, level 30, 3 digits (2.36 GB, 5.1 TB/s).  With 128-bit integer sums on the b
  // side (FMA-heavy pipe) and a reduced FP64 product a term on the a side it took 629 us, issue 53 %.
  if constexpr (MAXB > 0) {
    if (q < NTT_F64_MAX) {
      const F64Prime fp = f64[pid];
      // a job alone (or one that shares only its digits) loads its keys with its other operands, so that
      // it waits for memory once (one product at N = 2^16, level 30: 54.5 -> 51.5 us)
      constexpr bool OWN_KEYS = SHARE_DIGITS || JG == 1;
      auto run = [&](const KskJob& J, const D* ka_g, const D* kb_g, const D* vd) {
        V v[MAXB], ka[MAXB], kb[MAXB], y1{}, x0{}, y0{}, c0{};
#pragma unroll
        for (int d = 0; d < MAXB; ++d)
          if (d < beta) {
            if constexpr (OWN_KEYS) {
              ka[d] = ld_key(J, 0, d);
              kb[d] = ld_key(J, 1, d);
            }
            if constexpr (!SHARE_DIGITS) v[d] = ld_digit(J, d);
          }
        if (own >= 0 && J.x2) y1 = kld<CPT>(J.x2 + off);
        if (tensor) {
          x0 = kld<CPT>(J.a0 + off);
          y0 = kld<CPT>(J.b0 + off);
        }
        const bool add_c0 = J.c0 && i < l;
        if (add_c0) c0 = kld<CPT>(J.c0 + off);
        F64Acc sa[CPT], sb[CPT];
        D x1{}, fy1{};
        if (own >= 0 && J.x2) fy1 = kdbl<CPT>(y1);
#pragma unroll
        for (int d = 0; d < MAXB; ++d)
          if (d < beta) {
            D w;
            if constexpr (SHARE_DIGITS)
              w = vd[d];
            else
              w = kdbl<CPT>(v[d]);
            if (d == own && J.x2) {  // the own digit is x * x2 (tensor term a1 b1)
              x1 = w;
#pragma unroll
              for (int c = 0; c < CPT; ++c) w.c[c] = f_mulmod(w.c[c], fy1.c[c], fp.q, fp.qinv);
            }
            D fa, fb;
            if constexpr (OWN_KEYS) {
              fa = kdbl<CPT>(ka[d]);
              fb = kdbl<CPT>(kb[d]);
            } else {
              fa = ka_g[d];
              fb = kb_g[d];
            }
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
              sa[c].mac(w.c[c], fa.c[c]);
              sb[c].mac(w.c[c], fb.c[c]);
            }
          }
        if (tensor) {
          const D fx0 = kdbl<CPT>(x0), fy0 = kdbl<CPT>(y0);
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            const double py0 = f_mulmod(fy0.c[c], fp.pm, fp.q, fp.qinv), py1 = f_mulmod(fy1.c[c], fp.pm, fp.q, fp.qinv);
            sb[c].mac(fx0.c[c], py0);  // + P a0 b0
            sa[c].mac(fx0.c[c], py1);  // + P (a0 b1 + a1 b0)
            sa[c].mac(x1.c[c], py0);
          }
        }
        if (add_c0) {
          const D fc = kdbl<CPT>(c0);
#pragma unroll
          for (int c = 0; c < CPT; ++c) sb[c].mac(fc.c[c], fp.pm);
        }
        uint64_t ra[CPT], rb[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          ra[c] = f_canon(sa[c].fold(fp.w51, fp.q, fp.qinv), fp.q, fp.qinv);
          rb[c] = f_canon(sb[c].fold(fp.w51, fp.q, fp.qinv), fp.q, fp.qinv);
        }
        if (J.c0x) {
          const V cv = kld<CPT>(J.c0x + off);
#pragma unroll
          for (int c = 0; c < CPT; ++c) rb[c] = addmod(rb[c], cv.c[c], q);
        }
        store(J, ra, rb);
      };
      if constexpr (SHARE_DIGITS) {
        D vd[MAXB];  // the group's digit tile (hoisted rotations of one ciphertext), read once
#pragma unroll
        for (int d = 0; d < MAXB; ++d)
          if (d < beta) vd[d] = kdbl<CPT>(ld_digit(J0, d));
#pragma unroll
        for (int jj = 0; jj < JG; ++jj)
          if (jj < gn) run(L.j[g0 + jj], nullptr, nullptr, vd);
      } else if constexpr (OWN_KEYS) {
        run(L.j[g0], nullptr, nullptr, nullptr);
      } else {
        V ka[MAXB], kb[MAXB];
        D da[MAXB], db[MAXB];  // the group's key tile, read once
#pragma unroll
        for (int d = 0; d < MAXB; ++d)
          if (d < beta) {
            ka[d] = ld_key(J0, 0, d);
            kb[d] = ld_key(J0, 1, d);
          }
#pragma unroll
        for (int d = 0; d < MAXB; ++d)
          if (d < beta) {
            da[d] = kdbl<CPT>(ka[d]);
            db[d] = kdbl<CPT>(kb[d]);
          }
#pragma unroll
        for (int jj = 0; jj < JG; ++jj)
          if (jj < gn) run(L.j[g0 + jj], da, db, nullptr);
      }
      return;
    }
  }

  // 128-bit integer sums: larger primes, or any number of digits.
  const DevPrime p = primes[pid];
  auto run = [&](const KskJob& J, const V* ka_g, const V* kb_g, const V* vd) {
    U128 sa[CPT], sb[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) sa[c] = sb[c] = U128{0, 0};
    V x1{}, y1{};  // a1, b1 of this limb (own digit)
    auto digit = [&](int d, V v, const V& a_, const V& b_) {
      if (d == own && J.x2) {  // the own digit is x * x2 (tensor term a1 b1)
        x1 = v;
#pragma unroll
        for (int c = 0; c < CPT; ++c) v.c[c] = mulmod(v.c[c], y1.c[c], p);
      }
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        mac128(sa[c], v.c[c], a_.c[c]);
        mac128(sb[c], v.c[c], b_.c[c]);
      }
    };
    auto tensor_terms = [&](const V& x0, const V& y0) {
      const ShoupConst pm = pmod[i];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const uint64_t py0 = shoup(y0.c[c], pm.w, pm.ws, p.q), py1 = shoup(y1.c[c], pm.w, pm.ws, p.q);
        mac128(sb[c], x0.c[c], py0);  // + P a0 b0
        mac128(sa[c], x0.c[c], py1);  // + P (a0 b1 + a1 b0)
        mac128(sa[c], x1.c[c], py0);
      }
    };
    if constexpr (MAXB > 0) {
      V v[MAXB], ka[MAXB], kb[MAXB];
#pragma unroll
      for (int d = 0; d < MAXB; ++d)
        if (d < beta) {
          if (SHARE_DIGITS) {
            v[d] = vd[d];
            ka[d] = ld_key(J, 0, d);
            kb[d] = ld_key(J, 1, d);
          } else {
            v[d] = ld_digit(J, d);
            ka[d] = ka_g[d];
            kb[d] = kb_g[d];
          }
        }
      if (own >= 0 && J.x2) y1 = kld<CPT>(J.x2 + off);
      V x0{}, y0{};
      if (tensor) {
        x0 = kld<CPT>(J.a0 + off);
        y0 = kld<CPT>(J.b0 + off);
      }
#pragma unroll
      for (int d = 0; d < MAXB; ++d)
        if (d < beta) digit(d, v[d], ka[d], kb[d]);
      if (tensor) tensor_terms(x0, y0);
    } else {
      if (own >= 0 && J.x2) y1 = kld<CPT>(J.x2 + off);
      for (int d = 0; d < beta; ++d) digit(d, ld_digit(J, d), ld_key(J, 0, d), ld_key(J, 1, d));
      if (tensor) {
        // every Q limb has one own digit, so x1 / y1 hold a1 / b1 here
        if (beta > 12) {  // keep the sums below 2^128: at most 15 products of two values < 2^62
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            sa[c] = U128{reduce128(sa[c], p), 0};
            sb[c] = U128{reduce128(sb[c], p), 0};
          }
        }
        tensor_terms(kld<CPT>(J.a0 + off), kld<CPT>(J.b0 + off));
      }
    }
    uint64_t ra[CPT], rb[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      ra[c] = reduce128(sa[c], p);
      rb[c] = reduce128(sb[c], p);
    }
    if (J.c0 && i < l) {
      const ShoupConst pm = pmod[i];
      const V cv = kld<CPT>(J.c0 + off);
#pragma unroll
      for (int c = 0; c < CPT; ++c) rb[c] = addmod(rb[c], shoup(cv.c[c], pm.w, pm.ws, p.q), p.q);
    }
    if (J.c0x) {
      const V cv = kld<CPT>(J.c0x + off);
#pragma unroll
      for (int c = 0; c < CPT; ++c) rb[c] = addmod(rb[c], cv.c[c], p.q);
    }
    store(J, ra, rb);
  };
  if constexpr (MAXB > 0 && SHARE_DIGITS) {
    V vd[MAXB];  // the group's digit tile (hoisted rotations of one ciphertext), read once
#pragma unroll
    for (int d = 0; d < MAXB; ++d)
      if (d < beta) vd[d] = ld_digit(J0, d);
#pragma unroll
    for (int jj = 0; jj < JG; ++jj)
      if (jj < gn) run(L.j[g0 + jj], nullptr, nullptr, vd);
  } else if constexpr (MAXB > 0) {
    V ka[MAXB], kb[MAXB];  // the group's key tile, read once
#pragma unroll
    for (int d = 0; d < MAXB; ++d)
      if (d < beta) {
        ka[d] = ld_key(J0, 0, d);
        kb[d] = ld_key(J0, 1, d);
      }
#pragma unroll
    for (int jj = 0; jj < JG; ++jj)
      if (jj < gn) run(L.j[g0 + jj], ka, kb, nullptr);
  } else {
    for (int jj = 0; jj < gn; ++jj) run(L.j[g0 + jj], nullptr, nullptr, nullptr);
  }
}

__global__ void __launch_bounds__(EW_THREADS) moddown_finish_kernel(const __grid_constant__ FinJobList L,
                                                                    const DevPrime* primes, const ShoupConst* pinv,
                                                                    int logN) {
  const FinJob& J = L.j[blockIdx.z];
  const int j = blockIdx.y;
  if (j >= J.l) return;
  pdl_wait();
  const size_t off = ((size_t)j << logN) + blockIdx.x * blockDim.x + threadIdx.x;
  const DevPrime p = primes[j];
  const ShoupConst pi = pinv[j];
  uint64_t v = shoup(submod(J.x[off], J.conv[off], p.q), pi.w, pi.ws, p.q);
  if (J.add) v = addmod(v, J.add[off], p.q);
  J.out[off] = v;
}

__global__ void __launch_bounds__(EW_THREADS) tensor_kernel(const __grid_constant__ TensorJobList L,
                                                            const DevPrime* primes, int logN) {
  const TensorJob& J = L.j[blockIdx.z];
  const int j = blockIdx.y;
  if (j >= J.l) return;
  pdl_wait();
  const size_t off = ((size_t)j << logN) + blockIdx.x * blockDim.x + threadIdx.x;
  const DevPrime p = primes[j];
  const uint64_t x0 = J.a0[off], x1 = J.a1[off], y0 = J.b0[off], y1 = J.b1[off];
  J.d0[off] = mulmod(x0, y0, p);
  U128 acc{0, 0};
  mac128(acc, x0, y1);
  mac128(acc, x1, y0);
  J.d1[off] = reduce128(acc, p);
  if (J.d2) J.d2[off] = mulmod(x1, y1, p);
}

__global__ void __launch_bounds__(EW_THREADS) switch_kernel(const __grid_constant__ SwitchJobList L,
                                                            const DevPrime* primes, int logN) {
  const SwitchJob& J = L.j[blockIdx.z];
  const int j = blockIdx.y;
  if (j >= J.l - 1) return;
  pdl_wait();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const DevPrime om = primes[J.l - 1], nm = primes[j];
  J.out[((size_t)j << logN) + n] = switch_modulus(J.top[n], om, nm);
}

__global__ void __launch_bounds__(EW_THREADS) rescale_finish_kernel(const __grid_constant__ RescaleJobList L,
                                                                    const DevPrime* primes, const RescaleConst* rs,
                                                                    int logN, int n_q) {
  const RescaleJob& J = L.j[blockIdx.z];
  const int j = blockIdx.y;
  if (j >= J.l - 1) return;
  pdl_wait();
  const size_t off = ((size_t)j << logN) + blockIdx.x * blockDim.x + threadIdx.x;
  const DevPrime p = primes[j];
  const RescaleConst r = rs[(size_t)J.l * n_q + j];
  uint64_t a = shoup(J.x[off], r.qinv, r.qinv_s, p.q);
  uint64_t b = shoup(J.t[off], r.m, r.m_s, p.q);
  J.out[off] = addmod(a, b, p.q);
}

__global__ void __launch_bounds__(EW_THREADS) addsub_kernel(const __grid_constant__ AddSubJobList L,
                                                            const DevPrime* primes, int logN) {
  const AddSubJob& J = L.j[blockIdx.z];
  const int j = blockIdx.y;
  if (j >= J.l) return;
  pdl_wait();
  const size_t off = ((size_t)j << logN) + 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  const DevPrime p = primes[ext_prime(j, J.lq, J.nq)];
  const uint64_t q = p.q;
  const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(J.a + off);
  ulonglong2 y;
  if (J.sub >= EW_MUL_SCALAR) {
    y.x = y.y = J.b[j];
  } else {
    y = *reinterpret_cast<const ulonglong2*>(J.b + off);
  }
  ulonglong2 r;
  switch (J.sub) {
    case EW_SUB:
      r.x = submod(x.x, y.x, q);
      r.y = submod(x.y, y.y, q);
      break;
    case EW_MUL:
    case EW_MUL_SCALAR:
      r.x = mulmod(x.x, y.x, p);
      r.y = mulmod(x.y, y.y, p);
      break;
    default:  // EW_ADD, EW_ADD_SCALAR
      r.x = addmod(x.x, y.x, q);
      r.y = addmod(x.y, y.y, q);
  }
  *reinterpret_cast<ulonglong2*>(J.out + off) = r;
}

__global__ void __launch_bounds__(EW_THREADS) scalar_kernel(const __grid_constant__ ScalarJobList L,
                                                            const DevPrime* primes, int logN) {
  const ScalarJob& J = L.j[blockIdx.z];
  const int j = blockIdx.y;
  if (j >= J.l) return;
  pdl_wait();
  const size_t off = ((size_t)j << logN) + 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  const DevPrime p = primes[j];
  const uint64_t sc = J.s[j];
  const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(J.a + off);
  ulonglong2 r;
  if (J.op == EW_MUL_SCALAR) {
    r.x = mulmod(x.x, sc, p);
    r.y = mulmod(x.y, sc, p);
  } else {
    r.x = addmod(x.x, sc, p.q);
    r.y = addmod(x.y, sc, p.q);
  }
  *reinterpret_cast<ulonglong2*>(J.out + off) = r;
}

// Two adjacent coefficients per thread; sums of up to 15 products (< 2^124 each) stay below
// 2^128 before a reduction.
constexpr int LC_BLOCK = 4;  // terms per block of loads (lincomb_kernel, dot_plain_kernel)

// Memory bounds it, so warps in flight decide: with 114 registers (two CTAs an SM) 11 terms of 24 limbs at
// N = 2^16 took 54.8 us on 50-bit primes and 62 on 55-bit ones, with 80 (three) 39.2 and 51.
__global__ void __launch_bounds__(EW_THREADS, 3)
    dot_plain_kernel(const __grid_constant__ DotJob J, const DevPrime* primes, const F64Prime* f64, int logN) {
  const int lane = blockIdx.x, j = blockIdx.z;
  const int pid = ext_prime(j, J.lq, J.nq);
  const uint64_t q = primes[pid].q;
  const size_t off = ((size_t)j << logN) + 2 * (blockIdx.y * blockDim.x + threadIdx.x);
  pdl_wait();
  auto ld2 = [](const uint64_t* q) { return *reinterpret_cast<const ulonglong2*>(q); };
  ulonglong2 w[LC_BLOCK], x[LC_BLOCK], y[LC_BLOCK];
  auto load = [&](int t0) {  // as lincomb_kernel
#pragma unroll
    for (int u = 0; u < LC_BLOCK; ++u)
      if (t0 + u < J.n) {
        w[u] = ld2(J.pt[t0 + u] + off);
        x[u] = ld2(J.c0[lane][t0 + u] + off);
        y[u] = ld2(J.c1[lane][t0 + u] + off);
      }
  };
  load(0);  // before the form is known: the prime's load would hold these up
  ulonglong2 r0, r1;
  if (q < NTT_F64_MAX) {
    const F64Prime fp = f64[pid];
    F64Sum a0, a1, b0, b1;
    for (int t0 = 0; t0 < J.n; t0 += LC_BLOCK) {
      if (t0) load(t0);
      if (t0 >= 8)  // F64Sum: eight terms, then a block a fold
        a0.flush(fp.w51, fp.q, fp.qinv), a1.flush(fp.w51, fp.q, fp.qinv), b0.flush(fp.w51, fp.q, fp.qinv),
            b1.flush(fp.w51, fp.q, fp.qinv);
#pragma unroll
      for (int u = 0; u < LC_BLOCK; ++u)
        if (t0 + u < J.n) {
          const double w0 = f_from_u64(w[u].x), w1 = f_from_u64(w[u].y);
          a0.mac(w0, f_from_u64(x[u].x));
          a1.mac(w1, f_from_u64(x[u].y));
          b0.mac(w0, f_from_u64(y[u].x));
          b1.mac(w1, f_from_u64(y[u].y));
        }
    }
    r0 = make_ulonglong2(a0.residue(fp.w51, fp.q, fp.qinv), a1.residue(fp.w51, fp.q, fp.qinv));
    r1 = make_ulonglong2(b0.residue(fp.w51, fp.q, fp.qinv), b1.residue(fp.w51, fp.q, fp.qinv));
  } else {
    const DevPrime p = primes[pid];
    U128 a0{0, 0}, a1{0, 0}, b0{0, 0}, b1{0, 0};
    for (int t0 = 0; t0 < J.n; t0 += LC_BLOCK) {
      if (t0 && t0 % 12 == 0) {
        a0 = U128{reduce128(a0, p), 0};
        a1 = U128{reduce128(a1, p), 0};
        b0 = U128{reduce128(b0, p), 0};
        b1 = U128{reduce128(b1, p), 0};
      }
      if (t0) load(t0);
#pragma unroll
      for (int u = 0; u < LC_BLOCK; ++u)
        if (t0 + u < J.n) {
          mac128(a0, w[u].x, x[u].x);
          mac128(a1, w[u].y, x[u].y);
          mac128(b0, w[u].x, y[u].x);
          mac128(b1, w[u].y, y[u].y);
        }
    }
    r0 = make_ulonglong2(reduce128(a0, p), reduce128(a1, p));
    r1 = make_ulonglong2(reduce128(b0, p), reduce128(b1, p));
  }
  *reinterpret_cast<ulonglong2*>(J.out0[lane] + off) = r0;
  *reinterpret_cast<ulonglong2*>(J.out1[lane] + off) = r1;
}

// One CTA per (giant step, lane, coefficient tile, limb): a thread loads its coefficient of the
// lane's baby steps and of the giant step's diagonals in one round of independent loads and
// forms one output pair.  The CTAs of one (tile, limb) are adjacent (giant step fastest, then
// lane), so the other giant steps' reads of a baby-step tile and the other lanes' reads of a
// diagonal tile come from L2: DRAM reads each tile once.  (Looping over the giant steps inside a
// thread exposed one memory latency per giant step: 15 long-scoreboard stalls per issue.)
// NB: register capacity for the baby steps.
template <int NB>
__global__ void __launch_bounds__(EW_THREADS) bsgs_dot_kernel(const __grid_constant__ BsgsJob J,
                                                              const DevPrime* primes, const F64Prime* f64, int logN) {
  const int i = blockIdx.x % J.ng, lane = blockIdx.x / J.ng, j = blockIdx.z;
  const int pid = ext_prime(j, J.lq, J.nq);
  const DevPrime p = primes[pid];
  const size_t off = ((size_t)j << logN) + blockIdx.y * blockDim.x + threadIdx.x;
  pdl_wait();
  uint64_t a[NB], b[NB], w[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if (k < J.nb && J.pt[i][k]) {
      w[k] = J.pt[i][k][off];
      a[k] = J.x0[lane][k][off];
      b[k] = J.x1[lane][k][off];
    }
  if (p.q < NTT_F64_MAX) {
    const F64Prime fp = f64[pid];
    F64Sum s0, s1;
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      if (k == 8 || (k == 15 && k < J.nb)) {
        s0.flush(fp.w51, fp.q, fp.qinv);
        s1.flush(fp.w51, fp.q, fp.qinv);
      }
      if (k < J.nb && J.pt[i][k]) {
        const double d = f_from_u64(w[k]);
        s0.mac(d, f_from_u64(a[k]));
        s1.mac(d, f_from_u64(b[k]));
      }
    }
    J.out0[lane][i][off] = s0.residue(fp.w51, fp.q, fp.qinv);
    J.out1[lane][i][off] = s1.residue(fp.w51, fp.q, fp.qinv);
    return;
  }
  U128 s0{0, 0}, s1{0, 0};
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    if (k == 15) {  // keep the sums below 2^128: at most 15 products of values below 2^62
      s0 = U128{reduce128(s0, p), 0};
      s1 = U128{reduce128(s1, p), 0};
    }
    if (k < J.nb && J.pt[i][k]) {
      mac128(s0, w[k], a[k]);
      mac128(s1, w[k], b[k]);
    }
  }
  J.out0[lane][i][off] = reduce128(s0, p);
  J.out1[lane][i][off] = reduce128(s1, p);
}

// bsgs_dot_kernel with two consecutive coefficients per thread (16-byte loads and stores), for
// at most 8 baby steps (the products stay below 2^128 without an intermediate reduction) and
// operands whose addresses are 16-byte aligned (checked by the launcher).
// Primes below 2^50 sum in FP64 (F64AccPos): 8 baby and 8 giant steps on 30 limbs at N = 2^16 take 331 us
// (1.51 GB), the six transforms of a bootstrap 1360 us against 1770 with 128-bit integer sums.  One CTA
// walking the giant steps with the baby steps in registers took 549 us there.
__global__ void __launch_bounds__(EW_THREADS) bsgs_dot2_kernel(const __grid_constant__ BsgsJob J,
                                                               const DevPrime* primes, const F64Prime* f64, int logN) {
  constexpr int NB = 8;
  const int i = blockIdx.x % J.ng, lane = blockIdx.x / J.ng, j = blockIdx.z;
  const int pid = ext_prime(j, J.lq, J.nq);
  const DevPrime p = primes[pid];
  const size_t off = ((size_t)j << logN) + 2 * ((size_t)blockIdx.y * blockDim.x + threadIdx.x);
  pdl_wait();
  auto ld2 = [](const uint64_t* q) { return *reinterpret_cast<const ulonglong2*>(q); };
  ulonglong2 a[NB], b[NB], w[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if (k < J.nb && J.pt[i][k]) {
      w[k] = ld2(J.pt[i][k] + off);
      a[k] = ld2(J.x0[lane][k] + off);
      b[k] = ld2(J.x1[lane][k] + off);
    }
  if (p.q < NTT_F64_MAX) {
    const F64Prime fp = f64[pid];
    F64AccPos t0x, t0y, t1x, t1y;
#pragma unroll
    for (int k = 0; k < NB; ++k)
      if (k < J.nb && J.pt[i][k]) {
        const double wx = f_from_u64(w[k].x), wy = f_from_u64(w[k].y);
        t0x.mac(wx, f_from_u64(a[k].x));
        t0y.mac(wy, f_from_u64(a[k].y));
        t1x.mac(wx, f_from_u64(b[k].x));
        t1y.mac(wy, f_from_u64(b[k].y));
      }
    auto res = [&](const F64AccPos& t) { return f_canon(t.fold(fp.w51, fp.q, fp.qinv), fp.q, fp.qinv); };
    *reinterpret_cast<ulonglong2*>(J.out0[lane][i] + off) = ulonglong2{res(t0x), res(t0y)};
    *reinterpret_cast<ulonglong2*>(J.out1[lane][i] + off) = ulonglong2{res(t1x), res(t1y)};
    return;
  }
  U128 s0x{0, 0}, s0y{0, 0}, s1x{0, 0}, s1y{0, 0};
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if (k < J.nb && J.pt[i][k]) {
      mac128(s0x, w[k].x, a[k].x);
      mac128(s0y, w[k].y, a[k].y);
      mac128(s1x, w[k].x, b[k].x);
      mac128(s1y, w[k].y, b[k].y);
    }
  *reinterpret_cast<ulonglong2*>(J.out0[lane][i] + off) = ulonglong2{reduce128(s0x, p), reduce128(s0y, p)};
  *reinterpret_cast<ulonglong2*>(J.out1[lane][i] + off) = ulonglong2{reduce128(s1x, p), reduce128(s1y, p)};
}

// As dot_plain_kernel: 78 registers (three CTAs an SM) 41.3 us on 50-bit primes and 50.2 on 55-bit ones for
// 11 terms of 24 limbs, 64 (four) 36.9 and 46.5.
__global__ void __launch_bounds__(EW_THREADS, 4)
    lincomb_kernel(const __grid_constant__ LinCombJob J, const DevPrime* primes, const F64Prime* f64, int logN) {
  const int j = blockIdx.y, lane = blockIdx.z;
  const int pid = ext_prime(j, J.lq, J.nq);
  const uint64_t q = primes[pid].q;
  const size_t off = ((size_t)j << logN) + 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  pdl_wait();
  auto ld2 = [](const uint64_t* q) { return *reinterpret_cast<const ulonglong2*>(q); };
  // terms in blocks of LC_BLOCK whose loads are all issued before their products, so that a
  // thread waits for memory once per block rather than once per term; the 128-bit sums are reduced
  // every 12 terms (below 2^128: a residue plus 12 products of values below 2^62), the FP64 ones every 8
  ulonglong2 x[LC_BLOCK], y[LC_BLOCK];
  auto load = [&](int t0) {
#pragma unroll
    for (int u = 0; u < LC_BLOCK; ++u)
      if (t0 + u < J.n) {
        x[u] = ld2(J.x0[lane][t0 + u] + off);
        y[u] = ld2(J.x1[lane][t0 + u] + off);
      }
  };
  auto store = [&](ulonglong2 r0, ulonglong2 r1) {
    const uint64_t ad = J.add0[j];
    *reinterpret_cast<ulonglong2*>(J.out0[lane] + off) = make_ulonglong2(addmod(r0.x, ad, q), addmod(r0.y, ad, q));
    *reinterpret_cast<ulonglong2*>(J.out1[lane] + off) = r1;
  };
  load(0);  // before the form is known: the prime's load would hold these up
  if (q < NTT_F64_MAX) {
    const F64Prime fp = f64[pid];
    F64Sum a0, a1, b0, b1;
    for (int t0 = 0; t0 < J.n; t0 += LC_BLOCK) {
      if (t0) load(t0);
      if (t0 >= 8)  // F64Sum: eight terms, then a block a fold
        a0.flush(fp.w51, fp.q, fp.qinv), a1.flush(fp.w51, fp.q, fp.qinv), b0.flush(fp.w51, fp.q, fp.qinv),
            b1.flush(fp.w51, fp.q, fp.qinv);
#pragma unroll
      for (int u = 0; u < LC_BLOCK; ++u)
        if (t0 + u < J.n) {
          const double w = f_from_u64(J.s[t0 + u][j]);
          a0.mac(w, f_from_u64(x[u].x));
          a1.mac(w, f_from_u64(x[u].y));
          b0.mac(w, f_from_u64(y[u].x));
          b1.mac(w, f_from_u64(y[u].y));
        }
    }
    store(make_ulonglong2(a0.residue(fp.w51, fp.q, fp.qinv), a1.residue(fp.w51, fp.q, fp.qinv)),
          make_ulonglong2(b0.residue(fp.w51, fp.q, fp.qinv), b1.residue(fp.w51, fp.q, fp.qinv)));
  } else {
    const DevPrime p = primes[pid];
    U128 a0{0, 0}, a1{0, 0}, b0{0, 0}, b1{0, 0};
    for (int t0 = 0; t0 < J.n; t0 += LC_BLOCK) {
      if (t0 && t0 % 12 == 0) {
        a0 = U128{reduce128(a0, p), 0};
        a1 = U128{reduce128(a1, p), 0};
        b0 = U128{reduce128(b0, p), 0};
        b1 = U128{reduce128(b1, p), 0};
      }
      if (t0) load(t0);
#pragma unroll
      for (int u = 0; u < LC_BLOCK; ++u)
        if (t0 + u < J.n) {
          const uint64_t w = J.s[t0 + u][j];
          mac128(a0, w, x[u].x);
          mac128(a1, w, x[u].y);
          mac128(b0, w, y[u].x);
          mac128(b1, w, y[u].y);
        }
    }
    store(make_ulonglong2(reduce128(a0, p), reduce128(a1, p)), make_ulonglong2(reduce128(b0, p), reduce128(b1, p)));
  }
}

template <typename List, typename Job>
int fill(List& L, const Job* jobs, int n) {
  L.n = n;
  std::copy(jobs, jobs + n, L.j);
  return n;
}

}  // namespace

int kernel_binary_version(int device) {
  FIDES_CUDA(cudaSetDevice(device));
  cudaFuncAttributes a{};
  FIDES_CUDA(cudaFuncGetAttributes(&a, addsub_kernel));
  return a.binaryVersion;
}

void launch_conv(Context* c, const ConvJob* jobs, int n, cudaStream_t s) {
  static thread_local ConvJobList L;
  // Tables with a tensor-core form go to the tcgen05 kernel unless the SIMT engine is forced;
  // the rest are grouped by source width so each launch uses one specialised kernel.
  std::vector<ConvJob> tc;
  std::vector<ConvJob> byw[MAX_SRC + 1];
  const bool use_tc = c->conv_engine == CONV_TENSOR || (c->conv_engine == CONV_AUTO && kConvAutoTensor);
  for (int i = 0; i < n; ++i) {
    const ConvTable& t = jobs[i].t;
    if (t.n_src > MAX_SRC || t.n_dst > MAX_DST || t.n_src < 1) throw Error(-1, "basis conversion width out of range");
    if (use_tc && t.tc_b)
      tc.push_back(jobs[i]);
    else
      byw[t.n_src].push_back(jobs[i]);
  }
  if (!tc.empty()) launch_conv_tc(c, tc.data(), (int)tc.size(), s);
  for (int w = 1; w <= MAX_SRC; ++w) {
    const auto& v = byw[w];
    for (size_t off = 0; off < v.size(); off += MAX_CONV_JOBS) {
      int m = (int)std::min<size_t>(MAX_CONV_JOBS, v.size() - off);
      fill(L, v.data() + off, m);
      size_t smem = 0;
      double bytes = 0;
      for (int i = 0; i < m; ++i) {
        const ConvTable& t = L.j[i].t;
        smem = std::max(smem, (size_t)(t.n_src + t.lift) * t.n_dst * 8 + (size_t)t.n_dst * (sizeof(DevPrime) + 4));
        bytes += 8.0 * c->N * (t.n_src + t.n_dst);
      }
      dim3 grid(c->N / (2 * EW_THREADS), m);
      LaunchScope ls(c, s, KK_CONV, bytes);
      switch (w) {
#define FIDES_CONV_CASE(K)                                                                                    \
  case K: {                                                                                                   \
    static bool attr = false;                                                                                 \
    if (!attr) {                                                                                              \
      FIDES_CUDA(cudaFuncSetAttribute(conv_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)); \
      attr = true;                                                                                            \
    }                                                                                                         \
    launch_pdl(conv_kernel<K>, grid, EW_THREADS, smem, s, L, c->d_prime, c->logN);                            \
    break;                                                                                                    \
  }
        FIDES_CONV_CASE(1) FIDES_CONV_CASE(2) FIDES_CONV_CASE(3) FIDES_CONV_CASE(4) FIDES_CONV_CASE(5)
        FIDES_CONV_CASE(6) FIDES_CONV_CASE(7) FIDES_CONV_CASE(8) FIDES_CONV_CASE(9) FIDES_CONV_CASE(10)
        FIDES_CONV_CASE(11) FIDES_CONV_CASE(12) FIDES_CONV_CASE(13) FIDES_CONV_CASE(14) FIDES_CONV_CASE(15)
        FIDES_CONV_CASE(16)
#undef FIDES_CONV_CASE
        default: {
          static bool attr = false;
          if (!attr) {
            FIDES_CUDA(cudaFuncSetAttribute(conv_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
            attr = true;
          }
          launch_pdl(conv_kernel<0>, grid, EW_THREADS, smem, s, L, c->d_prime, c->logN);
        }
      }
    }
  }
}

void launch_dot_plain(Context* c, const DotJob& job, cudaStream_t s) {
  if (job.n < 1 || job.n > MAX_DOT_TERMS) throw Error(-1, "dot product needs 1..32 terms");
  if (job.lanes < 1 || job.lanes > MAX_DOT_LANES) throw Error(-1, "dot product needs 1..8 lanes");
  dim3 grid(job.lanes, c->N / (2 * EW_THREADS), job.l);
  LaunchScope ls(c, s, KK_ELEM, 8.0 * c->N * job.l * (job.n + job.lanes * (2.0 * job.n + 2)));
  launch_pdl(dot_plain_kernel, grid, EW_THREADS, 0, s, job, c->d_prime, c->d_f64, c->logN);
}

void launch_bsgs_dot(Context* c, const BsgsJob& job, cudaStream_t s) {
  if (job.nb < 1 || job.nb > MAX_BSGS_BABY || job.ng < 1 || job.ng > MAX_BSGS_GIANT || job.lanes < 1 ||
      job.lanes > MAX_BSGS_LANES || job.l < 1)
    throw Error(-1, "BSGS inner products need 1..16 baby steps, 1..16 giant steps, 1..8 lanes");
  int terms = 0;
  for (int i = 0; i < job.ng; ++i)
    for (int k = 0; k < job.nb; ++k) terms += job.pt[i][k] != nullptr;
  bool aligned = c->N >= 2 * EW_THREADS;  // the paired form: 16-byte aligned operands, a whole tile of pairs
  auto al = [&](const void* q) { aligned = aligned && (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  for (int i = 0; i < job.ng; ++i)
    for (int k = 0; k < job.nb; ++k)
      if (job.pt[i][k]) al(job.pt[i][k]);
  for (int ln = 0; ln < job.lanes; ++ln) {
    for (int k = 0; k < job.nb; ++k) al(job.x0[ln][k]), al(job.x1[ln][k]);
    for (int i = 0; i < job.ng; ++i) al(job.out0[ln][i]), al(job.out1[ln][i]);
  }
  LaunchScope ls(c, s, KK_ELEM, 8.0 * c->N * job.l * (terms + job.lanes * 2.0 * (job.nb + job.ng)));
  if (job.nb <= 8 && aligned) {
    dim3 grid2(job.lanes * job.ng, c->N / (2 * EW_THREADS), job.l);
    launch_pdl(bsgs_dot2_kernel, grid2, EW_THREADS, 0, s, job, c->d_prime, c->d_f64, c->logN);
    return;
  }
  dim3 grid(job.lanes * job.ng, c->N / EW_THREADS, job.l);
  if (job.nb <= 8)
    launch_pdl(bsgs_dot_kernel<8>, grid, EW_THREADS, 0, s, job, c->d_prime, c->d_f64, c->logN);
  else
    launch_pdl(bsgs_dot_kernel<MAX_BSGS_BABY>, grid, EW_THREADS, 0, s, job, c->d_prime, c->d_f64, c->logN);
}

void launch_lincomb(Context* c, const LinCombJob& job, cudaStream_t s) {
  if (job.n < 1 || job.n > MAX_LC_TERMS || job.l < 1 || job.l > MAX_LC_LIMBS || job.lanes < 1 ||
      job.lanes > MAX_LC_LANES)
    throw Error(-1, "linear combination needs 1..16 terms of 1..64 limbs in 1..8 lanes");
  dim3 grid(c->N / (2 * EW_THREADS), job.l, job.lanes);
  LaunchScope ls(c, s, KK_ELEM, 8.0 * c->N * job.l * job.lanes * (2.0 * job.n + 2));
  launch_pdl(lincomb_kernel, grid, EW_THREADS, 0, s, job, c->d_prime, c->d_f64, c->logN);
}

void launch_ksk(Context* c, const KskJob* jobs, int n, cudaStream_t s) {
  static thread_local KskJobList L;
  for (int off = 0; off < n; off += MAX_KSK_JOBS) {
    int m = std::min(MAX_KSK_JOBS, n - off);
    fill(L, jobs + off, m);
    // groups of consecutive jobs with one key, level and set of extras (a batch under one
    // switching key), or else with one digit set (hoisted rotations of one ciphertext)
    auto same_key = [](const KskJob& a, const KskJob& b) {
      return a.key == b.key && a.l == b.l && a.auto_k == b.auto_k && !a.x2 == !b.x2 && !a.a0 == !b.a0 &&
             !a.c0 == !b.c0 && !a.x == !b.x && !a.c0x == !b.c0x;
    };
    auto same_digits = [](const KskJob& a, const KskJob& b) {
      return a.digits == b.digits && a.x == b.x && a.x2 == b.x2 && a.l == b.l && !a.a0 == !b.a0 && !a.c0 == !b.c0 &&
             !a.c0x == !b.c0x;
    };
    // groups of up to MAX_KSK_GROUP jobs sharing a key, or else sharing a digit tile
    auto group = [&](auto same, int cap) {
      L.ngroups = 0;
      int gm = 1;
      for (int i = 0; i < m;) {
        int k = 1;
        while (i + k < m && k < cap && same(L.j[i], L.j[i + k])) ++k;
        L.gstart[L.ngroups] = (uint8_t)i;
        L.gcount[L.ngroups] = (uint8_t)k;
        ++L.ngroups;
        gm = std::max(gm, k);
        i += k;
      }
      return gm;
    };
    int gmax = group(same_key, MAX_KSK_GROUP);
    bool share_digits = false;
    if (gmax == 1) {
      gmax = group(same_digits, 4);
      share_digits = gmax > 1;
      if (!share_digits) group(same_key, MAX_KSK_GROUP);
    }
    int mx = 0;
    for (int i = 0; i < m; ++i) mx = std::max(mx, L.j[i].l + c->K);
    const int jg = gmax == 1 ? 1 : gmax == 2 ? 2 : 4;
    int maxb = 0;
    for (int i = 0; i < m; ++i) maxb = std::max(maxb, c->beta(L.j[i].l));
    dim3 grid(c->N / (2 * EW_THREADS), mx, L.ngroups);
    // algorithmic bytes: each job's digits, outputs and extra operands, and each group's key once
    double bytes = 0;
    for (int i = 0; i < m; ++i) {
      const int l = L.j[i].l, ext = l + c->K, b = c->beta(l);
      bytes += 8.0 * c->N * ((double)ext * (b + 2) + (L.j[i].c0 ? l : 0) + (L.j[i].a0 ? 2 * l : 0) +
                             (L.j[i].c0x ? ext : 0));
    }
    for (int g = 0; g < L.ngroups; ++g) {
      const int l = L.j[L.gstart[g]].l, b = c->beta(l), ext = l + c->K;
      // the shared tile once per group, the other per job
      bytes += 8.0 * c->N * (share_digits ? (double)b * ext + 2.0 * b * ext * L.gcount[g] - (double)b * ext * L.gcount[g]
                                          : 2.0 * b * ext);
    }
    LaunchScope ls(c, s, KK_KSK, bytes);
    auto go_list = [&](auto kern, const auto& list) {
      launch_pdl(kern, grid, EW_THREADS, 0, s, list, c->d_prime, c->d_pmod, c->d_f64, c->logN, c->n_q, c->K, c->dnum,
                 c->alpha);
    };
    if (jg == 1 && m <= FEW_JOBS && maxb <= 4) {
      static thread_local KskJobListT<FEW_JOBS> few;
      few.n = m;
      few.ngroups = L.ngroups;
      std::copy(L.gstart, L.gstart + L.ngroups, few.gstart);
      std::copy(L.gcount, L.gcount + L.ngroups, few.gcount);
      std::copy(L.j, L.j + m, few.j);
      switch (maxb) {
        case 1: go_list(ksk_kernel<1, 1, 2, FEW_JOBS>, few); break;
        case 2: go_list(ksk_kernel<2, 1, 2, FEW_JOBS>, few); break;
        case 3: go_list(ksk_kernel<3, 1, 2, FEW_JOBS>, few); break;
        default: go_list(ksk_kernel<4, 1, 2, FEW_JOBS>, few);
      }
      continue;
    }
    auto go = [&](auto kern) { go_list(kern, L); };
    // more than four digits: the general kernel (9 to 12 of them would name a shared-digit form of 1 to 4)
    switch (maxb > 4 ? 0 : maxb * 16 + jg + (share_digits ? 128 : 0)) {
#define FIDES_KSK_CASE(B, G)                     \
  case B * 16 + G:                               \
    go(ksk_kernel<B, G, 2, MAX_KSK_JOBS>);       \
    break;                                       \
  case 128 + B * 16 + G:                         \
    go(ksk_kernel<B, G, 2, MAX_KSK_JOBS, true>); \
    break;
      FIDES_KSK_CASE(1, 1) FIDES_KSK_CASE(1, 2) FIDES_KSK_CASE(1, 4)
      FIDES_KSK_CASE(2, 1) FIDES_KSK_CASE(2, 2) FIDES_KSK_CASE(2, 4)
      FIDES_KSK_CASE(3, 1) FIDES_KSK_CASE(3, 2) FIDES_KSK_CASE(3, 4)
      FIDES_KSK_CASE(4, 1) FIDES_KSK_CASE(4, 2) FIDES_KSK_CASE(4, 4)
#undef FIDES_KSK_CASE
      default:
        go(ksk_kernel<0, 1, 2, MAX_KSK_JOBS>);
    }
  }
}

void launch_moddown_finish(Context* c, const FinJob* jobs, int n, cudaStream_t s) {
  static thread_local FinJobList L;
  for (int off = 0; off < n; off += MAX_FIN_JOBS) {
    int m = std::min(MAX_FIN_JOBS, n - off);
    fill(L, jobs + off, m);
    int mx = 0;
    for (int i = 0; i < m; ++i) mx = std::max(mx, L.j[i].l);
    dim3 grid(c->N / EW_THREADS, mx, m);
    double bytes = 0;
    for (int i = 0; i < m; ++i) bytes += 8.0 * c->N * ((L.j[i].add ? 4.0 : 3.0) * L.j[i].l);
    LaunchScope ls(c, s, KK_ELEM, bytes);
    launch_pdl(moddown_finish_kernel, grid, EW_THREADS, 0, s, L, c->d_prime, c->d_pinv, c->logN);
  }
}

void launch_tensor(Context* c, const TensorJob* jobs, int n, cudaStream_t s) {
  static thread_local TensorJobList L;
  for (int off = 0; off < n; off += MAX_TENSOR_JOBS) {
    int m = std::min(MAX_TENSOR_JOBS, n - off);
    fill(L, jobs + off, m);
    int mx = 0;
    for (int i = 0; i < m; ++i) mx = std::max(mx, L.j[i].l);
    dim3 grid(c->N / EW_THREADS, mx, m);
    double bytes = 0;
    for (int i = 0; i < m; ++i) bytes += 8.0 * c->N * ((L.j[i].d2 ? 7.0 : 6.0) * L.j[i].l);
    LaunchScope ls(c, s, KK_ELEM, bytes);
    launch_pdl(tensor_kernel, grid, EW_THREADS, 0, s, L, c->d_prime, c->logN);
  }
}

void launch_switch_modulus(Context* c, const SwitchJob* jobs, int n, cudaStream_t s) {
  static thread_local SwitchJobList L;
  for (int off = 0; off < n; off += MAX_RS_JOBS) {
    int m = std::min(MAX_RS_JOBS, n - off);
    fill(L, jobs + off, m);
    int mx = 1;
    for (int i = 0; i < m; ++i) mx = std::max(mx, L.j[i].l - 1);
    dim3 grid(c->N / EW_THREADS, mx, m);
    double bytes = 0;
    for (int i = 0; i < m; ++i) bytes += 8.0 * c->N * (1.0 + (L.j[i].l - 1));
    LaunchScope ls(c, s, KK_ELEM, bytes);
    launch_pdl(switch_kernel, grid, EW_THREADS, 0, s, L, c->d_prime, c->logN);
  }
}

void launch_rescale_finish(Context* c, const RescaleJob* jobs, int n, cudaStream_t s) {
  static thread_local RescaleJobList L;
  for (int off = 0; off < n; off += MAX_RS_JOBS) {
    int m = std::min(MAX_RS_JOBS, n - off);
    fill(L, jobs + off, m);
    int mx = 1;
    for (int i = 0; i < m; ++i) mx = std::max(mx, L.j[i].l - 1);
    dim3 grid(c->N / EW_THREADS, mx, m);
    double bytes = 0;
    for (int i = 0; i < m; ++i) bytes += 8.0 * c->N * (3.0 * (L.j[i].l - 1));
    LaunchScope ls(c, s, KK_ELEM, bytes);
    launch_pdl(rescale_finish_kernel, grid, EW_THREADS, 0, s, L, c->d_prime, c->d_rescale, c->logN, c->n_q);
  }
}

void launch_addsub(Context* c, const AddSubJob* jobs, int n, cudaStream_t s) {
  static thread_local AddSubJobList L;
  for (int off = 0; off < n; off += MAX_ADDSUB_JOBS) {
    int m = std::min(MAX_ADDSUB_JOBS, n - off);
    fill(L, jobs + off, m);
    int mx = 1;
    double bytes = 0;
    for (int i = 0; i < m; ++i) {
      mx = std::max(mx, L.j[i].l);
      bytes += 8.0 * c->N * 3.0 * L.j[i].l;
    }
    dim3 grid(c->N / (2 * EW_THREADS), mx, m);
    LaunchScope ls(c, s, KK_ELEM, bytes);
    launch_pdl(addsub_kernel, grid, EW_THREADS, 0, s, L, c->d_prime, c->logN);
  }
}

void launch_scalar(Context* c, const ScalarJob* jobs, int n, cudaStream_t s) {
  static thread_local ScalarJobList L;
  for (int off = 0; off < n; off += MAX_SCALAR_JOBS) {
    int m = std::min(MAX_SCALAR_JOBS, n - off);
    fill(L, jobs + off, m);
    int mx = 1;
    double bytes = 0;
    for (int i = 0; i < m; ++i) {
      if (L.j[i].l > MAX_SCALAR_LIMBS) throw Error(-1, "scalar op on more than 64 limbs");
      mx = std::max(mx, L.j[i].l);
      bytes += 8.0 * c->N * 2.0 * L.j[i].l;
    }
    dim3 grid(c->N / (2 * EW_THREADS), mx, m);
    LaunchScope ls(c, s, KK_ELEM, bytes);
    launch_pdl(scalar_kernel, grid, EW_THREADS, 0, s, L, c->d_prime, c->logN);
  }
}

}  // namespace fides
