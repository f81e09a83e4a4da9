// Templates of the NTT pass kernels (see ntt.cuh).  Each ntt_inst_<logN>.cu instantiates
// the passes of one ring dimension so that the variants compile in parallel.
#pragma once
#include <algorithm>

#include "f64arith.cuh"
#include "launch.cuh"
#include "ntt.cuh"

namespace fides {
namespace nttk {

constexpr int COL = 0, ROW = 1;

// Residues per thread, 2^LE (LE = 4: 16, four butterfly stages per register chunk; LE = 3: 8,
// three stages per chunk, one more shared-memory exchange per pass, twice the threads), and
// sub-transforms per CTA (G: 4, 8 or 16) are template parameters of every pass, chosen per
// launch by the context's tables (fides_ctx_autotune).  The butterflies, their pairs and
// twiddles and their order are the same for every LE and G, so the results are identical.

// Asynchronous 16-byte global -> shared copies (cp.async), used to fetch an epilogue operand
// while the butterflies run.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Whether pass PASS of a transform stages its epilogue operand ep0 in shared memory: the
// forward row pass (the last one) with a ModDown / rescale epilogue.  A CTA's rows are one
// contiguous block of ep0, copied with cp.async at the start of the pass.
template <int PASS, bool FWD, int OUT>
struct EpStage {
  static constexpr bool on = PASS == ROW && FWD && (OUT == OUT_MODDOWN || OUT == OUT_MDRS || OUT == OUT_RESCALE);
};

// Twiddle loads carry an L2 evict-last policy: a launch streams hundreds of limbs through L2
// while every limb of one prime re-reads that prime's twiddle table, so the tables should
// outlive the streaming data in L2.
__device__ __forceinline__ uint64_t l2_evict_last_policy() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ ShoupConst ld_tw(const ShoupConst* p, uint64_t pol) {
  uint64_t w, ws;
  asm("ld.global.nc.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;" : "=l"(w), "=l"(ws) : "l"(p), "l"(pol));
  return ShoupConst{w, ws};
}
__device__ __forceinline__ double ld_twf(const double* p, uint64_t pol) {
  double v;
  asm("ld.global.nc.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double2 ld_twf2(const double* p, uint64_t pol) {
  double2 v;
  asm("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(p), "l"(pol));
  return v;
}

// Cooley-Tukey butterfly, Harvey lazy form: x, y in [0, 4q) -> [0, 4q).
__device__ __forceinline__ void ct_bf(uint64_t& x, uint64_t& y, ShoupConst w, uint64_t q, uint64_t q2) {
  uint64_t a = csub(x, q2);
  uint64_t t = shoup_lazy(y, w.w, w.ws, q);
  x = a + t;
  y = a - t + q2;
}

// The same with shoup_lazy4's product t below 4q (q < 2^61): x + t and x - t + 4q, so values grow by
// 4q a stage.
__device__ __forceinline__ void ct_bf4(uint64_t& x, uint64_t& y, ShoupConst w, uint64_t q, uint64_t q4) {
  const uint64_t t = shoup_lazy4(y, w.w, w.ws, q);
  const uint64_t a = x;
  x = a + t;
  y = a - t + q4;
}
// Where a forward chunk brings x back below `cm` before its butterflies (x is below 2 cm there): on
// the chunk's first stage always, on the third with `third`, on the others with `odd`.
struct Lazy4Red {
  uint64_t cm;
  bool third, odd;
};
// q < 2^59: values stay below 32q with one subtraction of 16q a chunk (of at most four stages);
// q < 2^60: below 16q with 8q every second stage; q < 2^61: below 8q with 4q every stage.
__device__ __forceinline__ Lazy4Red lazy4_red(uint64_t q) {
  return Lazy4Red{q < (1ull << 59) ? 16 * q : q < (1ull << 60) ? 8 * q : 4 * q, q >= (1ull << 59), q >= (1ull << 60)};
}

// Gentleman-Sande butterfly with a tracked bound B (a multiple of q, values < B <= 2^63):
// the sum doubles the bound unless `red` (B > 2^62), in which case it is brought back
// below B by one conditional subtraction; the difference path leaves a Shoup product in
// [0, 2q).  With q < 2^62 this degenerates to Harvey's form once B reaches 2q.  With shoup_lazy4
// (q < 2^61) it is in [0, 4q) instead: B starts at 2q there, so that a stage's 2B covers it.
__device__ __forceinline__ void gs_bf(uint64_t& x, uint64_t& y, ShoupConst w, uint64_t q, uint64_t B, bool red) {
  uint64_t s = x + y;
  if (red) s = csub(s, B);
  uint64_t d = x - y + B;
  y = shoup_lazy(d, w.w, w.ws, q);
  x = s;
}

// ---- FP64 butterflies for primes q < 2^50.  The residues are integers held in doubles and the
// twiddles w centred, |w| < q / 2.  Every operation below is exact while |y| <= 4q:
//   * y w = p + e exactly (p = fl(y w), e = fma(y, w, -p));
//   * k = rint(p (1/q)) from one fma with the rounding constant 1.5 2^52 (|y w / q| <= 2q < 2^51);
//     p and 1/q carry one rounding each, so |k - y w / q| <= 1/2 + |y w / q| 2^-52
//     <= 1/2 + |y| / (8q);
//   * p - k q is an integer below 2^53 in magnitude, so fma(-k, q, p) is exact, and so is
//     adding e: r = y w - k q with |r| <= q / 2 + |y| / 8.
// In units of q, a forward stage on values within B leaves B + 1/2 + B/8, or, if it reduces x to
// x - rint(x / q) q first, 1 + B/8.  One reducing stage a chunk of at most four stages (its first)
// keeps every value within 3.8; the last chunk of the transform reduces once more, so that its
// results are within 2, which f_to_canon needs.  An inverse stage on values within B leaves sums
// within 2B and products within 1/2 + B/4; every other stage reduces its sums, so B alternates
// between 1 and 2 (the last stage of an odd row pass reduces too).
// Between the two passes of a transform the doubles are stored as they are (their bits);
// only the last pass writes canonical residues.  The quotient from p needs no second table value
// (w / q), and the centred twiddles' margin saves most reductions: 8.75 (forward) and 9.5 (inverse)
// FP64 operations a butterfly and 8 bytes a twiddle, against 9.5 and 11 with w / q, plus two a
// twiddle where w was recovered from it.  On B200 the FP64 pipe runs this product at ~1.7x the rate
// of the 64-bit integer Shoup product.
// A value |v| < 2q -> its canonical residue in [0, q): v + 2q + 2^52 lies in [2^52, 2^53), where the
// double's low 52 bits are the integer v + 2q.
__device__ __forceinline__ uint64_t f_to_canon(double v, double q2_two52, uint64_t qi) {
  uint64_t u = (uint64_t)__double_as_longlong(__dadd_rn(v, q2_two52)) & ((1ull << 52) - 1);  // v + 2q
  u = u >= 2 * qi ? u - 2 * qi : u;
  return u >= qi ? u - qi : u;
}

struct PassArgs {
  const DevPrime* primes;
  const char* tw;              // twiddle tables of all primes (DevPrime::tw)
  const F64Prime* f64;         // [prime]
  const InvFinal* inv_fin;     // [prime]: the inverse transform's last stage
  const ShoupConst* pinv;      // [Q prime]: P^-1 mod q (OUT_MODDOWN)
  const RescaleConst* rescale; // [level][Q prime] (OUT_RESCALE, OUT_MDRS)
  const ShoupConst* pmod;      // [Q prime]: P mod q (IN_CONV_SW)
  const ShoupConst* pqinv;     // [level][Q prime]: (P q_(level-1))^-1 mod q (OUT_MDRS)
  int logN;
  int log1;  // size of the column sub-transform
  int n_q;
  bool wide;  // most of the limbs are of primes above 2^50
};

// Element index u of register r for thread t, when the register index spans bits
// [lo, lo + LE) of u.
template <int LO, int LE>
__device__ __forceinline__ int u_of(int t, int r) {
  // disjoint bit fields: '+' lets the compiler fold the register-index part into offsets
  return ((t >> LO) << (LO + LE)) + (r << LO) + (t & ((1 << LO) - 1));
}

template <int LE>
__device__ __forceinline__ int padu(int u) {
  return u + (u >> LE);
}

// Butterflies of pair bits [BLO, BHI] (in u) for a thread whose registers span bits
// [LO, LO + LE).  FWD walks bits high -> low, inverse low -> high.  tw: the chunk's twiddles of
// this thread (SLOTS heaps interleaved, see ntt.cuh).
template <int LE, int LOGP, int LO, int BHI, int BLO, int SLOTS, bool FWD, int PASS, bool LAZY4>
__device__ __forceinline__ void run_chunk(uint64_t (&x)[1 << LE], const ShoupConst* tw, const DevPrime& pr,
                                          const InvFinal& fin, uint64_t& B, uint64_t pol) {
  constexpr int E = 1 << LE;
  const Lazy4Red lr4 = lazy4_red(pr.q);
#pragma unroll
  for (int k = 0; k <= BHI - BLO; ++k) {
    const int b = FWD ? (BHI - k) : (BLO + k);
    const int rb = b - LO;
    const int H = E >> (rb + 1);  // twiddles of this stage
    const bool red = !FWD && B > (1ull << 62);
    if (FWD && LAZY4 && (k == 0 || (k == 2 ? lr4.third : lr4.odd))) {
#pragma unroll
      for (int r = 0; r < E; ++r)
        if (!(r >> rb & 1)) x[r] = csub(x[r], lr4.cm);
    }
#pragma unroll
    for (int hi = 0; hi < H; ++hi) {
      if (!FWD && PASS == COL && b == LOGP - 1) {
        // last inverse stage (global stage 0): fold N^-1 (times the limb's factor) into both outputs
#pragma unroll
        for (int lr = 0; lr < (1 << rb); ++lr) {
          const int r0 = (hi << (rb + 1)) | lr, r1 = r0 | (1 << rb);
          uint64_t a = x[r0], c = x[r1];
          x[r0] = shoup(a + c, fin.sum.w, fin.sum.ws, pr.q);
          x[r1] = shoup(a - c + B, fin.diff.w, fin.diff.ws, pr.q);
        }
      } else {
        const ShoupConst w = ld_tw(tw + (H + hi) * SLOTS, pol);
#pragma unroll
        for (int lr = 0; lr < (1 << rb); ++lr) {
          const int r0 = (hi << (rb + 1)) | lr, r1 = r0 | (1 << rb);
          if (FWD && LAZY4)
            ct_bf4(x[r0], x[r1], w, pr.q, 2 * pr.q2);
          else if (FWD)
            ct_bf(x[r0], x[r1], w, pr.q, pr.q2);
          else if (LAZY4) {
            const uint64_t sum = x[r0] + x[r1];
            x[r1] = shoup_lazy4(x[r0] - x[r1] + B, w.w, w.ws, pr.q);
            x[r0] = red ? csub(sum, B) : sum;
          } else
            gs_bf(x[r0], x[r1], w, pr.q, B, red);
        }
      }
    }
    if (!FWD && !red) B <<= 1;
  }
}

// run_chunk on FP64 residues (q < 2^50): the same stages, pairs and twiddles.
template <int LE, int LOGP, int LO, int BHI, int BLO, int SLOTS, bool FWD, int PASS>
__device__ __forceinline__ void run_chunk_f64(double (&x)[1 << LE], const double* tw, const F64Prime& fp,
                                              const InvFinal& fin, uint64_t pol) {
  constexpr int E = 1 << LE, NS = BHI - BLO + 1;
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    const int b = FWD ? (BHI - k) : (BLO + k);
    const int rb = b - LO;
    const int H = E >> (rb + 1);
    // forward: the chunk's first stage, and the last but one of the transform's last chunk (the
    // second where that is the first); inverse: every second stage of the pass, and a row pass's last
    const bool red = FWD ? (k == 0 || (PASS == ROW && BLO == 0 && NS >= 2 && k == (NS > 2 ? NS - 2 : 1)))
                         : ((b & 1) || (PASS == ROW && b == LOGP - 1));
    double2 w{};
#pragma unroll
    for (int hi = 0; hi < H; ++hi) {
      if (!FWD && PASS == COL && b == LOGP - 1) {
#pragma unroll
        for (int lr = 0; lr < (1 << rb); ++lr) {
          const int r0 = (hi << (rb + 1)) | lr, r1 = r0 | (1 << rb);
          const double a = x[r0], c = x[r1];
          x[r0] = f_mulmod(__dadd_rn(a, c), fin.fsum, fp.q, fp.qinv);
          x[r1] = f_mulmod(__dsub_rn(a, c), fin.fdiff, fp.q, fp.qinv);
        }
      } else {
        if (H == 1)
          w.x = ld_twf(tw + 1, pol);
        else if (hi & 1)
          w.x = w.y;
        else
          w = ld_twf2(tw + (H + hi) * SLOTS, pol);
#pragma unroll
        for (int lr = 0; lr < (1 << rb); ++lr) {
          const int r0 = (hi << (rb + 1)) | lr, r1 = r0 | (1 << rb);
          if (FWD) {
            const double a = red ? f_reduce(x[r0], fp.q, fp.qinv) : x[r0];
            const double r = f_mulmod(x[r1], w.x, fp.q, fp.qinv);
            x[r0] = __dadd_rn(a, r);
            x[r1] = __dsub_rn(a, r);
          } else {
            const double a = x[r0], c = x[r1], sum = __dadd_rn(a, c);
            x[r0] = red ? f_reduce(sum, fp.q, fp.qinv) : sum;
            x[r1] = f_mulmod(__dsub_rn(a, c), w.x, fp.q, fp.qinv);
          }
        }
      }
    }
  }
}

// Bound of the inverse transform's values after `stages` stages from the bound B of its input.
__device__ __forceinline__ uint64_t inv_bound(uint64_t B, int stages) {
  for (int i = 0; i < stages; ++i)
    if (B <= (1ull << 62)) B <<= 1;
  return B;
}



// Register span and twiddles of chunk c.
template <int LE, int LOGP, bool FWD, int C>
struct Chunk {
  static constexpr int BHI = tw_bhi(LOGP, FWD, LE, C), BLO = tw_blo(LOGP, FWD, LE, C);
  static constexpr int LO = tw_lo(LOGP, FWD, LE, C);
  static constexpr int SLOTS = tw_slots(LOGP, FWD, LE, C), OFF = tw_off(LOGP, FWD, LE, C);
};

template <int LE, int LOGP, int PASS, bool FWD, bool LAZY4, typename CH>
__device__ __forceinline__ void one_chunk(uint64_t (&x)[1 << LE], CH, int t, const ShoupConst* tw, const DevPrime& pr,
                                          const InvFinal& fin, uint64_t& B, uint64_t pol) {
  run_chunk<LE, LOGP, CH::LO, CH::BHI, CH::BLO, CH::SLOTS, FWD, PASS, LAZY4>(x, tw + CH::OFF + (t >> CH::LO), pr, fin,
                                                                             B, pol);
}
template <int LE, int LOGP, int PASS, bool FWD, typename CH>
__device__ __forceinline__ void one_chunk_f64(double (&x)[1 << LE], CH, int t, const double* tw, const F64Prime& fp,
                                              const InvFinal& fin, uint64_t pol) {
  run_chunk_f64<LE, LOGP, CH::LO, CH::BHI, CH::BLO, CH::SLOTS, FWD, PASS>(x, tw + CH::OFF + 2 * (t >> CH::LO), fp, fin, pol);
}

// Barrier between a pass's shared-memory exchanges: of the CTA, or of the warp where every
// sub-transform lies within one (WARP).
template <bool WARP>
__device__ __forceinline__ void pass_sync() {
  if constexpr (WARP)
    __syncwarp();
  else
    __syncthreads();
}

// The register chunks of one pass, separated by shared-memory exchanges.
template <int LE, int LOGP, int PASS, bool FWD, bool LAZY4, bool WARP, typename SIDX>
__device__ __forceinline__ void chunks(uint64_t (&x)[1 << LE], uint64_t* sm, SIDX sidx, int g, int t,
                                       const ShoupConst* tw, const DevPrime& pr, const InvFinal& fin, uint64_t& B,
                                       bool direct_load, uint64_t pol) {
  constexpr int E = 1 << LE;
  constexpr int NCH = (LOGP + LE - 1) / LE;
  using C0 = Chunk<LE, LOGP, FWD, 0>;
  one_chunk<LE, LOGP, PASS, FWD, LAZY4>(x, C0{}, t, tw, pr, fin, B, pol);
  if constexpr (NCH > 1) {
    using C1 = Chunk<LE, LOGP, FWD, 1>;
    if (!direct_load) pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) sm[sidx(g, u_of<C0::LO, LE>(t, r))] = x[r];
    pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) x[r] = sm[sidx(g, u_of<C1::LO, LE>(t, r))];
    one_chunk<LE, LOGP, PASS, FWD, LAZY4>(x, C1{}, t, tw, pr, fin, B, pol);
  }
  if constexpr (NCH > 2) {
    using C1 = Chunk<LE, LOGP, FWD, 1>;
    using C2 = Chunk<LE, LOGP, FWD, 2>;
    pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) sm[sidx(g, u_of<C1::LO, LE>(t, r))] = x[r];
    pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) x[r] = sm[sidx(g, u_of<C2::LO, LE>(t, r))];
    one_chunk<LE, LOGP, PASS, FWD, LAZY4>(x, C2{}, t, tw, pr, fin, B, pol);
  }
  static_assert(NCH <= 3, "sub-transform too large");
}

// chunks() on FP64 residues; the shared-memory exchanges move the doubles' bits.
template <int LE, int LOGP, int PASS, bool FWD, bool WARP, typename SIDX>
__device__ __forceinline__ void chunks_f64(double (&x)[1 << LE], uint64_t* smu, SIDX sidx, int g, int t,
                                           const double* tw, const F64Prime& fp, const InvFinal& fin, bool direct_load,
                                           uint64_t pol) {
  constexpr int E = 1 << LE;
  constexpr int NCH = (LOGP + LE - 1) / LE;
  double* sm = reinterpret_cast<double*>(smu);
  using C0 = Chunk<LE, LOGP, FWD, 0>;
  one_chunk_f64<LE, LOGP, PASS, FWD>(x, C0{}, t, tw, fp, fin, pol);
  if constexpr (NCH > 1) {
    using C1 = Chunk<LE, LOGP, FWD, 1>;
    if (!direct_load) pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) sm[sidx(g, u_of<C0::LO, LE>(t, r))] = x[r];
    pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) x[r] = sm[sidx(g, u_of<C1::LO, LE>(t, r))];
    one_chunk_f64<LE, LOGP, PASS, FWD>(x, C1{}, t, tw, fp, fin, pol);
  }
  if constexpr (NCH > 2) {
    using C1 = Chunk<LE, LOGP, FWD, 1>;
    using C2 = Chunk<LE, LOGP, FWD, 2>;
    pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) sm[sidx(g, u_of<C1::LO, LE>(t, r))] = x[r];
    pass_sync<WARP>();
#pragma unroll
    for (int r = 0; r < E; ++r) x[r] = sm[sidx(g, u_of<C2::LO, LE>(t, r))];
    one_chunk_f64<LE, LOGP, PASS, FWD>(x, C2{}, t, tw, fp, fin, pol);
  }
}

template <int LOGN, int PASS>
struct PassShape {
  static constexpr int LOG1 = (LOGN + 1) / 2, LOG2 = LOGN / 2;
  static constexpr int LOGP = PASS == COL ? LOG1 : LOG2;
};

// One pass of a transform of 2^LOGN points.  Every index is a compile-time function of
// LOGN, so global and shared addresses are a per-thread base plus immediate offsets.
// Threads of a pass CTA, and CTAs per SM the register budget is sized for: with 16 residues
// per thread 768 threads = 24 warps per SM, i.e. 80 registers (FIDES_NTT_THREADS_PER_SM
// overrides it); with 8, 1024 threads = 32 warps, 64 registers (no spills in the plain passes).
#ifndef FIDES_NTT_THREADS_PER_SM
#define FIDES_NTT_THREADS_PER_SM 768
#endif
template <int LOGN, int PASS, int G, int LE>
struct PassThreads {
  static constexpr int TPS = LE == 3 ? 1024 : FIDES_NTT_THREADS_PER_SM;
  static constexpr int NT = (1 << (PassShape<LOGN, PASS>::LOGP - LE)) * G;
  static constexpr int MINB = NT >= TPS ? 1 : (TPS / NT > 32 ? 32 : TPS / NT);
};

template <int LOGN, int PASS, bool FWD, int IN, int OUT, int G, int LE, typename List>
__global__ void __launch_bounds__(PassThreads<LOGN, PASS, G, LE>::NT, PassThreads<LOGN, PASS, G, LE>::MINB)
    ntt_pass(const PassArgs a, const __grid_constant__ List L) {
  constexpr int LOGP = PassShape<LOGN, PASS>::LOGP;
  constexpr int P = 1 << LOGP, E = 1 << LE, T = P / E, NT = T * G;
  constexpr int NCH = (LOGP + LE - 1) / LE;
  constexpr int PADP = P + P / E;
  extern __shared__ uint64_t sm[];

  constexpr int N = 1 << LOGN;
  LimbRef lr;
  {
    const LimbRun& R = L.run[L.run_of[blockIdx.y]];
    const int k = (int)blockIdx.y - R.first;
    const size_t at = (size_t)k * N;
    lr.ptr = R.ptr + at;
    lr.src = R.src ? R.src + at : nullptr;
    lr.pro = R.pro_step ? R.pro + at : R.pro;
    lr.ep0 = R.ep0 + at;
    lr.ep1 = R.ep1 ? R.ep1 + at : nullptr;
    lr.prime = R.prime + k;
    lr.aux = R.aux;
    lr.fin = R.fin ? R.fin + k : nullptr;
  }
  const DevPrime pr = a.primes[lr.prime];
  const char* tw_prime = a.tw + pr.tw;  // this prime's twiddle tables
  InvFinal fin{};
  if (!FWD && PASS == COL) fin = *(lr.fin ? lr.fin : a.inv_fin + lr.prime);
  uint64_t* data = lr.ptr;
  const int tid = threadIdx.x;
  int g, t;
  if (PASS == COL) {
    g = tid % G;
    t = tid / G;
  } else {
    t = tid % T;
    g = tid / T;
  }
  constexpr int S = N >> LOGP;  // stride of a column (COL) / number of rows (ROW)
  const int sub0 = blockIdx.x * G;
  const int sub = sub0 + g;
  // entry of the pass's (column) or the row's first twiddle
  const size_t tw0 = tw_start(LOGN, FWD, LE) +
                     (PASS == COL ? 0 : tw_sub(PassShape<LOGN, COL>::LOGP, FWD, LE) +
                                            (size_t)sub * tw_sub(LOGP, FWD, LE));

  auto gidx = [&](int s_, int u) -> int { return PASS == COL ? s_ + u * S : s_ * P + u; };
  // shared-memory index of element u of sub-transform gg.  One element (a row of G in a column
  // pass) of padding after every E: the threads of a half-warp read elements E apart in the next
  // chunk, which without it fall on the same banks (1.25 M conflicts in a column pass on 300 limbs)
  auto sidx = [&](int gg, int u) -> int { return PASS == COL ? padu<LE>(u) * G + gg : gg * PADP + padu<LE>(u); };
  // A row pass whose rows lie within a warp (T <= 32) exchanges, stages its loads and stores and
  // fetches its epilogue operand warp by warp: element k of thread tid is e = k WT + lane of the
  // warp's WT E elements.  Its warps then never wait for one another, so that one loads while
  // others compute.
  constexpr bool WARP = PASS == ROW && T <= 32;
  constexpr int WT = WARP && NT > 32 ? 32 : NT;  // threads that share a staged block
  const int blk = WARP ? tid / WT : 0, lane = tid % WT;

  uint64_t x[E];  // residues, or the bits of FP64 ones
  const bool f64 = pr.q < NTT_F64_MAX;  // uniform per CTA: one limb per CTA
  F64Prime fp{};
  if (f64) fp = a.f64[lr.prime];

  // ---- input of this pass: the first pass applies the prologue
  constexpr bool first_pass = FWD ? (PASS == COL) : (PASS == ROW);
  const uint64_t* in = (first_pass && lr.src) ? lr.src : data;
  DevPrime opr;
  if (IN == IN_SWITCH || IN == IN_CONV_SW) opr = a.primes[lr.aux - 1];
  ShoupConst pm{0, 0};
  if (IN == IN_CONV_SW) pm = a.pmod[lr.prime];
  auto load = [&](size_t i) -> uint64_t {
    if (first_pass && IN == IN_SWITCH) return switch_modulus(lr.pro[i], opr, pr);
    if (first_pass && IN == IN_SIGNED) return signed_mod(lr.pro[i], pr);
    if (first_pass && IN == IN_MUL) return mulmod(in[i], lr.pro[i], pr);
    if (first_pass && IN == IN_CONV_SW) return in[i];  // + P SwitchModulus(top) below
    return in[i];
  };
  // The prologues and epilogues of FP64 limbs are FP64 products too: with the butterflies at 8.75-9.5
  // operations that pipe has room, and a 64-bit integer product with its reduction takes the FMA-heavy
  // pipe four times as long.  An input need not be canonical: the first forward stage takes values
  // within 4q, the first inverse stage within q.  A top limb of a larger prime is switched in integers.
  const bool fp_switch = (IN == IN_SWITCH || IN == IN_CONV_SW) && opr.q < NTT_F64_MAX;
  auto centred_top = [&](uint64_t v) -> double {  // SwitchModulus: the centred lift, |.| <= 2^49
    const double t = f_from_u64(v);
    return v > (opr.q >> 1) ? __dadd_rn(t, -(double)(long long)opr.q) : t;
  };
  auto bits = [](double v) { return (uint64_t)__double_as_longlong(v); };
  // a signed 64-bit integer: its upper word times 2^32, reduced, plus its lower one (below q / 2)
  const bool fp_signed = IN == IN_SIGNED && pr.q >= (1ull << 33);
  auto signed_f64 = [&](uint64_t v) -> double {
    const double hi = __dadd_rn(__hiloint2double(0x45300000, (int)((uint32_t)(v >> 32) ^ 0x80000000u)),
                                -(0x1p84 + 0x1p63));
    const double lo = __dadd_rn(__hiloint2double(0x43300000, (int)(uint32_t)v), -F64_TWO52);
    return __dadd_rn(f_reduce(hi, fp.q, fp.qinv), lo);
  };
  auto load_f64 = [&](size_t i) -> uint64_t {
    if (!first_pass) return in[i];  // the first pass's doubles
    if (IN == IN_MUL) return bits(f_mulmod(f_from_u64(in[i]), f_from_u64(lr.pro[i]), fp.q, fp.qinv));  // within 3q/4
    return bits(f_from_u64(load(i)));
  };

  // ---- load chunk 0 (direct when lanes map to consecutive addresses, else staged)
  constexpr int LO0 = Chunk<LE, LOGP, FWD, 0>::LO;
  constexpr bool direct_load = (PASS == COL) || (LO0 == LOGP - LE);
  // conv + P SwitchModulus(top) (a column pass): the tile of the top limb is copied into the
  // exchange buffer by cp.async while the conv loads are in flight, so the prologue waits for
  // memory once (loading both operands per element serialised the loads: long-scoreboard
  // stalls 10x a plain pass's)
  constexpr bool STAGE_PRO = first_pass && IN == IN_CONV_SW;
  static_assert(!STAGE_PRO || PASS == COL, "the conv-switch prologue is a column-pass prologue");
  pdl_wait();  // nothing before this reads or writes limbs
  if constexpr (STAGE_PRO) {
#pragma unroll
    for (int k = 0; k < G * P / 2 / NT; ++k) {
      const int c = k * NT + tid, u = c / (G / 2), h = c % (G / 2);
      cp_async16(sm + padu<LE>(u) * G + 2 * h, lr.pro + (size_t)u * S + sub0 + 2 * h);
    }
    cp_async_commit();
  }
  auto fill = [&](auto ld) {
    if constexpr (direct_load) {
#pragma unroll
      for (int r = 0; r < E; ++r) x[r] = ld(gidx(sub, u_of<LO0, LE>(t, r)));
    } else {
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const int e = k * WT + lane;
        const int gg = blk * (WT / T) + e / P, u = e % P;
        sm[sidx(gg, u)] = ld(gidx(sub0 + gg, u));
      }
      pass_sync<WARP>();
#pragma unroll
      for (int r = 0; r < E; ++r) x[r] = sm[sidx(g, u_of<LO0, LE>(t, r))];
    }
  };

  // ---- epilogue operand: start fetching it into shared memory (after the data region)
  constexpr bool EPS = EpStage<PASS, FWD, OUT>::on;
  uint64_t* sep = sm + G * PADP;
  auto fetch_epilogue = [&] {
    if constexpr (EPS) {
      const uint64_t* e0 = lr.ep0 + (size_t)sub0 * P;
#pragma unroll
      for (int k = 0; k < E / 2; ++k) {
        const int at = blk * (WT * E) + 2 * (k * WT + lane);
        cp_async16(sep + at, e0 + at);
      }
      cp_async_commit();
    }
  };

  // ---- store (the last pass applies the epilogue)
  constexpr bool last_pass = !first_pass;
  ShoupConst pinv{0, 0};
  RescaleConst rsc{0, 0, 0, 0};
  if (OUT == OUT_MODDOWN) pinv = a.pinv[lr.prime];
  if (OUT == OUT_MDRS) pinv = a.pqinv[(size_t)lr.aux * a.n_q + lr.prime];
  if (OUT == OUT_RESCALE) rsc = a.rescale[(size_t)lr.aux * a.n_q + lr.prime];
  auto ep0 = [&](size_t i) -> uint64_t {
    if constexpr (EPS) return sep[i - (size_t)sub0 * P];
    return lr.ep0[i];
  };
  auto finish = [&](size_t i, uint64_t v, uint64_t e0) {
    if (OUT == OUT_MODDOWN || OUT == OUT_MDRS) {
      v = shoup(submod(e0, v, pr.q), pinv.w, pinv.ws, pr.q);
      if (OUT == OUT_MODDOWN && lr.ep1) v = addmod(v, lr.ep1[i], pr.q);
    } else if (OUT == OUT_RESCALE) {  // v: any 64 bits, not reduced yet
      v = addmod(shoup(e0, rsc.qinv, rsc.qinv_s, pr.q), shoup(v, rsc.m, rsc.m_s, pr.q), pr.q);
    }
    data[i] = v;
  };
  // the same on a transform's FP64 result, within 2q; every epilogue leaves less than 2q
  auto centred = [&](uint64_t w) -> double {
    const double d = f_from_u64(w);
    return w > (pr.q >> 1) ? __dadd_rn(d, -fp.q) : d;
  };
  double f_pinv = 0, f_qinv = 0, f_m = 0, f_q2t = 0;
  if (f64) {
    if (OUT == OUT_MODDOWN || OUT == OUT_MDRS) f_pinv = centred(pinv.w);
    if (OUT == OUT_RESCALE) f_qinv = centred(rsc.qinv), f_m = centred(rsc.m);
    f_q2t = __dadd_rn(2.0 * fp.q, F64_TWO52);
  }
  auto finish_f64 = [&](size_t i, uint64_t b, uint64_t e0) {
    if (!last_pass) {
      data[i] = b;
      return;
    }
    double v = __longlong_as_double((long long)b);
    if (OUT == OUT_MODDOWN || OUT == OUT_MDRS) {
      v = f_mulmod(__dsub_rn(f_from_u64(e0), v), f_pinv, fp.q, fp.qinv);  // |e0 - v| < 3q: within 0.875q
      if (OUT == OUT_MODDOWN && lr.ep1) v = __dadd_rn(v, f_from_u64(lr.ep1[i]));
    } else if (OUT == OUT_RESCALE) {
      v = __dadd_rn(f_mulmod(f_from_u64(e0), f_qinv, fp.q, fp.qinv), f_mulmod(v, f_m, fp.q, fp.qinv));
    }
    data[i] = f_to_canon(v, f_q2t, pr.q);
  };
  constexpr int LOL = Chunk<LE, LOGP, FWD, NCH - 1>::LO;
  constexpr bool direct_store = (PASS == COL) || (LOL == LOGP - LE);
  auto drain = [&](auto st) {
    if constexpr (EPS) {
      cp_async_wait_all();
      if (direct_store) pass_sync<WARP>();  // the staged store below synchronises anyway
    }
    if constexpr (direct_store) {
#pragma unroll
      for (int r = 0; r < E; ++r) {
        const size_t i = gidx(sub, u_of<LOL, LE>(t, r));
        st(i, x[r], OUT == OUT_PLAIN ? 0 : ep0(i));
      }
    } else {
      pass_sync<WARP>();
#pragma unroll
      for (int r = 0; r < E; ++r) sm[sidx(g, u_of<LOL, LE>(t, r))] = x[r];
      pass_sync<WARP>();
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const int e = k * WT + lane;
        const int gg = blk * (WT / T) + e / P, u = e % P;
        const size_t i = gidx(sub0 + gg, u);
        st(i, sm[sidx(gg, u)], OUT == OUT_PLAIN ? 0 : ep0(i));
      }
    }
  };

  const uint64_t pol = l2_evict_last_policy();
  if (f64) {
    if (first_pass && IN == IN_SIGNED && fp_signed)
      fill([&](size_t i) { return bits(signed_f64(lr.pro[i])); });
    else if (first_pass && IN == IN_SWITCH && fp_switch)
      fill([&](size_t i) { return bits(f_reduce(centred_top(lr.pro[i]), fp.q, fp.qinv)); });
    else
      fill(load_f64);
    fetch_epilogue();
    if constexpr (STAGE_PRO) {
      cp_async_wait_all();
      __syncthreads();
      auto add_top = [&](auto lift) {
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const double c = lift(sm[sidx(g, u_of<LO0, LE>(t, r))]);
          x[r] = bits(__dadd_rn(__longlong_as_double((long long)x[r]), f_mulmod(c, fp.pm, fp.q, fp.qinv)));
        }
      };
      if (fp_switch)
        add_top(centred_top);
      else
        add_top([&](uint64_t v) { return f_from_u64(switch_modulus(v, opr, pr)); });
    }
    double xf[E];
#pragma unroll
    for (int r = 0; r < E; ++r) xf[r] = __longlong_as_double((long long)x[r]);
    chunks_f64<LE, LOGP, PASS, FWD, WARP>(xf, sm, sidx, g, t, reinterpret_cast<const double*>(tw_prime) + tw0, fp,
                                          fin, direct_load && !STAGE_PRO, pol);
#pragma unroll
    for (int r = 0; r < E; ++r) x[r] = bits(xf[r]);
    drain(finish_f64);
    return;
  }
  fill(load);
  fetch_epilogue();
  if constexpr (STAGE_PRO) {
    cp_async_wait_all();
    __syncthreads();
#pragma unroll
    for (int r = 0; r < E; ++r)
      x[r] = addmod(x[r], shoup(switch_modulus(sm[sidx(g, u_of<LO0, LE>(t, r))], opr, pr), pm.w, pm.ws, pr.q), pr.q);
  }
  const ShoupConst* tw = reinterpret_cast<const ShoupConst*>(tw_prime) + tw0;
  const bool lazy4 = pr.q < (1ull << 61);
  uint64_t B = lazy4 ? pr.q2 : pr.q;  // inverse: bound of the values (a multiple of q)
  if (!FWD && PASS == COL) B = inv_bound(B, PassShape<LOGN, ROW>::LOGP);
  if (lazy4)
    chunks<LE, LOGP, PASS, FWD, true, WARP>(x, sm, sidx, g, t, tw, pr, fin, B, direct_load && !STAGE_PRO, pol);
  else
    chunks<LE, LOGP, PASS, FWD, false, WARP>(x, sm, sidx, g, t, tw, pr, fin, B, direct_load && !STAGE_PRO, pol);

  // ---- final reduction of the completed transform (the rescale's products take its place)
  if (FWD && PASS == ROW && OUT != OUT_RESCALE) {
    if (lazy4) {
#pragma unroll
      for (int r = 0; r < E; ++r) x[r] = shoup(x[r], 1, pr.one_s, pr.q);  // any 64-bit x
    } else {
#pragma unroll
      for (int r = 0; r < E; ++r) x[r] = csub(csub(x[r], pr.q2), pr.q);   // x < 4q
    }
  }
  drain(finish);
}


template <int LOGN, int PASS, bool FWD, int IN, int OUT, int G, int LE, typename List>
void launch_pass_g(Context* c, const PassArgs& a, const List& L, cudaStream_t s) {
  constexpr int LOGP = PassShape<LOGN, PASS>::LOGP;
  constexpr int P = 1 << LOGP, T = P / (1 << LE);
  constexpr int smem = G * (P + P / (1 << LE)) * (int)sizeof(uint64_t) +
                       (EpStage<PASS, FWD, OUT>::on ? G * P * (int)sizeof(uint64_t) : 0);
  static bool attr_set = false;  // per instantiation; set before first launch
  if (!attr_set) {
    FIDES_CUDA(cudaFuncSetAttribute(ntt_pass<LOGN, PASS, FWD, IN, OUT, G, LE, List>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set = true;
  }
  dim3 grid(((1 << LOGN) >> LOGP) / G, L.n);
  // algorithmic bytes: half of a transform's read + write of each limb (two passes)
  LaunchScope ls(c, s, KK_NTT, 8.0 * (1 << LOGN) * L.n);
  launch_pdl(ntt_pass<LOGN, PASS, FWD, IN, OUT, G, LE, List>, grid, T * G, smem, s, a, L);
}

// The pass with the sub-transforms-per-CTA and residues per thread the context's tables pick
// for this launch.
template <int LOGN, int PASS, bool FWD, int IN, int OUT, int LE, typename List>
void launch_pass_le(Context* c, const PassArgs& a, const List& L, cudaStream_t s) {
  switch (c->ntt_shape(!FWD, PASS, L.n)) {
    case 4: launch_pass_g<LOGN, PASS, FWD, IN, OUT, 4, LE>(c, a, L, s); break;
    case 8: launch_pass_g<LOGN, PASS, FWD, IN, OUT, 8, LE>(c, a, L, s); break;
    default: launch_pass_g<LOGN, PASS, FWD, IN, OUT, 16, LE>(c, a, L, s);
  }
}
template <int LOGN, int PASS, bool FWD, int IN, int OUT, typename List>
void launch_pass(Context* c, const PassArgs& a, const List& L, cudaStream_t s) {
  if constexpr (ntt_has_le3(LOGN)) {
    const bool wide_rescale = OUT == OUT_RESCALE && a.wide;
    if (LOGN >= 15 ? wide_rescale || c->ntt_residues(!FWD, PASS, L.n) == 8 : L.n <= NTT_LE3_SMALL) {
      launch_pass_le<LOGN, PASS, FWD, IN, OUT, 3>(c, a, L, s);
      return;
    }
  }
  launch_pass_le<LOGN, PASS, FWD, IN, OUT, 4>(c, a, L, s);
}

// The pass sequence of one transform for a given ring dimension.
template <int LOGN, typename List>
void run_transform(Context* c, const PassArgs& a, const List& L, bool inverse, NttIn in, NttOut out,
                   cudaStream_t s) {
  if (!inverse) {
    if (in == IN_SWITCH)
      launch_pass<LOGN, COL, true, IN_SWITCH, OUT_PLAIN>(c, a, L, s);
    else if (in == IN_SIGNED)
      launch_pass<LOGN, COL, true, IN_SIGNED, OUT_PLAIN>(c, a, L, s);
    else if (in == IN_CONV_SW)
      launch_pass<LOGN, COL, true, IN_CONV_SW, OUT_PLAIN>(c, a, L, s);
    else
      launch_pass<LOGN, COL, true, IN_PLAIN, OUT_PLAIN>(c, a, L, s);
    if (out == OUT_MODDOWN)
      launch_pass<LOGN, ROW, true, IN_PLAIN, OUT_MODDOWN>(c, a, L, s);
    else if (out == OUT_RESCALE)
      launch_pass<LOGN, ROW, true, IN_PLAIN, OUT_RESCALE>(c, a, L, s);
    else if (out == OUT_MDRS)
      launch_pass<LOGN, ROW, true, IN_PLAIN, OUT_MDRS>(c, a, L, s);
    else
      launch_pass<LOGN, ROW, true, IN_PLAIN, OUT_PLAIN>(c, a, L, s);
  } else {
    if (in == IN_MUL)
      launch_pass<LOGN, ROW, false, IN_MUL, OUT_PLAIN>(c, a, L, s);
    else
      launch_pass<LOGN, ROW, false, IN_PLAIN, OUT_PLAIN>(c, a, L, s);
    launch_pass<LOGN, COL, false, IN_PLAIN, OUT_PLAIN>(c, a, L, s);
  }
}

}  // namespace nttk

// Defined in ntt_inst_<logN>.cu.
#define FIDES_NTT_DECL(LN)                                                                                  \
  void ntt_transform_##LN(Context* c, const nttk::PassArgs& a, const NttLimbList& L, bool inverse, NttIn in, \
                          NttOut out, cudaStream_t s);                                                       \
  void ntt_transform_##LN(Context* c, const nttk::PassArgs& a, const NttLongList& L, bool inverse, NttIn in, \
                          NttOut out, cudaStream_t s);
FIDES_NTT_DECL(10)
FIDES_NTT_DECL(11)
FIDES_NTT_DECL(12)
FIDES_NTT_DECL(13)
FIDES_NTT_DECL(14)
FIDES_NTT_DECL(15)
FIDES_NTT_DECL(16)
FIDES_NTT_DECL(17)
#undef FIDES_NTT_DECL

}  // namespace fides
