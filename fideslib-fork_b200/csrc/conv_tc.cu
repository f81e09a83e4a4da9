// Tensor-core basis conversion (tcgen05, kind::i8).  The arithmetic identity is stated in
// conv_tc.hpp; this file holds the table builder and the kernel.
//
// One CTA converts runs of 128 coefficients (the MMA's M, one TMEM lane each) of one job:
//   1. warp 0 allocates 64 TMEM columns; the CTA starts cp.async copies of the table's B image
//      (the shared-memory form of the byte matrix) and of A, K-major: the eight bytes of every source
//      residue of its 128 coefficients, as they lie in memory;
//   2. per chunk of 8 destination limbs (64 columns: 8 byte planes each), thread 0 issues
//      K/32 MMAs (M 128, N 8 x limbs, K 32) and commits them to an mbarrier;
//   3. after a bounded wait, each warp reads its 32 TMEM lanes (tcgen05.ld 32x32b), folds the
//      eight s32 planes of each output into 64 bits and reduces modulo the destination prime.
// Operands use the no-swizzle K-major canonical layout: core matrices of 8 rows x 16 bytes,
// rows 16 bytes apart, 8-row groups 128 bytes apart (SBO) and the two 16-byte K halves of an
// MMA LBO apart.  A is stored as [K/16][128 rows][16 B], B as [K/16][8 nd_pad rows][16 B].
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "conv_tc.hpp"
#include "kernels.cuh"
#include "launch.cuh"

#ifndef FIDES_TC_SMEM_GUARD
#define FIDES_TC_SMEM_GUARD 0
#endif

namespace fides {

void build_tc_image(const uint64_t* mat, int ns, int nd, const std::vector<int>& dst_prime,
                    const uint64_t* primes, std::vector<uint8_t>& b, std::vector<TcDest>& dst,
                    int& kpad, int& nd_pad) {
  kpad = tc_kpad(ns);
  nd_pad = tc_nd_pad(nd);
  const int nb = 8 * nd_pad;  // B rows
  b.assign((size_t)kpad * nb, 0);
  dst.assign(nd_pad, TcDest{0, 0});
  for (int j = 0; j < nd; ++j) {
    const uint64_t p = primes[dst_prime[j]];
    const double qinv = 1.0 / (double)p;
    dst[j].nq = 0 - p;
    std::memcpy(&dst[j].qinv, &qinv, sizeof(double));
    for (int i = 0; i < ns; ++i)
      for (int a = 0; a < 8; ++a) {
        const uint64_t v = h_mulmod(mat[(size_t)i * nd + j] % p, h_powmod(2, 8 * a, p), p);
        const int k = 8 * i + a;
        for (int cb = 0; cb < 8; ++cb) {
          const int n = 8 * j + cb;
          b[((size_t)(k / 16) * nb + n) * 16 + (k % 16)] = (uint8_t)(v >> (8 * cb));
        }
      }
  }
}

namespace {

constexpr int TC_M = 128;          // coefficients per CTA = TMEM lanes = MMA M
constexpr int TC_DCHUNK = 8;       // destination limbs per MMA chunk
constexpr uint32_t TC_COLS = 64;   // TMEM columns held by one CTA (8 limbs x 8 byte planes)
// Shared memory of at least this size per CTA keeps at most 7 CTAs (448 TMEM columns of the
// SM's 512) resident, so tcgen05.alloc never waits for another CTA.
constexpr int TC_SMEM_FLOOR = 29 * 1024;

struct TcLayout {
  int o_dst, o_a, o_b, total;
};
__host__ __device__ inline TcLayout tc_layout(int kpad, int ndp) {
  TcLayout L;
  L.o_dst = 16;  // [0, 8): mbarrier, [8, 12): TMEM address
  L.o_a = (L.o_dst + ndp * (int)sizeof(TcDest) + 127) & ~127;
  L.o_b = L.o_a + TC_M * kpad;
  L.total = L.o_b + kpad * 8 * ndp;
  return L;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor: K-major, no swizzle, sm_100 descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::i8: s32 accumulator (bits 4-5 = 2), A and B unsigned
// (formats 0), both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__device__ __forceinline__ uint32_t idesc_u8(int n) {
  return (2u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
}

__device__ __forceinline__ void mma_u8(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
      :
      : "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ bool bar_try_wait(uint32_t bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(phase)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Waits for the barrier phase for at most about one second; false if it gave up.
__device__ bool bar_wait_bounded(uint32_t bar, uint32_t phase) {
  const uint64_t t0 = globaltimer();
  for (uint32_t it = 1;; ++it) {
    if (bar_try_wait(bar, phase)) return true;
    if ((it & 63) == 0 && globaltimer() - t0 > 1000000000ull) return false;
  }
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// The planes of two destination limbs: 16 columns, waited for.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&d)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]),
        "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_cp_async8(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void tc_cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(smem)), "l"(gmem) : "memory");
}
// sum_c 2^(8c) d[c] mod q for planes d[c] < 2^23 and a prime 2^48 < q < 2^62.
// V = x + 2^32 y with x, y < 2^49 (V < 2^79.01 for K <= 128) is reduced by floating-point
// Barrett reduction (the double-precision quotient estimate of NTL's MulMod): the integers
// x, y are formed with the exponent of 2^52 above them, so that they are doubles after one
// subtraction, and vd = fl(V), qinv = fl(1/q) give
// vd qinv within 2^-20 of V/q (V/q < 2^31.01); the fma adds 2^-17 with one more rounding of
// at most 2^-21, so t lies in (V/q + 2^-17.6, V/q + 2^-16.6) and qh = floor(t) is
// floor(V/q) or one more (qh < 2^32).  V - qh q lies in [-q, q), is computed exactly in
// wrapping 64-bit arithmetic (nq = -q) and needs one correction.  (Checked against 128-bit arithmetic
// on 40 M random, extreme and next-to-a-multiple-of-q plane sets over 4000 primes.)
// Written out in wide multiply-adds: as C++ the same steps took 4 % more of the kernel's time.
__device__ __forceinline__ uint64_t tc_fold(const uint32_t* d, uint64_t nq, double qinv) {
  const uint32_t a0 = d[0] + (d[1] << 8), a1 = d[2] + (d[3] << 8);  // < 2^32
  const uint32_t a2 = d[4] + (d[5] << 8), a3 = d[6] + (d[7] << 8);
  constexpr uint32_t EXP52 = 0x43300000u;  // upper word of 2^52
  uint64_t x, y;                           // 2^52's exponent over planes 0-3 and 4-7 (weight 2^32), each < 2^49
  asm("{.reg .b64 t;\n\tmov.b64 t, {%1, %3};\n\tmad.wide.u32 %0, %2, 65536, t;}" : "=l"(x) : "r"(a0), "r"(a1), "r"(EXP52));
  asm("{.reg .b64 t;\n\tmov.b64 t, {%1, %3};\n\tmad.wide.u32 %0, %2, 65536, t;}" : "=l"(y) : "r"(a2), "r"(a3), "r"(EXP52));
  const double two52 = 4503599627370496.0;
  const double xd = __longlong_as_double((long long)x) - two52, yd = __longlong_as_double((long long)y) - two52;
  const double vd = fma(yd, 4294967296.0, xd);
  const uint32_t qh = (uint32_t)__double2loint(__dadd_rd(fma(vd, qinv, 0x1p-17), two52));  // floor, < 2^32
  // x + 2^32 y + qh nq without the exponent
  uint64_t r;
  asm("{.reg .b64 t;\n\t.reg .b32 l, h;\n\t"
      "mad.wide.u32 t, %1, %2, %4;\n\tmov.b64 {l, h}, t;\n\tmad.lo.u32 h, %1, %3, h;\n\t"
      "add.u32 h, h, %5;\n\tsub.u32 h, h, %6;\n\tmov.b64 %0, {l, h};}"
      : "=l"(r)
      : "r"(qh), "r"((uint32_t)nq), "r"((uint32_t)(nq >> 32)), "l"(x), "r"((uint32_t)y), "r"(EXP52));
  if ((int64_t)r < 0) r -= nq;
  return r;
}

// Stores the folded outputs of one chunk of NDC destination limbs (8 byte-plane columns each,
// starting at TMEM address trow), two limbs a TMEM load.  (Loading the next pair while one is folded
// gained nothing: the warps of seven CTAs an SM cover the wait.)
// TOP: the job's last output becomes (top - v) P^-1 (ConvJob::top).
template <int NDC, bool CHECK, bool TOP>
__device__ __forceinline__ void tc_epilogue(uint32_t trow, int j0, int nd, const TcDest* dconst, const ConvJob& J,
                                            int logN, uint64_t* out, uint64_t top) {
#pragma unroll
  for (int h = 0; h < NDC / 2; ++h) {
    uint32_t d[16];
    tmem_ld16(trow + 16 * h, d);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = j0 + 2 * h + u;
      if (!CHECK || j < nd) {
        const TcDest P = dconst[j];
        uint64_t v = tc_fold(d + 8 * u, P.nq, __longlong_as_double((long long)P.qinv));
        if (TOP && j == nd - 1) v = shoup(submod(top, v, 0 - P.nq), J.top_pinv.w, J.top_pinv.ws, 0 - P.nq);
        out[(size_t)J.t.dst_pos(j) << logN] = v;
      }
    }
  }
}

// Each CTA converts `tiles` runs of 128 coefficients: the B image and the tables are fetched once, and
// the next run's sources are on their way while the last chunk of the current one is folded.  The kernel
// is bound by its instructions (issue 67-69 %, FMA-heavy pipe 41 %, DRAM 30 %): with a CTA a run and the
// sources staged through registers 48 ModUp conversions at N = 2^16, level 30 took 242 us and 32 ModDown
// conversions 159; 211 and 156 with several runs, 183 and 138 with tc_fold's wide multiply-adds as well
// (136 and 90 at the rate of a copy).
template <int CAP>
__global__ void __launch_bounds__(TC_M, 7)
    conv_tc_kernel(const __grid_constant__ ConvJobListT<CAP> L, const DevPrime* primes, int logN, uint32_t* status,
                   int tiles) {
  extern __shared__ __align__(1024) uint8_t sm[];
  const ConvJob& J = L.j[blockIdx.y];
  const ConvTable& T = J.t;
  const int ns = T.n_src, nd = T.n_dst, kpad = T.tc_kpad, ndp = T.tc_nd_pad;
  const int nchunks = (ndp + TC_DCHUNK - 1) / TC_DCHUNK;
  const TcLayout Ly = tc_layout(kpad, ndp);
  const int tid = threadIdx.x, warp = tid >> 5;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + 8);
  TcDest* dconst = reinterpret_cast<TcDest*>(sm + Ly.o_dst);
  uint8_t* sA = sm + Ly.o_a;
  uint8_t* sB = sm + Ly.o_b;
  const uint32_t bar_a = smem_addr(bar);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)),
                 "r"(TC_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_a), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  {  // B image: 16-byte cp.async copies (kpad 8 ndp bytes, a multiple of 256), waited for below
    const int n16 = kpad * ndp / 2;
    for (int k = tid; k < n16; k += TC_M) tc_cp_async16(sB + 16 * k, T.tc_b + 16 * k);
  }
  for (int j = tid; j < ndp; j += TC_M) dconst[j] = T.tc_dst[j];  // destination constants
  pdl_wait();  // tables only so far
  // A: the bytes of the sources of one run, the eight of source i at 16-byte K slice i / 2.  The K rows past
  // the last source are not written: B is zero there.
  const int coef0 = blockIdx.x * tiles * TC_M + tid;
  auto load_a = [&](int coef) {
    const uint64_t* src = J.src + ((size_t)T.src0 << logN) + coef;
    uint8_t* dst = sA + tid * 16;
    for (int i = 0; i < ns; ++i)
      tc_cp_async8(dst + (i >> 1) * (TC_M * 16) + (i & 1) * 8, src + ((size_t)i << logN));
  };
  load_a(coef0);
  bool ok = true;
  int phase = 0;  // of the mbarrier: one commit a chunk
  const uint32_t sa = smem_addr(sA), sb = smem_addr(sB);
  uint32_t tbase = 0;
  for (int tile = 0; ok && tile < tiles; ++tile) {
    asm volatile("cp.async.wait_all;" ::: "memory");  // this thread's sources and part of the B image
    if (T.lift) {  // reduced-noise lift: the number of sources above q / 2 is source row ns of the product
      uint64_t lifted = 0;
      for (int i = 0; i < ns; ++i)
        lifted += *reinterpret_cast<const uint64_t*>(sA + (i >> 1) * (TC_M * 16) + tid * 16 + (i & 1) * 8) >
                  (primes[T.src_prime[i]].q >> 1);
      *reinterpret_cast<uint64_t*>(sA + (ns >> 1) * (TC_M * 16) + tid * 16 + (ns & 1) * 8) = lifted;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // A and B, visible to the MMAs
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tbase = *slot;
    const uint32_t trow = tbase + ((uint32_t)(warp * 32) << 16);
    uint64_t* out = J.dst + coef0 + tile * TC_M;
    for (int c = 0; c < nchunks; ++c) {
      const int ndc = min(TC_DCHUNK, ndp - c * TC_DCHUNK);  // even: N = 8 ndc is a multiple of 16
      if (tid == 0) {
        const uint32_t idesc = idesc_u8(8 * ndc);
        for (int kc = 0; kc < kpad / 32; ++kc) {
          const uint64_t da = smem_desc(sa + kc * 2 * (TC_M * 16), TC_M * 16, 128);
          const uint64_t db = smem_desc(sb + (kc * 2 * (8 * ndp) + c * TC_DCHUNK * 8) * 16, 8 * ndp * 16, 128);
          mma_u8(tbase, da, db, idesc, kc > 0);
        }
        mma_commit(bar_a);
      }
      ok = __syncthreads_and(bar_wait_bounded(bar_a, phase));
      if (!ok) break;
      phase ^= 1;
      tc_fence_after();
      if (c + 1 == nchunks && tile + 1 < tiles) load_a(coef0 + (tile + 1) * TC_M);  // the MMAs have read A
      const int j0 = c * TC_DCHUNK;
      auto fold_chunk = [&](auto top_) {
        constexpr bool TOP = decltype(top_)::value;
        const uint64_t top = TOP ? J.top[coef0 + tile * TC_M] : 0;
        if (ndc == TC_DCHUNK && j0 + TC_DCHUNK <= nd)
          tc_epilogue<TC_DCHUNK, false, TOP>(trow, j0, nd, dconst, J, logN, out, top);
        else if (ndc == 2)
          tc_epilogue<2, true, TOP>(trow, j0, nd, dconst, J, logN, out, top);
        else if (ndc == 4)
          tc_epilogue<4, true, TOP>(trow, j0, nd, dconst, J, logN, out, top);
        else if (ndc == 6)
          tc_epilogue<6, true, TOP>(trow, j0, nd, dconst, J, logN, out, top);
        else
          tc_epilogue<8, true, TOP>(trow, j0, nd, dconst, J, logN, out, top);
      };
      if (J.top && c + 1 == nchunks)
        fold_chunk(std::true_type{});
      else
        fold_chunk(std::false_type{});
      tc_fence_before();
      __syncthreads();  // TMEM columns are free for the next chunk
      tc_fence_after();
    }
  }
  if (!ok) {
    // The commit of the chunk in flight has not arrived: its MMAs may still own the TMEM
    // columns.  tcgen05.commit arrives on the mbarrier only after every MMA this thread issued
    // before it has completed, so a second bounded wait on the same phase either sees them
    // finish (the dealloc below is then safe) or gives up after about another second, when
    // the tensor pipe is not progressing at all; the columns are freed in either case so the
    // CTA can exit, and the status word marks every output of the launch as incomplete (the
    // host's next synchronising call returns FIDES_ERR_TIMEOUT until it is cleared).
    if (tid == 0) {
      atomicOr(status, 1u);
      bar_wait_bounded(bar_a, phase);
    }
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(TC_COLS) : "memory");
  }
}

}  // namespace

namespace {
template <int CAP>
void launch_conv_tc_list(Context* c, const ConvJob* jobs, int m, cudaStream_t s) {
  static thread_local ConvJobListT<CAP> L;
  static bool attr = false;
  if (!attr) {
    FIDES_CUDA(cudaFuncSetAttribute(conv_tc_kernel<CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr = true;
  }
  L.n = m;
  std::copy(jobs, jobs + m, L.j);
  int smem = TC_SMEM_FLOOR;
  double bytes = 0;
  for (int i = 0; i < m; ++i) {
    const ConvTable& t = L.j[i].t;
    if (!t.tc_b) throw Error(-1, "basis conversion has no tensor-core form");
    smem = std::max(smem, tc_layout(t.tc_kpad, t.tc_nd_pad).total + FIDES_TC_SMEM_GUARD);
    bytes += 8.0 * c->N * (t.n_src + t.n_dst);
  }
  // runs a CTA: as many as leave four waves of seven CTAs an SM
  int tiles = 1;
  while (tiles < 8 && (long)(c->N / TC_M) * m / (2 * tiles) >= 4 * 7 * 148) tiles *= 2;
  dim3 grid(c->N / TC_M / tiles, m);
  LaunchScope ls(c, s, KK_CONV, bytes);
  launch_pdl(conv_tc_kernel<CAP>, grid, TC_M, smem, s, L, c->d_prime, c->logN, c->d_status, tiles);
}
}  // namespace

void launch_conv_tc(Context* c, const ConvJob* jobs, int n, cudaStream_t s) {
  for (int off = 0; off < n; off += MAX_CONV_JOBS) {
    const int m = std::min(MAX_CONV_JOBS, n - off);
    if (m <= FEW_JOBS)
      launch_conv_tc_list<FEW_JOBS>(c, jobs + off, m, s);
    else
      launch_conv_tc_list<MAX_CONV_JOBS>(c, jobs + off, m, s);
  }
}

}  // namespace fides
