// Negacyclic NTT / INTT over lists of limbs.
//
// Replaces the reference's NTT_/INTT_/NTTBatch_ kernels (src/NTT.cu:42-802) and their
// launchers ApplyNTT/ApplyINTT (src/CKKS/LimbPartition.cu:433-550).  Same transform
// (forward: Cooley-Tukey with bit-reversed psi powers, output in bit-reversed EVALUATION
// order; inverse: Gentleman-Sande with N^-1 folded into the last stage), a different
// schedule:
//   * N = 2^LOG1 x 2^LOG2.  Pass COL runs global stages [0, LOG1) on strided columns,
//     pass ROW runs stages [LOG1, logN) on contiguous rows.  Forward = COL then ROW,
//     inverse = ROW then COL; each pass reads and writes every limb once.
//   * each thread keeps 2^LE elements in registers (16, or 8: where the autotuner picks it at
//     N >= 2^15, for small launches at N = 2^12 to 2^14, and for rescales above 2^50, below) and
//     runs LE stages per chunk; chunks exchange through padded shared memory;
//   * primes below 2^50 run FP64 butterflies (exact integers in doubles, ntt_impl.cuh), larger ones lazy
//     butterflies with one 64-bit Shoup product each (primes < 2^62): below 2^61 the forward transform
//     lets values grow by 4q a stage and subtracts once a chunk, at every second or at every stage, by
//     the size of q; above it keeps Harvey's [0, 4q) form; the inverse tracks a bound B (a multiple
//     of q) and subtracts only once B passes 2^62;
//   * one launch covers any list of limbs (any polynomials, any levels): blockIdx.y
//     indexes a limb of a list of runs (pointers + prime id) passed by value;
//   * the first pass may read from a separate source (out of place) or compute its input
//     (prologue), and the last pass may combine its result with other operands before
//     storing (epilogue) -- the reference's NTT fusion modes (src/NTT.cuh:39-69,
//     src/NTTfusions.cuh:12-336) as compile-time variants.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>

#include "context.hpp"

namespace fides {

// What the first pass loads.
enum NttIn {
  IN_PLAIN = 0,    // x = src[i]  (src = ptr when in place)
  IN_MUL = 1,      // inverse only: x = src[i] * pro[i] mod q   (tensor term a1 b1)
  IN_SWITCH = 2,   // forward only: x = SwitchModulus(pro[i]) from prime aux - 1 (rescale)
  IN_CONV_SW = 3,  // forward only: x = src[i] + P SwitchModulus(pro[i]) from prime aux - 1
  IN_SIGNED = 4,   // forward only: x = pro[i] read as a signed 64-bit integer, reduced mod q (encode)
};
// What the last pass stores to ptr.
enum NttOut {
  OUT_PLAIN = 0,
  OUT_MODDOWN = 1,   // forward only: out = (ep0[i] - v) P^-1 (+ ep1[i])     (ModDown finish)
  OUT_RESCALE = 2,   // forward only: out = qinv_l ep0[i] + QlQlInv_l v, l = aux (rescale finish)
  OUT_MDRS = 3,      // forward only: out = (ep0[i] - v) (P q_(l-1))^-1, l = aux
};

// ---- Twiddle tables.  A pass runs the stages of one register chunk (2^le residues per thread) after
// another; in each chunk a thread needs 2^le - 1 twiddles, one heap of them: entry (number of twiddles
// of the stage) + hi is twiddle hi of that stage, so a full chunk's stages use entries 1, 2-3, 4-7, ...
// Threads that share the register span's upper bits (th = t >> lo) share the heap.  A chunk's heaps are
// stored interleaved by th, so the lanes of a warp read consecutive addresses:
//   integer twiddles (16 bytes, w and its Shoup companion): entry i of th at i * slots + th;
//   FP64 twiddles (8 bytes): entries in pairs, i of th at ((i >> 1) * slots + th) * 2 + (i & 1).
// Stored by natural index, the twiddles of a chunk's last stage lay 64 bytes apart from lane to lane,
// and their loads alone were 40-55 % of the passes' L1 wavefronts (the L1 data pipe was 80 % busy).
// With this layout and the FP64 butterflies' single 8-byte twiddle (ntt_impl.cuh) 300 limbs of 50-bit
// primes at N = 2^16 take 124.5 us forward and 128.3 us inverse, against 140.3 and 150.7 (copying them
// twice, as two passes must, takes 100).
// A table (one prime, direction and le): the column pass's chunks, then those of each row of the row
// pass.
constexpr int tw_chunks(int logp, int le) { return (logp + le - 1) / le; }
// lowest bit of the register span of chunk c
constexpr int tw_lo(int logp, bool fwd, int le, int c) {
  return fwd ? (logp - (c + 1) * le > 0 ? logp - (c + 1) * le : 0) : (c * le + le <= logp ? c * le : logp - le);
}
// the pair bits [blo, bhi] of chunk c
constexpr int tw_bhi(int logp, bool fwd, int le, int c) {
  return fwd ? logp - 1 - c * le : (c * le + le - 1 < logp - 1 ? c * le + le - 1 : logp - 1);
}
constexpr int tw_blo(int logp, bool fwd, int le, int c) {
  return fwd ? (logp - (c + 1) * le > 0 ? logp - (c + 1) * le : 0) : c * le;
}
constexpr int tw_slots(int logp, bool fwd, int le, int c) { return 1 << (logp - le - tw_lo(logp, fwd, le, c)); }
constexpr int tw_off(int logp, bool fwd, int le, int c) {
  int o = 0;
  for (int k = 0; k < c; ++k) o += tw_slots(logp, fwd, le, k) << le;
  return o;
}
constexpr int tw_sub(int logp, bool fwd, int le) { return tw_off(logp, fwd, le, tw_chunks(logp, le)); }
constexpr size_t tw_table(int logN, bool fwd, int le) {
  return (size_t)tw_sub((logN + 1) / 2, fwd, le) + ((size_t)tw_sub(logN / 2, fwd, le) << ((logN + 1) / 2));
}
// Passes with 8 residues per thread exist for these rings.
constexpr bool ntt_has_le3(int logN) { return logN >= 12; }
// At N >= 2^15 the context's tables choose between 16 and 8; below, launches of up to this many limbs
// take 8: their time is that of one CTA, and its threads then run half the butterflies one after another
// (one rotation at N = 2^13, level 3: 48 -> 41 us; one product at N = 2^14, level 9: 63 -> 49).
constexpr int NTT_LE3_SMALL = 32;
// A row pass with the rescale epilogue takes 8 at N >= 2^15 whatever the tables say where most limbs are of
// primes above 2^50: its two integer products a residue are a chain that only more warps hide (16 rescales of
// 24 limbs at N = 2^16 414-418 us with 16, 380 with 8; a plain transform 292 and 296, FP64 limbs 220 and 240,
// so the tables, timed on plain transforms, would choose 16).
// Start of the table of (direction, le) in a prime's block, and the block's size, in entries.
constexpr size_t tw_start(int logN, bool fwd, int le) {
  size_t o = 0;
  if (le == 3) o += tw_table(logN, true, 4) + tw_table(logN, false, 4);
  return o + (fwd ? 0 : tw_table(logN, true, le));
}
constexpr size_t tw_block(int logN) {
  return tw_table(logN, true, 4) + tw_table(logN, false, 4) +
         (ntt_has_le3(logN) ? tw_table(logN, true, 3) + tw_table(logN, false, 3) : 0);
}
// primes with the FP64 butterflies
constexpr uint64_t NTT_F64_MAX = 1ull << 50;

struct LimbRef {
  uint64_t* ptr;          // output (and input of the first pass when src is null)
  const uint64_t* src;    // optional input of the first pass
  const uint64_t* pro;    // prologue operand
  const uint64_t* ep0;    // epilogue operands
  const uint64_t* ep1;
  int prime;
  int aux;  // IN_SWITCH / IN_CONV_SW / OUT_RESCALE / OUT_MDRS: the level l being rescaled (top prime l - 1)
  const InvFinal* fin;    // inverse only: last-stage factors of this limb (null: the prime's own)
};

inline LimbRef lref(uint64_t* p, int prime) { return LimbRef{p, nullptr, nullptr, nullptr, nullptr, prime, 0, nullptr}; }

#ifndef FIDES_MAX_NTT_LIMBS
#define FIDES_MAX_NTT_LIMBS 448
#endif
constexpr int MAX_NTT_LIMBS = FIDES_MAX_NTT_LIMBS;

// A launch's limbs as runs: limb k of a run has every pointer k limbs further (pro: unless the run
// shares one prologue limb) and prime id prime + k.  Launches of the library's operations have a few
// runs a polynomial, so the kernel parameters stay small: 448 limb descriptors (28 KB) cost 3-5 us
// of host time a launch more than 256 bytes, at 3-4.6 us, and runs 0.5.
struct LimbRun {
  uint64_t* ptr;
  const uint64_t *src, *pro, *ep0, *ep1;
  const InvFinal* fin;
  int16_t prime, aux;
  int16_t first;     // index of the run's first limb in the launch
  int16_t pro_step;  // 1: pro advances with the limb
};
template <int RUNS>
struct NttLimbListT {
  static constexpr int max_runs = RUNS;
  int n, runs;
  LimbRun run[RUNS];
  std::conditional_t<RUNS <= 256, uint8_t, uint16_t> run_of[MAX_NTT_LIMBS];
};
// Limbs that do not follow one another (one limb of each of many plaintexts or ciphertexts, a caller's
// own list) make a run each.  A chunk of more than 96 runs takes the passes built with a run for every
// limb (26 KB of parameters): split at 96 runs, decoding 400 plaintexts took 74 us at N = 2^12 and
// 62 at 2^11, with one launch pair 51 and 33.
constexpr int MAX_NTT_RUNS = 96;
using NttLimbList = NttLimbListT<MAX_NTT_RUNS>;
using NttLongList = NttLimbListT<MAX_NTT_LIMBS>;
static_assert(MAX_NTT_LIMBS < 32768, "LimbRun holds the index");

// Launch a full forward or inverse transform over `n` limbs (any n; split internally).
// The prologue/epilogue modes apply to every limb of the call.
void ntt_limbs(Context* c, const LimbRef* limbs, int n, bool inverse, cudaStream_t s, NttIn in = IN_PLAIN,
               NttOut out = OUT_PLAIN);
// Convenience: n_polys polynomials of `n_limbs` consecutive limbs starting at `data`,
// limb i of each poly using prime id prime_ids[i].
void ntt_polys(Context* c, uint64_t* data, int n_polys, int n_limbs, const int* prime_ids, bool inverse,
               cudaStream_t s);

}  // namespace fides
