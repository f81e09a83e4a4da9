// Negacyclic NTT / INTT: launch planning (see ntt.cuh for the design, ntt_impl.cuh for
// the kernels).
#include <algorithm>
#include <vector>

#include "ntt_impl.cuh"

namespace fides {

namespace {
// limbs[from, n) as runs in L, which holds those of the limbs before; returns the first limb that does
// not fit (n: all do).
template <typename List>
int fill_runs(List& L, const LimbRef* limbs, int from, int n, size_t N) {
  // b lies one limb after a, or both are null
  auto next = [N](const uint64_t* a, const uint64_t* b) { return b == (a ? a + N : nullptr); };
  L.n = n;
  for (int i = from; i < n; ++i) {
    const LimbRef& x = limbs[i];
    bool joins = false;
    if (i) {
      const LimbRef& y = limbs[i - 1];
      LimbRun& r = L.run[L.runs - 1];
      joins = next(y.ptr, x.ptr) & next(y.src, x.src) & next(y.ep0, x.ep0) & next(y.ep1, x.ep1) &
              (x.prime == y.prime + 1) & (x.aux == y.aux) & (x.fin == (y.fin ? y.fin + 1 : nullptr));
      if (joins) {
        const bool same = x.pro == y.pro, step = next(y.pro, x.pro);
        if (i - r.first == 1) r.pro_step = !same && step;
        joins = r.pro_step ? step : same;
      }
    }
    if (!joins) {
      if (L.runs == List::max_runs) return i;
      L.run[L.runs++] = LimbRun{x.ptr, x.src, x.pro, x.ep0, x.ep1, x.fin, (int16_t)x.prime, (int16_t)x.aux, (int16_t)i, 0};
    }
    L.run_of[i] = L.runs - 1;
  }
  return n;
}
}  // namespace

void ntt_limbs(Context* c, const LimbRef* limbs, int n, bool inverse, cudaStream_t s, NttIn in, NttOut out) {
  if (n <= 0) return;
  if (c->logN < 10) throw Error(-1, "GPU NTT needs logN >= 10");
  const bool ok = inverse ? ((in == IN_PLAIN || in == IN_MUL) && out == OUT_PLAIN)
                          : ((in == IN_PLAIN || in == IN_SWITCH || in == IN_CONV_SW || in == IN_SIGNED) &&
                             (out == OUT_PLAIN || out == OUT_MODDOWN || out == OUT_RESCALE || out == OUT_MDRS));
  if (!ok) throw Error(-1, "NTT prologue/epilogue not available in this direction");
  nttk::PassArgs a;
  a.primes = c->d_prime;
  a.tw = c->d_tw;
  a.f64 = c->d_f64;
  a.inv_fin = c->d_inv_fin;
  a.pinv = c->d_pinv;
  a.rescale = c->d_rescale;
  a.pmod = c->d_pmod;
  a.pqinv = c->d_pqinv;
  a.logN = c->logN;
  a.log1 = (c->logN + 1) / 2;
  a.n_q = c->n_q;
  {
    uint64_t nf = 0;
    for (int i = 0; i < n; ++i) nf += c->primes[limbs[i].prime] < NTT_F64_MAX;
    c->ntt_limbs_by_form[0] += nf;
    c->ntt_limbs_by_form[1] += (uint64_t)n - nf;
    a.wide = 2 * nf < (uint64_t)n;
  }
  auto launch = [&](const auto& list) {
    switch (c->logN) {
      case 10: ntt_transform_10(c, a, list, inverse, in, out, s); break;
      case 11: ntt_transform_11(c, a, list, inverse, in, out, s); break;
      case 12: ntt_transform_12(c, a, list, inverse, in, out, s); break;
      case 13: ntt_transform_13(c, a, list, inverse, in, out, s); break;
      case 14: ntt_transform_14(c, a, list, inverse, in, out, s); break;
      case 15: ntt_transform_15(c, a, list, inverse, in, out, s); break;
      case 16: ntt_transform_16(c, a, list, inverse, in, out, s); break;
      case 17: ntt_transform_17(c, a, list, inverse, in, out, s); break;
      default: throw Error(-1, "GPU NTT supports logN 10..17");
    }
  };
  static thread_local NttLimbList L;
  static thread_local NttLongList all;
  // balanced chunks of at most the context's chunk size, both passes of a chunk back to back
  const int cap = c->ntt_chunk > 0 ? std::min(c->ntt_chunk, MAX_NTT_LIMBS) : MAX_NTT_LIMBS;
  const int nchunks = (n + cap - 1) / cap, per = (n + nchunks - 1) / nchunks;
  for (int off = 0; off < n; off += per) {
    const int m = std::min(per, n - off);
    L.runs = 0;
    const int k = fill_runs(L, limbs + off, 0, m, c->N);
    if (k == m) {
      launch(L);
      continue;
    }
    all.runs = L.runs;
    std::copy(L.run, L.run + L.runs, all.run);
    std::copy(L.run_of, L.run_of + k, all.run_of);
    fill_runs(all, limbs + off, k, m, c->N);
    launch(all);
  }
}

void ntt_polys(Context* c, uint64_t* data, int n_polys, int n_limbs, const int* prime_ids, bool inverse,
               cudaStream_t s) {
  std::vector<LimbRef> v((size_t)n_polys * n_limbs);
  for (int p = 0; p < n_polys; ++p)
    for (int i = 0; i < n_limbs; ++i)
      v[(size_t)p * n_limbs + i] = lref(data + ((size_t)p * n_limbs + i) * c->N, prime_ids[i]);
  ntt_limbs(c, v.data(), (int)v.size(), inverse, s);
}

}  // namespace fides
