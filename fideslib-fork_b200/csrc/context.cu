// Context creation: host-side table construction and upload.
//
// Replaces SetupConstants (reference src/ConstantsGPU.cu:132-640) and the CRT tables the
// reference takes from OpenFHE's raw parameters (RawCiphertext.cu:258-633):
//   - twiddles psi_rev[j] = psi^brev(j) with Shoup companions (ConstantsGPU.cu:246-318);
//   - ModUp tables PartQlHatInvModq / PartQlHatModp per (level, digit), digits being
//     OpenFHE's contiguous partition of alpha = ceil(n_q / dnum) primes (Context.cu:268-339);
//   - ModDown tables PHatInvModp / PHatModq / PInvModq (ConstantsGPU.cu:480-534);
//   - rescale constants q_l^-1 and QlQlInvModqlDivqlModq (RawCiphertext.cu:318-440), the
//     latter equal to -q_l^-1 mod q_j because q_j divides Q_{l-1}.
#include <cmath>
#include <algorithm>
#include <cstring>
#include <thread>

#include "context.hpp"
#include "conv_tc.hpp"
#include "ntt.cuh"

namespace fides {

typedef unsigned __int128 u128;

uint64_t h_mulmod(uint64_t a, uint64_t b, uint64_t q) { return (uint64_t)(((u128)a * b) % q); }
uint64_t h_powmod(uint64_t a, uint64_t e, uint64_t q) {
  uint64_t r = 1 % q;
  a %= q;
  for (; e; e >>= 1) {
    if (e & 1) r = h_mulmod(r, a, q);
    a = h_mulmod(a, a, q);
  }
  return r;
}
uint64_t h_invmod(uint64_t a, uint64_t q) { return h_powmod(a % q, q - 2, q); }

// Smallest primitive root g of q, then psi = g^((q-1)/2N) (the reference's standalone rule).
uint64_t h_root_2n(uint64_t q, int logN) {
  std::vector<uint64_t> fact;
  uint64_t phi = q - 1, n = phi;
  for (uint64_t i = 2; i * i <= n; ++i)
    if (n % i == 0) {
      fact.push_back(i);
      while (n % i == 0) n /= i;
    }
  if (n > 1) fact.push_back(n);
  uint64_t g = 2;
  for (;; ++g) {
    bool ok = true;
    for (uint64_t f : fact)
      if (h_powmod(g, phi / f, q) == 1) {
        ok = false;
        break;
      }
    if (ok) break;
  }
  return h_powmod(g, (q - 1) / (2ull << logN), q);
}

ShoupConst h_shoup(uint64_t w, uint64_t q) {
  ShoupConst c;
  c.w = w;
  c.ws = (uint64_t)(((u128)w << 64) / q);
  return c;
}

static uint32_t h_brev(uint32_t x, int bits) {
  uint32_t r = 0;
  for (int i = 0; i < bits; ++i) r |= ((x >> i) & 1u) << (bits - 1 - i);
  return r;
}

uint32_t h_auto_index(int logN, int rotation) {
  const int64_t N = 1ll << logN;
  if (rotation == 2 * N - 1) return (uint32_t)(2 * N - 1);
  int64_t h = N / 2, r = rotation % h;
  if (r < 0) r += h;
  return (uint32_t)h_powmod(5, (uint64_t)(2 * N - r), (uint64_t)(2 * N));
}

static double h_centred(uint64_t w, uint64_t q) { return w > q / 2 ? -(double)(q - w) : (double)w; }
static InvFinal inv_final(uint64_t sum, uint64_t diff, uint64_t q) {
  return InvFinal{h_shoup(sum, q), h_shoup(diff, q), h_centred(sum, q), h_centred(diff, q)};
}

static bool h_is_prime(uint64_t n) {
  static const uint64_t b[] = {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37};
  if (n < 2) return false;
  for (uint64_t p : b) {
    if (n == p) return true;
    if (n % p == 0) return false;
  }
  uint64_t d = n - 1;
  int s = 0;
  while (!(d & 1)) d >>= 1, ++s;
  for (uint64_t a : b) {
    uint64_t x = h_powmod(a, d, n);
    if (x == 1 || x == n - 1) continue;
    bool comp = true;
    for (int r = 1; r < s && comp; ++r) {
      x = h_mulmod(x, x, n);
      if (x == n - 1) comp = false;
    }
    if (comp) return false;
  }
  return true;
}

Scratch::Scratch(Context* c, size_t b, cudaStream_t st) : ctx(c), s(st), bytes(b) {
  if (b == 0) return;
  size_t now = ctx->scratch_in_use.fetch_add(b) + b;
  if (ctx->scratch_limit && now > ctx->scratch_limit) {
    ctx->scratch_in_use.fetch_sub(b);
    throw Error(-3, "scratch limit exceeded: need " + std::to_string(now) + " bytes, limit " +
                        std::to_string(ctx->scratch_limit));
  }
  size_t peak = ctx->scratch_peak.load();
  while (now > peak && !ctx->scratch_peak.compare_exchange_weak(peak, now)) {
  }
  cudaError_t e = cudaMallocFromPoolAsync(&p, b, ctx->pool, s);
  if (e != cudaSuccess) {
    ctx->scratch_in_use.fetch_sub(b);
    cudaGetLastError();
    throw Error(-3, std::string("device scratch allocation failed: ") + cudaGetErrorString(e));
  }
}

void reserve_scratch(Context* c, size_t bytes) {
  if (bytes == 0) return;
  FIDES_CUDA(cudaSetDevice(c->device));
  cudaStream_t s = nullptr;
  FIDES_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  void* p = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, c->pool, s);
  if (e == cudaSuccess) e = cudaFreeAsync(p, s);
  cudaError_t e2 = cudaStreamSynchronize(s);
  cudaStreamDestroy(s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error(-3, std::string("scratch reservation failed: ") + cudaGetErrorString(e));
  }
  FIDES_CUDA(e2);
}

Scratch::~Scratch() {
  if (p) {
    cudaFreeAsync(p, s);
    ctx->scratch_in_use.fetch_sub(bytes);
  }
}

static cudaEvent_t take_event(Context* c) {
  if (!c->ev_pool.empty()) {
    cudaEvent_t e = c->ev_pool.back();
    c->ev_pool.pop_back();
    return e;
  }
  cudaEvent_t e;
  FIDES_CUDA(cudaEventCreate(&e));
  return e;
}

LaunchScope::LaunchScope(Context* ctx, cudaStream_t st, int kind, double bytes) : c(ctx), s(st) {
  c->launches.fetch_add(1);
  if (!c->profiling) return;
  std::lock_guard<std::mutex> g(c->prof_mu);
  ProfileRec r{kind, take_event(c), take_event(c), bytes};
  FIDES_CUDA(cudaEventRecord(r.beg, s));
  c->prof.push_back(r);
  idx = (int)c->prof.size() - 1;
}

LaunchScope::~LaunchScope() {
  if (idx < 0) return;
  std::lock_guard<std::mutex> g(c->prof_mu);
  cudaEventRecord(c->prof[idx].end, s);
}

template <typename T>
static void append(std::vector<char>& blob, const std::vector<T>& v, size_t& off) {
  size_t a = 16;
  size_t o = (blob.size() + a - 1) / a * a;
  blob.resize(o + sizeof(T) * v.size());
  if (!v.empty()) std::memcpy(blob.data() + o, v.data(), sizeof(T) * v.size());
  off = o;
}

Context* create_context(int logN, int n_q, int K, int dnum, const uint64_t* primes, const uint64_t* psi, int device) {
  if (logN < 4 || logN > 17) throw Error(-1, "logN must be in [4, 17]");
  if (n_q < 1 || K < 0 || dnum < 1 || dnum > n_q) throw Error(-1, "need n_q >= 1, K >= 0, 1 <= dnum <= n_q");
  if (n_q + K > 256) throw Error(-1, "at most 256 primes");
  const int np = n_q + K;
  const uint64_t N = 1ull << logN;
  for (int i = 0; i < np; ++i) {
    uint64_t q = primes[i];
    if (q >= (1ull << 62) || q < 3 || (q - 1) % (2 * N) != 0 || !h_is_prime(q))
      throw Error(-1, "prime " + std::to_string(i) + " = " + std::to_string(q) +
                          " is not a prime < 2^62 with q = 1 mod 2N");
    for (int j = 0; j < i; ++j)
      if (primes[j] == q) throw Error(-1, "primes must be distinct");
  }
  auto* c = new Context();
  c->device = device;
  c->logN = logN;
  c->N = (int)N;
  c->n_q = n_q;
  c->K = K;
  c->dnum = dnum;
  c->alpha = (n_q + dnum - 1) / dnum;
  c->primes.assign(primes, primes + np);
  c->psi.resize(np);
  for (int i = 0; i < np; ++i) {
    uint64_t q = primes[i];
    uint64_t p = (psi && psi[i]) ? psi[i] : h_root_2n(q, logN);
    if (h_powmod(p, N, q) != q - 1) {
      delete c;
      throw Error(-1, "psi[" + std::to_string(i) + "] is not a primitive 2N-th root of unity");
    }
    c->psi[i] = p;
  }
  try {
    FIDES_CUDA(cudaSetDevice(device));
    // ---- per-prime constants and twiddles
    std::vector<DevPrime> hp(np);
    std::vector<InvFinal> fin(np);
    std::vector<F64Prime> f64(np);
    // NTT twiddles (the transforms start at N = 2^10): 8-byte entries where the FP64 butterflies
    // run, 16-byte ones elsewhere
    std::vector<size_t> tw_at(np + 1, 0);
    for (int i = 0; i < np; ++i)
      tw_at[i + 1] = tw_at[i] + (logN < 10 ? 0 : tw_block(logN) * (primes[i] < NTT_F64_MAX ? 8 : 16));
    std::vector<uint64_t> twid(tw_at[np] / sizeof(uint64_t));
    auto work = [&](int i) {
      uint64_t q = primes[i];
      DevPrime& d = hp[i];
      d.q = q;
      d.q2 = 2 * q;
      d.one_s = (uint64_t)(((u128)1 << 64) / q);
      d.r64 = (uint64_t)(((u128)1 << 64) % q);
      d.r64_s = h_shoup(d.r64, q).ws;
      const uint64_t ninv = h_invmod(N % q, q);
      d.tw = tw_at[i];
      std::vector<uint64_t> pw(N), ipw(N);
      uint64_t ip = h_invmod(c->psi[i], q);
      pw[0] = ipw[0] = 1;
      for (uint64_t j = 1; j < N; ++j) {
        pw[j] = h_mulmod(pw[j - 1], c->psi[i], q);
        ipw[j] = h_mulmod(ipw[j - 1], ip, q);
      }
      const double qd = (double)q;  // exact for q < 2^53; used only for q < 2^50
      auto centred = [&](uint64_t w) { return h_centred(w, q); };
      fin[i] = inv_final(ninv, h_mulmod(ipw[h_brev(1, logN)], ninv, q), q);
      uint64_t pmq = i < n_q ? 1 % q : 0;  // P mod q
      for (int k = 0; k < K; ++k) pmq = h_mulmod(pmq, primes[n_q + k] % q, q);
      f64[i] = F64Prime{qd, 1.0 / qd, centred((1ull << 51) % q), centred(pmq)};
      if (logN < 10) return;
      // the twiddle tables (layout in ntt.cuh); the twiddle of global stage s, block m is the
      // (2^s + m)-th power in bit-reversed order
      for (int le = 4; le >= (ntt_has_le3(logN) ? 3 : 4); --le)
        for (bool fwd : {true, false}) {
          const std::vector<uint64_t>& w = fwd ? pw : ipw;
          const size_t start = tw_start(logN, fwd, le);
          double* fd = reinterpret_cast<double*>(reinterpret_cast<char*>(twid.data()) + tw_at[i]) + start;
          ShoupConst* sh = reinterpret_cast<ShoupConst*>(reinterpret_cast<char*>(twid.data()) + tw_at[i]) + start;
          const int log1 = (logN + 1) / 2;
          size_t base = 0;  // of this sub-transform
          for (int pass = 0; pass < 2; ++pass) {
            const int logp = pass ? logN / 2 : log1, sbase = pass ? log1 : 0, subs = pass ? 1 << log1 : 1;
            for (int sub = 0; sub < subs; ++sub, base += tw_sub(logp, fwd, le))
              for (int ch = 0; ch < tw_chunks(logp, le); ++ch) {
                const int lo = tw_lo(logp, fwd, le, ch), slots = tw_slots(logp, fwd, le, ch);
                const size_t off = base + tw_off(logp, fwd, le, ch);
                for (int b = tw_blo(logp, fwd, le, ch); b <= tw_bhi(logp, fwd, le, ch); ++b) {
                  const int sig = logp - 1 - b, H = (1 << le) >> (b - lo + 1);
                  for (int th = 0; th < slots; ++th)
                    for (int hi = 0; hi < H; ++hi) {
                      const uint32_t m = (1u << (sbase + sig)) + ((uint32_t)sub << sig) +
                                         ((uint32_t)th << (lo + le - b - 1)) + (uint32_t)hi;
                      const uint64_t v = w[h_brev(m, logN)];
                      const int e = H + hi;
                      if (q < NTT_F64_MAX)
                        fd[off + (size_t)((e >> 1) * slots + th) * 2 + (e & 1)] = centred(v);
                      else
                        sh[off + (size_t)e * slots + th] = h_shoup(v, q);
                    }
                }
              }
          }
        }
    };
    {
      unsigned nt = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
      std::vector<std::thread> th;
      for (unsigned t = 0; t < nt; ++t)
        th.emplace_back([&, t] {
          for (int i = (int)t; i < np; i += (int)nt) work(i);
        });
      for (auto& t : th) t.join();
    }
    // ---- P mod q_j, P^-1 mod q_j, rescale constants
    std::vector<ShoupConst> pinv(n_q), pmod(n_q);
    for (int j = 0; j < n_q; ++j) {
      uint64_t q = primes[j], P = 1;
      for (int k = 0; k < K; ++k) P = h_mulmod(P, primes[n_q + k] % q, q);
      pmod[j] = h_shoup(P, q);
      pinv[j] = h_shoup(h_invmod(P, q), q);
    }
    std::vector<RescaleConst> rs((size_t)(n_q + 1) * n_q);
    std::vector<ShoupConst> pqinv((size_t)(n_q + 1) * n_q, ShoupConst{0, 0});
    for (int l = 2; l <= n_q; ++l) {
      uint64_t qt = primes[l - 1];
      for (int j = 0; j < l - 1; ++j) {
        uint64_t q = primes[j];
        uint64_t qi = h_invmod(qt % q, q);
        uint64_t m = qi ? q - qi : 0;
        RescaleConst& r = rs[(size_t)l * n_q + j];
        ShoupConst a = h_shoup(qi, q), b = h_shoup(m, q);
        r.qinv = a.w;
        r.qinv_s = a.ws;
        r.m = b.w;
        r.m_s = b.ws;
        if (K > 0) pqinv[(size_t)l * n_q + j] = h_shoup(h_mulmod(pinv[j].w, qi, q), q);
      }
    }
    // ---- conversion tables
    struct HostConv {
      std::vector<int> src_prime, dst_prime;
      int src0 = 0, dst_skip = 0, dst_gap = 0;
      std::vector<uint64_t> pre;  // (Q_src / q_i)^-1 mod q_i
      std::vector<uint64_t> mat;
      std::vector<uint8_t> tc_b;  // empty: no tensor-core form
      std::vector<TcDest> tc_dst;
      int kpad = 0, ndp = 0, lift = 0;
    };
    auto build_conv = [&](const std::vector<int>& spr, const std::vector<int>& dpr, int lift) {
      HostConv h;
      h.src_prime = spr;
      h.dst_prime = dpr;
      h.lift = lift;
      int ns = (int)spr.size(), nd = (int)dpr.size();
      h.pre.resize(ns);
      h.mat.resize((size_t)(ns + lift) * nd);
      for (int j = 0; j < nd && lift; ++j) {  // row ns: [-Q_src]_{p_j} (reference ReducedNoiseConstants.cu)
        uint64_t pj = primes[dpr[j]], v = 1 % pj;
        for (int k = 0; k < ns; ++k) v = h_mulmod(v, primes[spr[k]] % pj, pj);
        h.mat[(size_t)ns * nd + j] = v ? pj - v : 0;
      }
      for (int i = 0; i < ns; ++i) {
        uint64_t qi = primes[spr[i]], hq = 1;
        for (int k = 0; k < ns; ++k)
          if (k != i) hq = h_mulmod(hq, primes[spr[k]] % qi, qi);
        h.pre[i] = h_invmod(hq, qi);
        for (int j = 0; j < nd; ++j) {
          uint64_t pj = primes[dpr[j]], v = 1 % pj;
          for (int k = 0; k < ns; ++k)
            if (k != i) v = h_mulmod(v, primes[spr[k]] % pj, pj);
          h.mat[(size_t)i * nd + j] = v;
        }
      }
      if (conv_tc_fits(logN, ns + lift, nd, primes, dpr))
        build_tc_image(h.mat.data(), ns + lift, nd, dpr, primes, h.tc_b, h.tc_dst, h.kpad, h.ndp);
      return h;
    };
    // [lift][l]: the plain tables and the reduced-noise ones
    std::vector<std::vector<HostConv>> hmu[2] = {std::vector<std::vector<HostConv>>(n_q + 1),
                                                 std::vector<std::vector<HostConv>>(n_q + 1)};
    std::vector<HostConv> hmd[2] = {std::vector<HostConv>(n_q + 1), std::vector<HostConv>(n_q + 1)};
    for (int lift = 0; lift < 2; ++lift)
      for (int l = 1; l <= n_q; ++l) {
        int b = c->beta(l);
        for (int d = 0; d < b; ++d) {
          int s0 = d * c->alpha, s1 = std::min((d + 1) * c->alpha, l);
          std::vector<int> spr, dpr;
          for (int i = s0; i < s1; ++i) spr.push_back(i);
          for (int i = 0; i < l; ++i)
            if (i < s0 || i >= s1) dpr.push_back(i);
          for (int k = 0; k < K; ++k) dpr.push_back(n_q + k);
          hmu[lift][l].push_back(build_conv(spr, dpr, lift));
          HostConv& h = hmu[lift][l].back();
          h.src0 = h.dst_skip = s0;
          h.dst_gap = s1 - s0;
        }
        if (K > 0) {
          std::vector<int> spr, dpr;
          for (int k = 0; k < K; ++k) spr.push_back(n_q + k);
          for (int j = 0; j < l; ++j) dpr.push_back(j);
          hmd[lift][l] = build_conv(spr, dpr, lift);
        }
      }
    c->pinv = pinv;
    // ---- the sources' factors, folded into the inverse transforms that precede the conversions
    auto scaled = [&](int prime, uint64_t pre) {
      const uint64_t q = primes[prime];
      return inv_final(h_mulmod(fin[prime].sum.w, pre, q), h_mulmod(fin[prime].diff.w, pre, q), q);
    };
    std::vector<std::vector<InvFinal>> fin_up(n_q + 1);
    for (int l = 1; l <= n_q; ++l)
      for (const HostConv& h : hmu[0][l])
        for (size_t i = 0; i < h.pre.size(); ++i) fin_up[l].push_back(scaled(h.src_prime[i], h.pre[i]));
    std::vector<InvFinal> fin_down;
    if (K > 0)
      for (int k = 0; k < K; ++k) fin_down.push_back(scaled(n_q + k, hmd[0][1].pre[k]));
    // ---- pack everything into one device blob
    std::vector<char> blob;
    size_t o_prime, o_tw, o_fin, o_fin_down, o_pinv, o_pmod, o_rs, o_pq, o_f64;
    append(blob, hp, o_prime);
    append(blob, twid, o_tw);
    append(blob, fin, o_fin);
    append(blob, fin_down, o_fin_down);
    std::vector<size_t> o_fin_up(n_q + 1, 0);
    for (int l = 1; l <= n_q; ++l) append(blob, fin_up[l], o_fin_up[l]);
    append(blob, pinv, o_pinv);
    append(blob, pmod, o_pmod);
    append(blob, rs, o_rs);
    append(blob, pqinv, o_pq);
    append(blob, f64, o_f64);
    struct Off {
      size_t spr, dpr, mat, tcb, tcd;
      int ns, nd, kpad, ndp, lift, src0, dst_skip, dst_gap;
    };
    auto put = [&](const HostConv& h) {
      Off o;
      append(blob, h.src_prime, o.spr);
      append(blob, h.dst_prime, o.dpr);
      append(blob, h.mat, o.mat);
      append(blob, h.tc_b, o.tcb);
      append(blob, h.tc_dst, o.tcd);
      o.ns = (int)h.src_prime.size();
      o.nd = (int)h.dst_prime.size();
      o.kpad = h.tc_b.empty() ? 0 : h.kpad;
      o.ndp = h.ndp;
      o.lift = h.lift;
      o.src0 = h.src0;
      o.dst_skip = h.dst_skip;
      o.dst_gap = h.dst_gap;
      return o;
    };
    std::vector<std::vector<Off>> omu[2] = {std::vector<std::vector<Off>>(n_q + 1),
                                            std::vector<std::vector<Off>>(n_q + 1)};
    std::vector<Off> omd[2] = {std::vector<Off>(n_q + 1), std::vector<Off>(n_q + 1)};
    for (int lift = 0; lift < 2; ++lift)
      for (int l = 1; l <= n_q; ++l) {
        for (auto& h : hmu[lift][l]) omu[lift][l].push_back(put(h));
        if (K > 0) omd[lift][l] = put(hmd[lift][l]);
      }
    FIDES_CUDA(cudaMalloc(&c->d_tables, blob.size()));
    FIDES_CUDA(cudaMemcpy(c->d_tables, blob.data(), blob.size(), cudaMemcpyHostToDevice));
    char* base = static_cast<char*>(c->d_tables);
    c->d_prime = reinterpret_cast<DevPrime*>(base + o_prime);
    c->d_tw = base + o_tw;
    c->d_inv_fin = reinterpret_cast<InvFinal*>(base + o_fin);
    c->moddown_fin = reinterpret_cast<const InvFinal*>(base + o_fin_down);
    c->modup_fin.resize(n_q + 1);
    for (int l = 1; l <= n_q; ++l) c->modup_fin[l] = reinterpret_cast<const InvFinal*>(base + o_fin_up[l]);
    c->d_pinv = reinterpret_cast<ShoupConst*>(base + o_pinv);
    c->d_pmod = reinterpret_cast<ShoupConst*>(base + o_pmod);
    c->d_rescale = reinterpret_cast<RescaleConst*>(base + o_rs);
    c->d_pqinv = reinterpret_cast<ShoupConst*>(base + o_pq);
    c->d_f64 = reinterpret_cast<F64Prime*>(base + o_f64);
    auto mk = [&](const Off& o) {
      ConvTable t;
      t.n_src = o.ns;
      t.n_dst = o.nd;
      t.src0 = o.src0;
      t.src_prime = reinterpret_cast<const int*>(base + o.spr);
      t.dst_skip = o.dst_skip;
      t.dst_gap = o.dst_gap;
      t.dst_prime = reinterpret_cast<const int*>(base + o.dpr);
      t.mat = reinterpret_cast<const uint64_t*>(base + o.mat);
      t.lift = o.lift;
      if (o.kpad) {
        t.tc_b = reinterpret_cast<const uint8_t*>(base + o.tcb);
        t.tc_dst = reinterpret_cast<const TcDest*>(base + o.tcd);
        t.tc_kpad = o.kpad;
        t.tc_nd_pad = o.ndp;
      }
      return t;
    };
    c->modup_tab.resize(n_q + 1);
    c->moddown_tab.resize(n_q + 1);
    c->modup_tab_rn.resize(n_q + 1);
    c->moddown_tab_rn.resize(n_q + 1);
    for (int l = 1; l <= n_q; ++l) {
      for (auto& o : omu[0][l]) c->modup_tab[l].push_back(mk(o));
      for (auto& o : omu[1][l]) c->modup_tab_rn[l].push_back(mk(o));
      if (K > 0) {
        c->moddown_tab[l] = mk(omd[0][l]);
        c->moddown_tab_rn[l] = mk(omd[1][l]);
      }
    }
    // ---- scratch pool: keep freed blocks cached for reuse
    FIDES_CUDA(cudaDeviceGetDefaultMemPool(&c->pool, device));
    uint64_t thr = UINT64_MAX;
    FIDES_CUDA(cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &thr));
    FIDES_CUDA(cudaMalloc(&c->d_status, sizeof(uint32_t)));
    FIDES_CUDA(cudaMemset(c->d_status, 0, sizeof(uint32_t)));
    // ---- special-FFT twiddles for slot encode / decode (stage len = 2h, position j < h)
    {
      const size_t nh = (size_t)c->N / 2;
      std::vector<double> tw(2 * nh, 0.0);
      for (size_t h = 1; h < nh; h <<= 1) {
        const uint64_t m4 = 8 * h;  // 4 len
        uint64_t e = 1;             // 5^j mod 4 len
        for (size_t j = 0; j < h; ++j) {
          const double ang = -2.0 * M_PI * (double)e / (double)m4;
          tw[2 * (h + j)] = std::cos(ang);
          tw[2 * (h + j) + 1] = std::sin(ang);
          e = (e * 5) % m4;
        }
      }
      FIDES_CUDA(cudaMalloc(&c->d_sfft, tw.size() * sizeof(double)));
      FIDES_CUDA(cudaMemcpy(c->d_sfft, tw.data(), tw.size() * sizeof(double), cudaMemcpyHostToDevice));
    }
  } catch (...) {
    destroy_context(c);
    throw;
  }
  return c;
}

void destroy_context(Context* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  cudaDeviceSynchronize();
  for (auto& r : c->prof) {
    cudaEventDestroy(r.beg);
    cudaEventDestroy(r.end);
  }
  for (auto e : c->ev_pool) cudaEventDestroy(e);
  if (c->d_tables) cudaFree(c->d_tables);
  if (c->d_status) cudaFree(c->d_status);
  if (c->d_sfft) cudaFree(c->d_sfft);
  if (c->pinned) cudaFreeHost(c->pinned);
  delete c;
}

}  // namespace fides
