// Epstein-Nesbet PT2 on the device: deterministic, pseudo-stochastic and stochastic stages
// (K6 in PT mode + K7).
//
// Reference: Solver<S>::get_energy_pt_dtm / _psto / _sto (src/solver/solver.h:636-1153) and
// mapreduce_sum (:1155-1177).  Each stage visits source dets i (all var dets, or a stochastic
// sample) and emits the connected dets a in the heat-bath window [eps / |c_i|, INF) that fall
// in the current hash batch (rehash(DetHasher(a)) % n_batches), are not variational and have
// |H_ai c_i| >= eps.  The reference accumulates (a -> sum) in a distributed hash map; here
// the (a, values) pairs are grouped by det (group.cu) and reduced in a fixed order, and a second kernel forms each unique a's contribution with its diagonal H_aa.
//   dtm : value  = H_ai c_i                          contribution S0^2 / (E - H_aa)
//   psto: values = [hc, hc if |hc| >= eps_dtm]      contribution (S0^2 - S1^2) / (E - H_aa)
//   sto : values = the five sums of solver.h:1093-1103, contribution of :1117-1124
// Stochastic iterations are independent: the host draws every iteration's sample with the
// reference's generator and distributions (std::default_random_engine, alias tables of
// src/util.cc:128-175), a chunk of iterations is processed in one device pass with the
// iteration index stored above the orbital bits of the key, and the reference's stopping
// rules are then applied iteration by iteration.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <numeric>
#include <queue>
#include <random>
#include <future>
#include <stack>
#include <thread>
#include <unordered_map>

#include "ctx.h"
#include "group.cuh"
#include "heatbath.cuh"
#include "kernels.h"
#include "walk.cuh"

namespace shci {

namespace {

constexpr int kPtWarps = 8;  // 8 warps per CTA; the walks are capped at 64 registers for
                              // four CTAs per SM (PT2 1.29 -> 1.26 s at n = 40)
enum : int { kDtm = 0, kPsto = 1, kSto = 2 };

struct PtParams {
  double eps;        // emission threshold |H_ai c_i| >= eps (and window eps / |c_i|)
  double eps_dtm;    // psto: second column threshold
  double eps_psto;   // sto: column split threshold
  uint64_t n_batches;
  uint64_t batch_magic;  // floor((2^64 - 1) / n_batches) for batch_of (set by set_batches)
  uint32_t low_mask;     // n_batches - 1 where the low bits of the hash are enough, else 0
  uint64_t batch;    // dtm / psto: the batch being computed
  double factor;     // sto: 1 / (n_samples - n_dtm - 1)
  int iter_shift;    // sto: bit position of the iteration index in the emitted up key
  int pilot;         // sto: sample-size pilot (only single excitations face the |H c| test)
};

// Stochastic sources: entry e = (det, iteration, count, weight, batch, deterministic?).  With
// ent_off, source m groups the entries [ent_off[m], ent_off[m+1]) of one det (its draws in the
// iterations of one device pass): the det's window is walked and each candidate hashed once,
// then tested against every entry's batch.  Without it, source m is entry m.
struct StoSources {
  const uint32_t* det;
  const uint32_t* iter;
  const double* count;
  const double* weight;
  const uint32_t* batch;
  const uint8_t* is_dtm;
  const uint32_t* ent_off;  // optional: entries of each source
};

__device__ __forceinline__ uint32_t ent_begin(const StoSources& S, uint32_t k) {
  return S.ent_off ? S.ent_off[k] : k;
}
__device__ __forceinline__ uint32_t ent_end(const StoSources& S, uint32_t k) {
  return S.ent_off ? S.ent_off[k + 1] : k + 1;
}

__device__ __forceinline__ uint32_t src_det(const StoSources& S, uint32_t k, int mode) {
  return mode == kSto ? S.det[ent_begin(S, k)] : k;
}

// h % n_batches exactly, without a 64-bit division: a mask for powers of two, else the
// quotient estimate floor(h * magic / 2^64) with magic = floor((2^64 - 1) / n_batches), which
// is at most 2 below the true quotient, corrected by subtraction.
__device__ __forceinline__ uint64_t batch_of(const PtParams& Q, uint64_t h) {
  const uint64_t nb = Q.n_batches;
  if ((nb & (nb - 1)) == 0) return h & (nb - 1);
  uint64_t r = h - __umul64hi(h, Q.batch_magic) * nb;
  if (r >= nb) r -= nb;
  if (r >= nb) r -= nb;
  return r;
}

void set_batches(PtParams& Q, uint64_t n_batches) {
  Q.n_batches = n_batches;
  Q.batch_magic = n_batches ? ~0ull / n_batches : 0;
  // Powers of two up to kLowBatches need only the low bits of the hash (55 instructions for 85): a
  // pseudo-stochastic batch of 16 at n = 40 5.3 -> 5.1 ms, six stochastic iterations 11.7 -> 11.4.
  const bool low = n_batches > 1 && n_batches <= kLowBatches && (n_batches & (n_batches - 1)) == 0;
  Q.low_mask = low ? static_cast<uint32_t>(n_batches - 1) : 0u;
}

// Window entries of each source: an upper bound of its candidates.
template <int MODE>
__global__ void __launch_bounds__(kPtWarps * 32, 4)
    k_pt_count(SelParams P, PtParams Q, StoSources S, uint32_t n_src, uint64_t* cnt_out) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t wpg = gridDim.x * kPtWarps;
  for (uint32_t k = blockIdx.x * kPtWarps + (threadIdx.x >> 5); k < n_src; k += wpg) {
    const uint32_t i = src_det(S, k, MODE);
    const double ac = fabs(P.coef[i]);
    const double eps_min = Q.eps / ac;
    const double eps_max = 1.0e100 / ac;
    const uint64_t up = P.up[i], dn = P.dn[i];
    uint64_t tot = 0;
    const int n_slots = P.n_elecs + P.n_pairs;
    for (int s0 = 0; s0 < n_slots; s0 += 32) {
      uint32_t lo = 0, c = 0;
      if (s0 + (int)lane < n_slots) slot_range(P, up, dn, s0 + lane, eps_min, eps_max, &lo, &c);
      uint64_t cc = c;
#pragma unroll
      for (int o = 16; o; o >>= 1) cc += __shfl_xor_sync(kFull, cc, o);
      tot += cc;
    }
    if (lane == 0) cnt_out[k] = tot;
  }
}

template <int MODE>
constexpr int n_cols() {
  return MODE == kDtm ? 1 : MODE == kPsto ? 2 : 5;
}

// Single-excitation elements in 64-bit fixed point.  H_ij of a single excitation p -> q is
// +-(h_pq + sum_o (pq|oo) [2 (pq|oo) for a doubly occupied o] - sum_o (po|oq)), about 2 n_e
// table entries (chem_system.cc:544-577); in FP64 that chain of dependent additions kept
// the FP64 pipe (about two operations per SM cycle on GB300) half busy in the emission.  Here
// every entry is rounded once to a multiple of 2^-s and the sum is exact on the integer pipe;
// |fixed - FP64| <= margin (entry rounding plus the FP64 evaluation's own rounding).  A
// value within margin |c_i| of a threshold is formed again in FP64, so every keep / split
// decision is the FP64 one; kept values differ from it by at most margin |c_i|.
struct SingleFix {
  const long long* h1;  // [n*n]
  const long long* d;   // [n^3] (pq|oo) at (p n + q) n + o
  const long long* x;   // [n^3] (po|oq) at (p n + q) n + o
  int n;
  double inv_scale;     // 2^-s
  double margin;
};

__device__ __forceinline__ double h_one_fix(const SingleFix& F, uint64_t ui, uint64_t di,
                                            uint64_t uj, uint64_t dj) {
  const uint64_t xu = ui ^ uj;
  const bool alpha = xu != 0;
  const uint64_t si = alpha ? ui : di, sj = alpha ? uj : dj;
  uint64_t oppo = alpha ? di : ui;
  const uint64_t x = si ^ sj;
  const int oi = ctz64(si & x), oj = ctz64(sj & x);
  const int n = F.n;
  const size_t row = (size_t)(oi * n + oj) * n;
  const long long* D = F.d + row;
  const long long* X = F.x + row;
  long long e = __ldg(F.h1 + oi * n + oj);
  for (uint64_t m = si & ~(1ull << oi) & ~(1ull << oj); m; m &= m - 1) {
    const int o = ctz64(m);
    e -= __ldg(X + o);
    const long long dd = __ldg(D + o);
    if (oppo >> o & 1) {
      oppo &= ~(1ull << o);
      e += 2 * dd;
    } else {
      e += dd;
    }
  }
  for (uint64_t m = oppo; m; m &= m - 1) e += __ldg(D + ctz64(m));
  return flip_sign(static_cast<double>(e) * F.inv_scale, move_parity(si, oi, oj));
}

// A piece of a source's window: entries [begin, begin + len) of its slots' ranges in walk order.
// Its members go to out[off[p], off[p] + cnt[p]), densely; cnt may come out larger than the
// region, whose excess is then not written (the caller emits that piece again).
struct PtPieces {
  const uint32_t* src;
  const uint32_t* begin;
  const uint32_t* len;
  const uint64_t* off;  // [n + 1]
  uint32_t* cnt;
  uint32_t* work;  // pieces taken so far
  uint32_t n;
  uint64_t base;  // off of the output arrays' first entry
};

constexpr uint32_t kPtQ = 64;    // queue lengths (< 32 waiting + 32 pushed)

struct PtWarp {
  WalkWarp w;
  // stage 1 queue: entries whose targets are free (x: slot code with the targets, y: piece)
  uint2 a[kPtQ];
  // stage 2 queue (several batches): members
  uint64_t b_u[kPtQ], b_d[kPtQ];
  uint32_t b_piece[kPtQ];
  uint8_t b_ent[kPtQ];
};

// Emits the members of each piece into its region: the window entries whose targets are free, that
// fall in the current hash batch, are not variational and have |H_ai c_i| >= eps (the handler's
// order, solver.h:703-713).  A warp takes a piece at a time.
//
// Most window entries go to occupied orbitals (four of five at n = 40, 10 alpha + 10 beta: the
// large |H| couple neighbouring orbitals), and one candidate in n_batches is in the batch, so the
// work is done in three stages, each on full warps: stage 1 tests the targets of 32 entries
// against the source's strings and queues what passes; stage 2 builds 32 of those determinants and,
// with several batches, hashes them and queues the members; the last stage evaluates 32 members.
// Queues carry over from piece to piece.  Members keep their walk order within a piece.
// Warps take pieces from a counter, the next one while they walk (a fixed share left a tenth of the
// chip idle: 26.3 -> 24.4 ms over the stages of an n = 40 run).
// At n = 40, 40,000 dets: 19.4 -> 4.1 ms deterministic (297M window entries), 11.3 -> 4.0 ms a
// pseudo-stochastic batch of 16 (walk and hash are most of the work left), 21.4 -> 8.6 ms for six
// stochastic iterations; n = 26, 30,000 dets: 5.3 -> 1.3 ms, of which the heaviest determinant's
// window on one warp had been half.  (Before: build and hash at the walk, an output slot for
// every window entry, a warp per source.)
template <int MODE>
__global__ void __launch_bounds__(kPtWarps * 32, 4)
    k_pt_emit(SelParams P, PtParams Q, StoSources S, SingleFix F, PtPieces pc,
              PtRec<n_cols<MODE>()>* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char pt_smem[];
  PtWarp& W = reinterpret_cast<PtWarp*>(pt_smem)[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t ah = 0, an = 0, bh = 0, bn = 0;           // warp-uniform ring states
  uint32_t run_piece = 0xffffffffu, run_cnt = 0;      // kept members of the last piece seen

  // Last stage: evaluates the lanes' members (piece 0xffffffff: no member) and writes the kept
  // ones.  A piece's members arrive in order, over one or several calls (one entry's, in the
  // stochastic stage).
  auto finish = [&](uint32_t piece, uint64_t cu, uint64_t cd, uint32_t ent) {
    const bool act = piece != 0xffffffffu;
    bool ok = false;
    double hc = 0.0, count = 1.0, weight = 1.0;
    bool dtm_src = true;
    uint64_t iter_tag = 0;
    if (act) {
      const uint32_t kk = pc.src[piece];
      const uint32_t i = src_det(S, kk, MODE);
      if (MODE == kSto) {
        const uint32_t e = ent_begin(S, kk) + ent;
        dtm_src = S.is_dtm[e] != 0;
        count = dtm_src ? 1.0 : S.count[e];
        weight = dtm_src ? 1.0 : S.weight[e];
        iter_tag = static_cast<uint64_t>(S.iter[e]) << Q.iter_shift;
      }
      ok = !in_set(P, cu, cd);
      // the pilot's handler tests |H_ai c_i| for single excitations only (solver.h:958-962)
      const uint64_t up = P.up[i], dn = P.dn[i];
      const bool one = popc64(up ^ cu) + popc64(dn ^ cd) == 2;
      if (ok && (MODE != kSto || !Q.pilot || one)) {
        const double coef = P.coef[i];
        if (one) {
          hc = h_one_fix(F, up, dn, cu, cd) * coef;
          const double a = fabs(hc), m = F.margin * fabs(coef);
          bool near = fabs(a - Q.eps) <= m;
          if (MODE == kPsto) near = near || fabs(a - Q.eps_dtm) <= m;
          if (MODE == kSto) near = near || fabs(a - Q.eps_psto) <= m;
          if (near) hc = h_one(P.I, up, dn, cu, cd) * coef;
        } else {
          hc = h_two(P.I, up, dn, cu, cd) * coef;
        }
        if (fabs(hc) < Q.eps) ok = false;
      }
    }
    const unsigned keep = __ballot_sync(kFull, ok);
    const unsigned mates = __match_any_sync(kFull, piece);
    uint32_t before, after;
    if (MODE == kSto) {
      // members of several pieces alternate (an entry of each in turn): the count so far is read
      const int lead = __ffs(mates) - 1;
      before = 0;
      if (act && static_cast<int>(lane) == lead)
        before = atomicAdd(&pc.cnt[piece], static_cast<uint32_t>(__popc(keep & mates)));
      before = __shfl_sync(kFull, before, lead);
      after = 0;
    } else {
      before = piece == run_piece ? run_cnt : 0u;
      after = before + __popc(keep & mates);
    }
    if (ok) {
      uint64_t pos = pc.off[piece] + before + __popc(keep & mates & lt);
      if (pos < pc.off[piece + 1]) {
        pos -= pc.base;
        PtRec<n_cols<MODE>()> r{};
        r.u = cu | iter_tag;
        r.d = cd;
        r.v[0] = hc;
        if constexpr (MODE == kPsto) r.v[1] = fabs(hc) >= Q.eps_dtm ? hc : 0.0;
        if constexpr (MODE == kSto) {
          // solver.h:1093-1103
          const double x = count * hc / weight;
          const bool above = fabs(hc) > Q.eps_psto;
          double v2 = 0.0, v3 = 0.0, v4 = 0.0;
          if (!dtm_src) {
            v2 = count * hc / weight * sqrt(Q.factor);
            if (above) v3 = v2;
            else v4 = x * x * (1. - weight / count + Q.factor);
          }
          r.v[0] = x;
          r.v[1] = above ? x : 0.0;
          r.v[2] = v2;
          r.v[3] = v3;
          r.v[4] = v4;
        }
        out[pos] = r;
      }
    }
    if (MODE != kSto) {
      if (act && lane == 31u - __clz(mates)) pc.cnt[piece] = after;  // the running count
      const int last = 31 - __clz(__ballot_sync(kFull, act));
      run_piece = __shfl_sync(kFull, piece, last);
      run_cnt = __shfl_sync(kFull, after, last);
    }
  };

  auto drain_b = [&](uint32_t m) {
    __syncwarp();
    const uint32_t sl = (bh + lane) & (kPtQ - 1);
    const bool act = lane < m;
    const uint32_t piece = act ? W.b_piece[sl] : 0xffffffffu;
    const uint64_t cu = act ? W.b_u[sl] : 0, cd = act ? W.b_d[sl] : 0;
    const uint32_t ent = act ? W.b_ent[sl] : 0;
    __syncwarp();
    bh += m;
    bn -= m;
    finish(piece, cu, cd, ent);
  };

  // Stage 2: the m oldest entries of stage 1's queue.
  auto drain_a = [&](uint32_t m) {
    __syncwarp();
    const uint32_t sl = (ah + lane) & (kPtQ - 1);
    const bool act = lane < m;
    const uint2 entry = W.a[sl];
    const uint32_t piece = act ? entry.y : 0xffffffffu, code = entry.x;
    __syncwarp();
    ah += m;
    an -= m;
    uint64_t cu = 0, cd = 0;
    uint32_t kk = 0;
    if (act) {
      kk = pc.src[piece];
      const uint32_t i = src_det(S, kk, MODE);
      cu = P.up[i];
      cd = P.dn[i];
      apply_entry(code, &cu, &cd);
    }
    if (Q.n_batches <= 1) {
      if (MODE != kSto) {
        finish(piece, cu, cd, 0);
        return;
      }
    }
    uint64_t b = 0;
    if (Q.low_mask) b = batch_hash_low(cu, cd) & Q.low_mask;
    else if (Q.n_batches > 1) b = batch_of(Q, rehash(det_hash(cu, cd)));
    uint32_t e0 = 0, ne = act ? 1u : 0u;
    if (MODE == kSto && act) {
      e0 = ent_begin(S, kk);
      ne = ent_end(S, kk) - e0;
    }
    const uint32_t most = MODE == kSto ? __reduce_max_sync(kFull, ne) : 1u;
    for (uint32_t e = 0; e < most; e++) {
      const bool mine =
          e < ne && (Q.n_batches <= 1 || b == (MODE == kSto ? S.batch[e0 + e] : Q.batch));
      const unsigned bal = __ballot_sync(kFull, mine);
      if (!bal) continue;
      if (mine) {
        const uint32_t t = (bh + bn + __popc(bal & lt)) & (kPtQ - 1);
        W.b_u[t] = cu;
        W.b_d[t] = cd;
        W.b_piece[t] = piece;
        W.b_ent[t] = static_cast<uint8_t>(e);
      }
      bn += __popc(bal);
      if (bn >= 32u) drain_b(32u);
    }
  };

  // Queues the lanes' entries that passed.
  auto push_a = [&](bool pass, uint32_t x, uint32_t piece) {
    const unsigned bal = __ballot_sync(kFull, pass);
    if (!bal) return;
    if (pass) W.a[(ah + an + __popc(bal & lt)) & (kPtQ - 1)] = make_uint2(x, piece);
    an += __popc(bal);
    if (an >= 32u) drain_a(32u);
  };

  uint32_t next = 0;  // (lane 0) taken while the piece before is walked
  if (lane == 0) next = atomicAdd(pc.work, 1u);
  for (;;) {
    const uint32_t piece = __shfl_sync(kFull, next, 0);
    if (piece >= pc.n) break;
    if (lane == 0) next = atomicAdd(pc.work, 1u);
    const uint32_t kk = pc.src[piece];
    const uint32_t skip = pc.begin[piece], left = pc.len[piece];
    const uint32_t i = src_det(S, kk, MODE);
    const double ac = fabs(P.coef[i]);
    const double eps_min = Q.eps / ac;
    const double eps_max = 1.0e100 / ac;
    const uint64_t up = P.up[i], dn = P.dn[i];
    walk_window(P, W.w, up, dn, eps_min, eps_max, skip, left,
                [&](bool, bool free, uint32_t x, uint32_t) { push_a(free, x, piece); });
  }
  while (an) drain_a(an < 32u ? an : 32u);
  while (bn) drain_b(bn < 32u ? bn : 32u);
}

// Members of each piece that were written: none of one whose region was too small (*over counts
// those).
__global__ void k_pt_kept(const uint32_t* __restrict__ cnt, const uint64_t* __restrict__ off,
                          uint32_t n, uint64_t* __restrict__ kept, unsigned* over) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const bool fits = cnt[p] <= off[p + 1] - off[p];
    kept[p] = fits ? cnt[p] : 0u;
    if (!fits) atomicAdd(over, 1u);
  }
}

// Copies each piece's members from its region to dst[p] (eight lanes a piece: most pieces hold
// a few members when there are many batches).
template <int NV>
__global__ void __launch_bounds__(256)
    k_pt_collect(const uint64_t* __restrict__ off, uint64_t base, const uint64_t* __restrict__ dst,
                 const uint64_t* __restrict__ total, uint32_t n, const PtRec<NV>* __restrict__ rec,
                 PtRec<NV>* __restrict__ out) {
  constexpr uint64_t W = sizeof(PtRec<NV>) / sizeof(uint4);
  const uint4* __restrict__ in = reinterpret_cast<const uint4*>(rec);
  uint4* __restrict__ o = reinterpret_cast<uint4*>(out);
  const unsigned sub = threadIdx.x & 7;
  const uint32_t step = gridDim.x * (blockDim.x >> 3);
  for (uint32_t p = blockIdx.x * (blockDim.x >> 3) + (threadIdx.x >> 3); p < n; p += step) {
    const uint64_t a = (off[p] - base) * W, b = dst[p] * W;
    const uint64_t m = (p + 1 < n ? dst[p + 1] : *total) * W - b;
    for (uint64_t k = sub; k < m; k += 8) o[b + k] = in[a + k];
  }
}

// Diagonal H_aa of the PT dets in 64-bit fixed point.  The diagonal is a sum of about
// n_e^2 / 2 table entries (h_pp, J - K for same-spin pairs, J for opposite-spin pairs,
// chem_system.cc:495-542); on GB300 the FP64 pipe retires about two operations per SM cycle,
// so ~300 FP64 additions per PT det made the contribution kernel FP64-bound.  Here every
// entry is rounded once to a multiple of 2^-s (s chosen so that no sum can reach 2^62) and the
// sum is an exact integer sum on the integer pipe: |error| <= (number of terms) * 2^-(s+1),
// about 1e-13 Ha at n = 40 (s = 51), where the FP64 sum carries a comparable rounding error.
//
// A sum of integers may be taken in any order without changing it, so a det is summed from the
// filling of the lowest orbitals: of the D orbitals that differ from it, the energies in its field
// (a hole's negative) and the pairs among them, D (D + 1) / 2 entries (36 for a fourfold excitation)
// against n_e (n_e + 1) / 2 (210 for 20 electrons).  A det that differs in n_e orbitals or more is
// summed directly.  (Sums may wrap on the way; the last one is in range.)  Contributions of an
// n = 40 run with 20 electrons: 3.9 -> 1.65 ms over its stages, 0.26 -> 0.22 ms at n = 26 with 14
// (where the FP64 division and the reads of the records weigh more).
struct DiagFix {
  const long long* tab;  // [n] h_pp, [n*n] J - K, [n*n] J, [n] and [n] alpha and beta energies
  int n;
  double inv_scale;      // 2^-s
  double e_core;
  uint64_t ref_up, ref_dn;
  unsigned long long e_ref;
};

// Sum of the entries of a row over the orbitals of `plus` less that over those of `minus`.
__device__ __forceinline__ unsigned long long row_sum(const long long* __restrict__ row,
                                                      uint64_t plus, uint64_t minus) {
  unsigned long long t = 0;
  for (; plus; plus &= plus - 1) t += __ldg(row + ctz64(plus));
  for (; minus; minus &= minus - 1) t -= __ldg(row + ctz64(minus));
  return t;
}

__device__ __forceinline__ double h_diag_fix(const DiagFix& F, uint64_t up, uint64_t dn) {
  const int n = F.n;
  const long long* jk = F.tab + n;
  const long long* jj = jk + n * n;
  uint64_t xu = up ^ F.ref_up, xd = dn ^ F.ref_dn;
  unsigned long long acc = F.e_ref;
  const long long *eu = jj + n * n, *ed = eu + n;
  if (popc64(xu) + popc64(xd) >= popc64(up) + popc64(dn)) {
    xu = up;
    xd = dn;
    acc = 0;
    eu = ed = F.tab;
  }
  for (uint64_t m = xu; m; m &= m - 1) {
    const int a = ctz64(m);
    const uint64_t rest = m & (m - 1);
    const unsigned long long t = __ldg(eu + a) + row_sum(jk + a * n, rest & up, rest & ~up) +
                                 row_sum(jj + a * n, xd & dn, xd & ~dn);
    acc += (up >> a & 1) ? t : 0ull - t;
  }
  for (uint64_t m = xd; m; m &= m - 1) {
    const int a = ctz64(m);
    const uint64_t rest = m & (m - 1);
    const unsigned long long t = __ldg(ed + a) + row_sum(jk + a * n, rest & dn, rest & ~dn);
    acc += (dn >> a & 1) ? t : 0ull - t;
  }
  return static_cast<double>(static_cast<long long>(acc)) * F.inv_scale + F.e_core;
}

// x[k] = contribution of unique PT det k (mapper of solver.h:727-732, 856-862, 1117-1124)
template <int MODE>
__global__ void k_pt_x(DiagFix D, const PtRec<n_cols<MODE>()>* __restrict__ rec, size_t m,
                       double e_var, double n_batches, uint64_t orb_mask, double* x) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    const PtRec<n_cols<MODE>()> r = rec[k];
    const double haa = h_diag_fix(D, r.u & orb_mask, r.d);
    double v;
    if constexpr (MODE == kDtm) {
      v = r.v[0] * r.v[0] / (e_var - haa);
    } else if constexpr (MODE == kPsto) {
      const double d = r.v[0] * r.v[0] - r.v[1] * r.v[1];
      v = d / (e_var - haa);
    } else {
      const double f = n_batches / (e_var - haa);
      v = (r.v[0] * r.v[0] - r.v[1] * r.v[1] + r.v[2] * r.v[2] - r.v[3] * r.v[3] - r.v[4]) * f;
    }
    x[k] = v;
  }
}

// Sums of x and x^2 over segments [starts[g], starts[g+1]) in a fixed order (the map-reduce of
// solver.h:1155-1177, whose thread-local FP64 sums this replaces): pass 1 reduces chunks of
// kRedChunk elements of each segment (block (chunk, g)), pass 2 reduces each segment's chunk
// partials.  Every partial is a compensated double-double sum (Dd), so the result does not
// lose accuracy with the number of PT dets (1e8 and more); only the chunking fixes the order,
// so results are reproducible.
// A chunk is 32 elements a thread: chunks of 65,536 elements left two thirds of the chip idle below
// 10M determinants (0.89 -> 0.57 ms for 12.6M, 0.46 -> 0.11 ms for 1.9M).
constexpr uint32_t kRedChunk = 1u << 13;

__device__ __forceinline__ void block_sum2(Dd* a, Dd* b) {
  __shared__ Dd s1[8], s2[8];
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    *a = dd_add(*a, dd_shfl_xor(*a, o));
    *b = dd_add(*b, dd_shfl_xor(*b, o));
  }
  if ((threadIdx.x & 31) == 0) {
    s1[threadIdx.x >> 5] = *a;
    s2[threadIdx.x >> 5] = *b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Dd ta, tb;
    for (int w = 0; w < 8; w++) {
      ta = dd_add(ta, s1[w]);
      tb = dd_add(tb, s2[w]);
    }
    *a = ta;
    *b = tb;
  }
}

__global__ void __launch_bounds__(256)
    k_seg_partial2(const double* __restrict__ x, const uint64_t* __restrict__ starts,
                   uint32_t n_chunks, double* part) {
  const uint32_t g = blockIdx.y, ch = blockIdx.x;
  const uint64_t b0 = starts[g] + (uint64_t)ch * kRedChunk;
  const uint64_t e = starts[g + 1];
  const uint64_t b1 = b0 + kRedChunk < e ? b0 + kRedChunk : e;
  // a thread's sums with the rounding errors of their additions kept apart (added up in FP64 and
  // joined at the end: 16 FP64 operations an element instead of 24)
  Dd a, b;
  for (uint64_t k = b0 + threadIdx.x; k < b1; k += blockDim.x) {
    const double v = x[k];
    double e;
    two_sum64(a.hi, v, &a.hi, &e);
    a.lo += e;
    // v^2 as an exact product pair: sq rounded, its FMA error
    const double sq = v * v;
    two_sum64(b.hi, sq, &b.hi, &e);
    b.lo += e + fma(v, v, -sq);
  }
  a = dd_add(a, 0.0);
  b = dd_add(b, 0.0);
  block_sum2(&a, &b);
  if (threadIdx.x == 0) {
    double* o = part + 4 * ((size_t)g * n_chunks + ch);
    o[0] = a.hi;
    o[1] = a.lo;
    o[2] = b.hi;
    o[3] = b.lo;
  }
}

__global__ void __launch_bounds__(256)
    k_seg_final2(const double* __restrict__ part, uint32_t n_chunks, double* out) {
  const uint32_t g = blockIdx.x;
  Dd a, b;
  for (uint32_t k = threadIdx.x; k < n_chunks; k += blockDim.x) {
    const double* p = part + 4 * ((size_t)g * n_chunks + k);
    Dd ta, tb;
    ta.hi = p[0];
    ta.lo = p[1];
    tb.hi = p[2];
    tb.lo = p[3];
    a = dd_add(a, ta);
    b = dd_add(b, tb);
  }
  block_sum2(&a, &b);
  if (threadIdx.x == 0) {
    out[2 * g] = a.hi + a.lo;
    out[2 * g + 1] = b.hi + b.lo;
  }
}

}  // namespace

// out[2g], out[2g+1] = sum, sum of squares of x over segment g (total length m).
void seg_reduce2(shci_ctx* c, const double* x, const uint64_t* starts, uint32_t nseg, size_t m,
                 double* out) {
  cudaStream_t s = c->stream;
  const uint32_t n_chunks = static_cast<uint32_t>((m + kRedChunk - 1) / kRedChunk) + 1;
  DevBuf<double> part;
  part.mt = &c->mem;
  part.resize(4 * (size_t)n_chunks * nseg);
  k_seg_partial2<<<dim3(n_chunks, nseg), 256, 0, s>>>(x, starts, n_chunks, part.p);
  SHCI_LAUNCH_CHECK();
  k_seg_final2<<<nseg, 256, 0, s>>>(part.p, n_chunks, out);
  SHCI_LAUNCH_CHECK();
  SHCI_CUDA(cudaStreamSynchronize(s));
  c->launches += 2;
}

namespace {

// starts[it] = first k with (rec[k].u >> shift) >= it, for it = 0..n_it (tags ascending)
__global__ void k_iter_starts(const PtRec<5>* rec, size_t m, int shift, uint32_t n_it,
                              uint64_t* starts) {
  const uint32_t it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it > n_it) return;
  size_t lo = 0, hi = m;
  while (lo < hi) {
    const size_t mid = (lo + hi) >> 1;
    if ((rec[mid].u >> shift) < it) lo = mid + 1;
    else hi = mid;
  }
  starts[it] = lo;
}

// Fixed-point diagonal tables of the context's integrals (built once per set of integrals).
DiagFix diag_fix(shci_ctx* c) {
  const auto& I = c->I;
  const int n = static_cast<int>(I.n);
  if (!c->dfix_valid) {
    std::vector<double> v(n + 2 * (size_t)n * n, 0.0);
    for (int p = 0; p < n; p++) v[p] = I.h(p, p);
    for (int a = 0; a < n; a++)
      for (int b = 0; b < n; b++) {
        const double J = I.g(a, a, b, b), K = I.g(a, b, b, a);
        v[n + (size_t)a * n + b] = J - K;
        v[n + (size_t)n * n + (size_t)a * n + b] = J;
      }
    double mx = 0.0;
    for (double x : v) mx = std::max(mx, std::fabs(x));
    const int n_e = static_cast<int>(I.n_up + I.n_dn);
    const double bound = (static_cast<double>(n_e) + static_cast<double>(n_e) * n_e) * mx;
    int s = 60;
    while (s > 0 && bound * std::ldexp(1.0, s) >= std::ldexp(1.0, 62)) s--;
    std::vector<long long> t(v.size() + 2 * n);
    for (size_t k = 0; k < v.size(); k++) t[k] = std::llround(std::ldexp(v[k], s));
    // energies in the field of the lowest filling (unsigned: they may wrap), and its own
    const long long *jk = t.data() + n, *jj = jk + (size_t)n * n;
    unsigned long long e_ref = 0;
    for (int sp = 0; sp < 2; sp++) {
      const int same = static_cast<int>(sp ? I.n_dn : I.n_up);
      const int other = static_cast<int>(sp ? I.n_up : I.n_dn);
      for (int a = 0; a < n; a++) {
        unsigned long long e = t[a];
        for (int b = 0; b < same; b++)
          if (b != a) e += jk[(size_t)a * n + b];
        for (int b = 0; b < other; b++) e += jj[(size_t)a * n + b];
        t[v.size() + (size_t)sp * n + a] = static_cast<long long>(e);
      }
      for (int a = 0; a < same; a++) {
        e_ref += t[a];
        for (int b = 0; b < a; b++) e_ref += jk[(size_t)a * n + b];
        for (int b = 0; sp == 0 && b < other; b++) e_ref += jj[(size_t)a * n + b];
      }
    }
    c->dfix_ref = e_ref;
    c->dfix.mt = &c->mem;
    c->dfix.resize(t.size());
    SHCI_CUDA(cudaMemcpyAsync(c->dfix.p, t.data(), t.size() * 8, cudaMemcpyHostToDevice,
                              c->stream));
    SHCI_CUDA(cudaStreamSynchronize(c->stream));
    c->dfix_scale = s;
    c->dfix_valid = true;
  }
  auto lowest = [](unsigned k) { return k >= 64 ? ~0ull : (1ull << k) - 1ull; };
  return DiagFix{c->dfix.p,      n,           std::ldexp(1.0, -c->dfix_scale), I.e_core,
                 lowest(I.n_up), lowest(I.n_dn), c->dfix_ref};
}

// Fixed-point single-excitation tables (built with the diagonal tables, once per set of
// integrals).  Scale: the largest |sum| (h_pq plus at most 2 n_e entries, doubled ones
// counted twice) stays below 2^62.  margin = the rounding of the entries (2^-(s+1) each,
// twice for a doubled one) + the FP64 evaluation's rounding (each of its <= 2 n_e + 1
// additions within 2^-53 of a partial sum <= bound) + the final product by c_i, generously.
SingleFix single_fix(shci_ctx* c) {
  const auto& I = c->I;
  const int n = static_cast<int>(I.n);
  // new integrals invalidate the diagonal tables; rebuild these with them
  const bool stale = !c->dfix_valid || c->sfix.n != (size_t)n * n + 2 * (size_t)n * n * n;
  diag_fix(c);
  if (stale) {
    const size_t n2 = (size_t)n * n, n3 = n2 * n;
    std::vector<double> v(n2 + 2 * n3, 0.0);
    for (int p = 0; p < n; p++)
      for (int q = 0; q < n; q++) {
        v[(size_t)p * n + q] = I.h(p, q);
        for (int o = 0; o < n; o++) {
          v[n2 + ((size_t)p * n + q) * n + o] = I.g(p, q, o, o);
          v[n2 + n3 + ((size_t)p * n + q) * n + o] = I.g(p, o, o, q);
        }
      }
    double mh = 0.0, mt = 0.0;
    for (size_t k = 0; k < n2; k++) mh = std::max(mh, std::fabs(v[k]));
    for (size_t k = n2; k < v.size(); k++) mt = std::max(mt, std::fabs(v[k]));
    const int n_e = static_cast<int>(I.n_up + I.n_dn);
    const double terms = 3.0 * n_e + 1.0;  // bound on the number of entries, doubles twice
    const double bound = mh + terms * mt;
    int s = 60;
    while (s > 0 && bound * std::ldexp(1.0, s) >= std::ldexp(1.0, 62)) s--;
    std::vector<long long> t(v.size());
    for (size_t k = 0; k < v.size(); k++) t[k] = std::llround(std::ldexp(v[k], s));
    c->sfix.mt = &c->mem;
    c->sfix.resize(t.size());
    SHCI_CUDA(cudaMemcpyAsync(c->sfix.p, t.data(), t.size() * 8, cudaMemcpyHostToDevice,
                              c->stream));
    SHCI_CUDA(cudaStreamSynchronize(c->stream));
    c->sfix_scale = s;
    c->sfix_margin = 4.0 * (terms * std::ldexp(1.0, -(s + 1)) + terms * bound * std::ldexp(1.0, -52));
  }
  const size_t n2 = (size_t)n * n, n3 = n2 * n;
  return SingleFix{c->sfix.p, c->sfix.p + n2, c->sfix.p + n2 + n3, n,
                   std::ldexp(1.0, -c->sfix_scale), c->sfix_margin};
}

struct PtSetup {
  SelParams P{};
  DevBuf<uint32_t> pairs;
  unsigned grid = 0;
};

void pt_setup(shci_ctx* c, PtSetup& st) {
  if (!c->Q.built) throw ArgError("heat-bath queues not built (call shci_build_queues)");
  HostScope hs(c->prof, "pt2_host_pt_setup");
  sync_dets(c);
  cudaStream_t s = c->stream;
  const int n_elecs = static_cast<int>(c->I.n_up + c->I.n_dn);
  rebuild_det_set(c);
  std::vector<uint32_t> pairs;
  for (int a = 0; a < n_elecs; a++)
    for (int b = a + 1; b < n_elecs; b++) pairs.push_back(a | (b << 16));
  st.pairs.mt = &c->mem;
  st.pairs.resize(pairs.empty() ? 1 : pairs.size());
  if (!pairs.empty())
    SHCI_CUDA(cudaMemcpyAsync(st.pairs.p, pairs.data(), pairs.size() * 4, cudaMemcpyHostToDevice, s));
  SelParams& P = st.P;
  P.I = c->dI;
  P.up = c->d_up.p;
  P.dn = c->d_dn.p;
  P.coef = c->d_coef.p;
  P.d_off = c->Q.d_off.p;
  P.d_H = c->Q.d_H.p;
  P.d_rs = c->Q.d_rs.p;
  P.s_off = c->Q.s_off.p;
  P.s_S = c->Q.s_S.p;
  P.s_r = c->Q.s_r.p;
  P.pair_tab = st.pairs.p;
  P.set_hash = c->set_hash.p;
  P.set_hash_mask = c->set_hash_mask;
  P.max_hci = c->Q.max_hci;
  P.max_singles = c->Q.max_singles;
  P.n_orbs = c->I.n;
  P.n_up = static_cast<int>(c->I.n_up);
  P.n_elecs = n_elecs;
  P.n_pairs = static_cast<int>(pairs.size());
  P.no_doubles = c->has_doubles ? 0 : 1;
  P.inactive = c->inactive_orbs;
  int sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  st.grid = static_cast<unsigned>(sms) * 8u;
}

// Pieces by host arrays (those to be emitted again), with exact sizes.
struct PieceRerun {
  std::vector<uint32_t> src, begin, len;
  std::vector<uint64_t> off{0};
};

// Region estimate with several batches: SHCI_PT_SLOTS="slack,pad" replaces 1.3 and 64.
void make_pt_pieces(shci_ctx* c, const DevBuf<uint64_t>& entries, uint32_t n_src,
                    uint64_t n_batches, const uint32_t* ent_off, PieceList& L) {
  double slack = 1.3, pad = 64.0;
  if (const char* e = std::getenv("SHCI_PT_SLOTS")) std::sscanf(e, "%lf,%lf", &slack, &pad);
  HostScope hs(c->prof, "pt2_host_offsets");
  make_pieces(c, entries, n_src, n_batches, slack, pad, ent_off, L);
}

// Emits the members of the pieces for one batch (or set of iterations), appending them to rec
// after the first *bn.  Pieces whose region overflowed are appended to *over with their
// exact sizes.  The accumulation is sorted and reduced in place whenever it grows past kCap, to
// keep it bounded.
template <int MODE>
void pt_emit_append(shci_ctx* c, PtSetup& st, const PtParams& Q, const StoSources& S,
                    const PieceList& L, DevBuf<PtRec<n_cols<MODE>()>>& rec, size_t* bn,
                    int tag_bits, PieceRerun* over) {
  constexpr int NV = n_cols<MODE>();
  cudaStream_t s = c->stream;
  const uint64_t kCap = 1ull << 27;
  uint64_t run = kCap;  // regions of a launch at most; fewer where these find no room
  DevBuf<PtRec<NV>> out;
  DevBuf<uint64_t> d_dst;
  DevBuf<uint32_t> d_cnt;
  out.mt = &c->mem;
  d_dst.mt = &c->mem;
  d_cnt.mt = &c->mem;
  const SingleFix F = single_fix(c);
  const size_t smem = sizeof(PtWarp) * kPtWarps;
  SHCI_CUDA(cudaFuncSetAttribute(k_pt_emit<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
  size_t k0 = 0;
  uint64_t base = 0;  // off[k0]
  while (k0 < L.n) {
    uint64_t end = 0;
    const size_t k1 = piece_run(c, L, k0, base, run, &end);
    const uint64_t tot = end - base;
    const uint32_t n = static_cast<uint32_t>(k1 - k0);
    try {
      out.resize(std::max<uint64_t>(tot, 1), 1.25);
    } catch (const OomError&) {
      if (n == 1 || tot <= kCap >> 8) throw;
      run = std::max(tot / 4, kCap >> 8);
      continue;
    }
    d_cnt.resize((size_t)n + 2);  // (the overflow count and the pieces taken after the pieces' counts)
    d_dst.resize((size_t)n + 1);
    SHCI_CUDA(cudaMemsetAsync(d_cnt.p, 0, ((size_t)n + 2) * 4, s));
    const PtPieces pc{L.src.p + k0, L.begin.p + k0, L.len.p + k0, L.off.p + k0, d_cnt.p,
                      d_cnt.p + n + 1, n, base};
    {
      ProfScope ps(c->prof, s, "pt2_emit");
      k_pt_emit<MODE><<<grid_for((size_t)n * 32, kPtWarps * 32, st.grid / 2), kPtWarps * 32, smem, s>>>(
          st.P, Q, S, F, pc, out.p);
      SHCI_LAUNCH_CHECK();
    }
    uint64_t got = 0;
    unsigned n_over = 0;
    {
      ProfScope ps(c->prof, s, "pt2_compact");
      k_pt_kept<<<grid_for(n, 256), 256, 0, s>>>(d_cnt.p, pc.off, n, d_dst.p, d_cnt.p + n);
      SHCI_LAUNCH_CHECK();
      exclusive_scan_u64_async(d_dst.p, d_dst.p, n, s, c->sort, d_dst.p + n);
      SHCI_CUDA(cudaMemcpyAsync(&got, d_dst.p + n, 8, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaMemcpyAsync(&n_over, d_cnt.p + n, 4, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaStreamSynchronize(s));
      if (got) {
        rec.n = *bn;
        rec.grow_keep(*bn + got, s);
        k_pt_collect<NV><<<grid_for((size_t)n * 8, 256), 256, 0, s>>>(
            pc.off, base, d_dst.p, d_dst.p + n, n, out.p, rec.p + *bn);
        SHCI_LAUNCH_CHECK();
        *bn += got;
      }
    }
    c->launches += 5;
    if (n_over) {
      std::vector<uint32_t> cnt(n), src(n), begin(n), len(n);
      std::vector<uint64_t> off((size_t)n + 1);
      SHCI_CUDA(cudaMemcpyAsync(cnt.data(), d_cnt.p, n * 4ull, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaMemcpyAsync(src.data(), pc.src, n * 4ull, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaMemcpyAsync(begin.data(), pc.begin, n * 4ull, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaMemcpyAsync(len.data(), pc.len, n * 4ull, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaMemcpyAsync(off.data(), pc.off, (n + 1ull) * 8, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaStreamSynchronize(s));
      for (uint32_t k = 0; k < n; k++)
        if (cnt[k] > off[k + 1] - off[k]) {
          over->src.push_back(src[k]);
          over->begin.push_back(begin[k]);
          over->len.push_back(len[k]);
          over->off.push_back(over->off.back() + cnt[k]);
        }
    }
    if (*bn > kCap)  // keep the accumulation buffer bounded
      *bn = group_records<NV>(c, rec, *bn, st.P.n_orbs, tag_bits);
    k0 = k1;
    base = end;
  }
}

// Emits and reduces the members of the pieces for one batch / set of iterations; returns the
// number of distinct dets, which rec then holds.  Pieces whose estimated
// region overflowed are emitted again, after the others, with the sizes they turned out to have.
template <int MODE>
size_t pt_emit_reduce(shci_ctx* c, PtSetup& st, const PtParams& Q, const StoSources& S,
                      const PieceList& L, DevBuf<PtRec<n_cols<MODE>()>>& rec, int tag_bits) {
  constexpr int NV = n_cols<MODE>();
  cudaStream_t s = c->stream;
  size_t bn = 0;
  PieceRerun over;
  pt_emit_append<MODE>(c, st, Q, S, L, rec, &bn, tag_bits, &over);
  if (!over.src.empty()) {
    PieceList again(c);
    const size_t n = again.n = over.src.size();
    again.tot = over.off.back();
    again.src.resize(n);
    again.begin.resize(n);
    again.len.resize(n);
    again.off.resize(n + 1);
    SHCI_CUDA(cudaMemcpyAsync(again.src.p, over.src.data(), n * 4, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(again.begin.p, over.begin.data(), n * 4, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(again.len.p, over.len.data(), n * 4, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(again.off.p, over.off.data(), (n + 1) * 8, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
    PieceRerun over2;
    pt_emit_append<MODE>(c, st, Q, S, again, rec, &bn, tag_bits, &over2);
    if (!over2.src.empty()) throw std::logic_error("PT2 emission: exact regions overflowed");
  }
  {
    ProfScope ps(c->prof, s, "pt2_reduce");
    bn = group_records<NV>(c, rec, bn, st.P.n_orbs, tag_bits);
  }
  return bn;
}

// Window entries of each source (device).
template <int MODE>
void pt_counts(shci_ctx* c, PtSetup& st, const PtParams& Q, const StoSources& S, uint32_t n_src,
               DevBuf<uint64_t>& cnt) {
  cudaStream_t s = c->stream;
  cnt.mt = &c->mem;
  cnt.resize(n_src ? n_src : 1);
  if (!n_src) return;
  ProfScope ps(c->prof, s, "pt2_count");
  k_pt_count<MODE><<<grid_for((size_t)n_src * 32, kPtWarps * 32, st.grid), kPtWarps * 32, 0, s>>>(
      st.P, Q, S, n_src, cnt.p);
  SHCI_LAUNCH_CHECK();
  c->launches += 1;
}

// Sum and sum of squares of the contributions of one reduced batch (dtm / psto).
template <int MODE>
void pt_batch_sums(shci_ctx* c, const DevBuf<PtRec<n_cols<MODE>()>>& rec, size_t bn, double e_var,
                   double* sum, double* sumsq) {
  *sum = *sumsq = 0.0;
  if (!bn) return;
  cudaStream_t s = c->stream;
  DevBuf<double> x, out;
  DevBuf<uint64_t> starts;
  x.mt = out.mt = starts.mt = &c->mem;
  x.resize(bn);
  out.resize(2);
  starts.resize(2);
  {
    ProfScope ps(c->prof, s, "pt2_contrib");
    k_pt_x<MODE><<<grid_for(bn, 256), 256, 0, s>>>(diag_fix(c), rec.p, bn, e_var, 1.0, ~0ull,
                                                   x.p);
    SHCI_LAUNCH_CHECK();
    const uint64_t st2[2] = {0, bn};
    SHCI_CUDA(cudaMemcpyAsync(starts.p, st2, 16, cudaMemcpyHostToDevice, s));
    seg_reduce2(c, x.p, starts.p, 1, bn, out.p);
  }
  double h[2];
  SHCI_CUDA(cudaMemcpyAsync(h, out.p, 16, cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  *sum = h[0];
  *sumsq = h[1];
  c->launches += 2;
}

// Runs one batch of n_batches in *parts parts: the batches b + n_batches j, j < *parts, of n_batches *
// *parts, which together hold the dets of batch b (the remainder by the larger number fixes that by
// the smaller).  Where their records find no room there are twice as many from then on.
constexpr uint64_t kMaxParts = 1024;
template <class F>
void pt_in_parts(shci_ctx* c, uint64_t n_batches, uint64_t* parts, F&& run) {
  for (;;) {
    try {
      run();
      return;
    } catch (const OomError&) {
      if (*parts >= kMaxParts || n_batches * *parts >= 1ull << 31) throw;
    }
    *parts *= 2;
    // scratch that the attempt has grown
    c->u0.release();
    c->sort.kalt32.release();
    c->sort.valt32.release();
  }
}

// Deterministic-style batched stage (dtm: MODE kDtm, psto: kPsto) with the batch accumulation,
// uncertainty and (psto) early stopping of solver.h:691-764, 818-895.
template <int MODE>
Pt2Out pt_batched(shci_ctx* c, double e_var, PtParams Q, size_t n_batches, double target_error,
                  double eps_pt) {
  PtSetup st;
  pt_setup(c, st);
  const uint32_t n_var = static_cast<uint32_t>(c->up.size());
  StoSources S{};
  // window entries per source (size the automatic batch count and the regions)
  Q.batch = 0;
  DevBuf<uint64_t> entries;
  pt_counts<MODE>(c, st, Q, S, n_var, entries);
  if (n_batches == 0) {
    // Automatic batch count: 48 device bytes a window entry within 40 % of the free HBM.  A record
    // costs about 100 while it is grouped (32 and half as much for growth, 32 gathered, 19 for keys,
    // indexes and their sorted copies), but one window entry in two or fewer makes one (four of five
    // targets are occupied at n = 40), and a batch that still finds no room is taken in parts.  (The
    // dtm energy does not depend on the batch count.)
    uint64_t tot = 0;
    {
      DevBuf<uint64_t> sum;
      sum.mt = &c->mem;
      sum.resize(n_var);
      tot = exclusive_scan_u64(entries.p, sum.p, n_var, c->stream, c->sort);
    }
    size_t free_b = 0, total_b = 0;
    SHCI_CUDA(cudaMemGetInfo(&free_b, &total_b));
    free_b += c->mem.cached;  // cached blocks return to the driver on demand
    const double per = 48.0 * (MODE == kDtm ? 1.0 : 1.3);
    n_batches = static_cast<size_t>(std::ceil(tot * per / (0.4 * free_b)));
    if (n_batches < 1) n_batches = 1;
  }
  set_batches(Q, n_batches);
  PieceList pieces(c);
  make_pt_pieces(c, entries, n_var, n_batches, nullptr, pieces);
  entries.release();
  Pt2Out out;
  double esum = 0.0, esq = 0.0;
  size_t n_sum = 0;
  DevBuf<PtRec<n_cols<MODE>()>> rec;
  rec.mt = &c->mem;
  uint64_t parts = 1, listed = 1;  // listed: those that the pieces' regions are made for
  for (size_t batch = 0; batch < n_batches; batch++) {
    size_t bn = 0;
    double bs = 0.0, bsq = 0.0;
    pt_in_parts(c, n_batches, &parts, [&]() {
      if (listed != parts) {
        rec.release();
        set_batches(Q, n_batches * parts);
        DevBuf<uint64_t> again;
        pt_counts<MODE>(c, st, Q, S, n_var, again);
        make_pt_pieces(c, again, n_var, n_batches * parts, nullptr, pieces);
        listed = parts;
      }
      bn = 0;
      bs = bsq = 0.0;
      for (uint64_t j = 0; j < parts; j++) {
        Q.batch = batch + n_batches * j;
        const size_t m = pt_emit_reduce<MODE>(c, st, Q, S, pieces, rec, 0);
        double sum, sumsq;
        pt_batch_sums<MODE>(c, rec, m, e_var, &sum, &sumsq);
        bn += m;
        bs += sum;
        bsq += sumsq;
      }
    });
    n_sum += bn;
    esum += bs;
    esq += bsq;
    out.value = esum / (batch + 1) * n_batches;
    if (batch == n_batches - 1) {
      out.uncert = 0.0;
    } else {
      const double avg = esum / n_sum;
      const double sd = std::sqrt(esq / n_sum - avg * avg);
      if (MODE == kDtm) {
        out.uncert = sd * std::sqrt((double)n_sum) / (batch + 1) * (n_batches - batch - 1);
      } else {
        const double mean_sd = sd / std::sqrt((double)n_sum);
        out.uncert = mean_sd * n_sum / (batch + 1) * (n_batches - batch - 1);
      }
    }
    out.n_batches_done = batch + 1;
    if (MODE == kPsto) {
      if (out.uncert <= target_error * 0.5) break;
      if (Q.eps <= eps_pt && out.uncert <= target_error) break;
    }
  }
  out.n_pt_dets = n_sum;
  c->prof.flush();
  return out;
}

// f(begin, end) over [0, n) in contiguous chunks, one per host thread (chunk k on thread k).
template <class F>
void host_chunks(size_t n, F f) {
  const size_t k = std::max<size_t>(1, std::min<size_t>(host_threads(), (n + 65535) / 65536));
  std::vector<std::thread> th;
  for (size_t t = 1; t < k; t++) th.emplace_back(f, t, n * t / k, n * (t + 1) / k);
  f(size_t{0}, size_t{0}, n / k);
  for (auto& x : th) x.join();
}

// Vose alias tables, as src/util.cc:128-175.  The scaled probabilities and the initial
// small / large stacks are formed in chunks on the host threads (each chunk's indices in
// order, the chunks concatenated in order: the stacks the sequential pass would build); the
// pairing loop is sequential.
void alias_tables(const std::vector<double>& p, std::vector<double>& np, std::vector<size_t>& al) {
  const size_t L = p.size();
  np.assign(L, 0.0);
  al.assign(L, 0);
  std::vector<double> t(L);
  std::vector<size_t> small, large;  // used as stacks (back = top)
  std::vector<std::vector<size_t>> cs(host_threads()), cl(host_threads());
  host_chunks(L, [&](size_t k, size_t b, size_t e) {
    for (size_t i = b; i < e; i++) {
      t[i] = p[i] * L;
      if (t[i] < 1.) cs[k].push_back(i);
      else cl[k].push_back(i);
    }
  });
  small.reserve(L);
  large.reserve(L);
  for (auto& v : cs) small.insert(small.end(), v.begin(), v.end());
  for (auto& v : cl) large.insert(large.end(), v.begin(), v.end());
  while (!small.empty() && !large.empty()) {
    const size_t l = large.back(), s = small.back();
    np[s] = t[s];
    al[s] = l;
    t[l] = t[l] + t[s] - 1.;
    if (t[l] < 1.) {
      large.pop_back();
      small.back() = l;
    } else {
      small.pop_back();
    }
  }
  for (size_t i : large) np[i] = 1.;
  for (size_t i : small) np[i] = 1.;
}

}  // namespace

Pt2Out pt2_dtm(shci_ctx* c, double energy_var, double eps_pt_dtm, size_t n_batches) {
  PtParams Q{};
  Q.eps = eps_pt_dtm;
  return pt_batched<kDtm>(c, energy_var, Q, n_batches, 0.0, 0.0);
}

Pt2Out pt2_psto(shci_ctx* c, double energy_var, double eps_pt_dtm, double eps_pt_psto,
                size_t n_batches, double target_error, double eps_pt) {
  if (n_batches == 0) throw ArgError("n_batches must be >= 1");
  PtParams Q{};
  Q.eps = eps_pt_psto;
  Q.eps_dtm = eps_pt_dtm;
  return pt_batched<kPsto>(c, energy_var, Q, n_batches, target_error, eps_pt);
}

// Number of unique PT dets in hash batch 0 of 128 of the given sources (the sample-size
// pilot of solver.h:942-972; no |H_ai c_i| test on double excitations).
size_t pilot_pt_dets(shci_ctx* c, PtSetup& st, const std::vector<size_t>& src, double eps_pt,
                     int shift) {
  if (src.empty()) return 0;
  cudaStream_t s = c->stream;
  const uint32_t n_src = static_cast<uint32_t>(src.size());
  std::vector<uint32_t> h_det(src.begin(), src.end()), h_zero(n_src, 0u);
  std::vector<double> h_one(n_src, 1.0);
  std::vector<uint8_t> h_dtm(n_src, 1);
  DevBuf<uint32_t> d_det, d_zero, d_batch;
  DevBuf<double> d_one;
  DevBuf<uint8_t> d_dtm;
  d_det.mt = d_zero.mt = d_batch.mt = d_one.mt = d_dtm.mt = &c->mem;
  d_batch.resize(n_src);
  d_det.resize(n_src);
  d_zero.resize(n_src);
  d_one.resize(n_src);
  d_dtm.resize(n_src);
  SHCI_CUDA(cudaMemcpyAsync(d_det.p, h_det.data(), n_src * 4, cudaMemcpyHostToDevice, s));
  SHCI_CUDA(cudaMemcpyAsync(d_zero.p, h_zero.data(), n_src * 4, cudaMemcpyHostToDevice, s));
  SHCI_CUDA(cudaMemcpyAsync(d_one.p, h_one.data(), n_src * 8, cudaMemcpyHostToDevice, s));
  SHCI_CUDA(cudaMemcpyAsync(d_dtm.p, h_dtm.data(), n_src, cudaMemcpyHostToDevice, s));
  StoSources S{d_det.p, d_zero.p, d_one.p, d_one.p, d_batch.p, d_dtm.p};
  PtParams Q{};
  Q.eps = eps_pt;
  Q.eps_psto = eps_pt;
  Q.factor = 0.0;
  Q.iter_shift = shift;
  Q.pilot = 1;
  size_t n = 0;
  uint64_t parts = 1;
  pt_in_parts(c, 128, &parts, [&]() {
    set_batches(Q, 128 * parts);
    DevBuf<uint64_t> entries;
    pt_counts<kSto>(c, st, Q, S, n_src, entries);
    PieceList pieces(c);
    make_pt_pieces(c, entries, n_src, 128 * parts, nullptr, pieces);
    DevBuf<PtRec<5>> rec;
    rec.mt = &c->mem;
    n = 0;
    for (uint64_t j = 0; j < parts; j++) {
      const std::vector<uint32_t> b(n_src, static_cast<uint32_t>(128 * j));
      SHCI_CUDA(cudaMemcpyAsync(d_batch.p, b.data(), n_src * 4, cudaMemcpyHostToDevice, s));
      n += pt_emit_reduce<kSto>(c, st, Q, S, pieces, rec, 5);
    }
  });
  return n;
}

size_t psto_auto_batches(shci_ctx* c, double eps_pt_psto, double pt_mem_avail, double mem_usage,
                         size_t* n_pilot) {
  const int shift = c->I.n;
  if (shift > 57) throw ArgError("the automatic psto batch count supports n_orbs <= 57");
  PtSetup st;
  pt_setup(c, st);
  std::vector<size_t> src;
  for (size_t i = 50; i < c->up.size(); i += 100) src.push_back(i);
  const size_t n_pt = pilot_pt_dets(c, st, src, eps_pt_psto, shift);
  if (n_pilot) *n_pilot = n_pt;
  const size_t bytes_per_entry = 2 * 16 + 16;  // solver.h:402, 774
  const double mem = static_cast<double>(static_cast<size_t>(pt_mem_avail)) * mem_usage;
  size_t nb = static_cast<size_t>(std::ceil(2.5 * 128 * 100 * static_cast<double>(n_pt) *
                                            static_cast<double>(bytes_per_entry) / mem));
  if (nb < 16) nb = 16;
  return nb;
}

// Stochastic stage (solver.h:898-1153).  n_dets_in_sample = 0: the sample size comes from
// the reference's 1,000-draw pilot and the PT memory pt_mem_avail (solver.h:942-1006);
// semisto: the variational dets above the quantile of the top quarter of the unique-sample
// target are summed deterministically in every iteration and the others sampled with
// renormalised weights (solver.h:1009-1036).  psto_uncert is the uncertainty of the preceding
// stage (it enters the second stopping rule).  info = {n_dets_in_sample, n_dtm,
// n_unique_target} of the run.
Pt2Out pt2_sto(shci_ctx* c, double energy_var, double eps_pt_psto, double eps_pt,
               size_t n_batches, size_t n_dets_in_sample, bool semisto, unsigned random_seed,
               size_t max_iterations, double target_error, double psto_uncert,
               double pt_mem_avail, double mem_usage, std::vector<double>* loops,
               size_t* info) {
  if (n_batches == 0) throw ArgError("n_batches must be >= 1");
  if (n_dets_in_sample == 1) throw ArgError("n_dets_in_sample_pt_sto must be 0 (automatic) or >= 2");
  if (semisto && n_dets_in_sample != 0)
    throw ArgError("semisto_sto with n_dets_in_sample_pt_sto set has no deterministic dets in "
                   "the reference (its 25% quantile heap is empty: solver.h:1009-1021); set "
                   "semisto_sto to false or leave n_dets_in_sample_pt_sto unset");
  const size_t n_var = c->up.size();
  std::vector<double> coefs(n_var);
  sync_dets(c);
  cudaStream_t s = c->stream;
  SHCI_CUDA(cudaMemcpyAsync(coefs.data(), c->d_coef.p, n_var * 8, cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  const int shift = c->I.n;
  if (shift > 57) throw ArgError("stochastic PT2 supports n_orbs <= 57");
  const auto t_setup = std::chrono::steady_clock::now();
  // probabilities and their running sums (solver.h:921-933)
  double sum_w = 0.0;
  for (size_t i = 0; i < n_var; i++) sum_w += std::abs(coefs[i]);
  std::vector<double> probs(n_var), cum;
  host_chunks(n_var, [&](size_t, size_t b, size_t e) {
    for (size_t i = b; i < e; i++) probs[i] = std::abs(coefs[i]) / sum_w;
  });
  if (n_dets_in_sample == 0) {  // the pilot draws by inverse CDF
    cum.resize(n_var);
    for (size_t i = 0; i < n_var; i++) cum[i] = i > 0 ? probs[i] + cum[i - 1] : probs[i];
  }
  std::default_random_engine gen(random_seed);
  std::uniform_real_distribution<double> ur(0., 1.);
  PtSetup st;
  pt_setup(c, st);
  size_t n_target = 0;
  if (n_dets_in_sample == 0) {
    // pilot (solver.h:944-972): 1,000 inverse-CDF draws, PT dets of the unique ones in batch
    // 0 of 128, scaled to a batch of n_batches
    std::vector<uint8_t> seen(n_var, 0);
    std::vector<size_t> list;
    for (size_t k = 0; k < 1000; k++) {
      const size_t id = std::lower_bound(cum.begin(), cum.end(), ur(gen)) - cum.begin();
      if (id < n_var && !seen[id]) {
        seen[id] = 1;
        list.push_back(id);
      } else if (id >= n_var) {
        throw ArgError("coefficient weights do not sum to 1 (empty or non-finite wavefunction)");
      }
    }
    const size_t n_pt = pilot_pt_dets(c, st, list, eps_pt, shift);
    const size_t n_pt_batch = n_pt * 128 / n_batches;
    const size_t bytes_per_entry = 2 * 16 + 40;  // solver.h:402, 905 (two 64-bit chunks)
    const size_t cap = n_var / 8 + 1;
    // a pilot without PT dets is a division by zero in the reference; the cap is taken
    n_target = cap;
    if (n_pt_batch > 0) {
      const double t = static_cast<double>(static_cast<size_t>(pt_mem_avail)) * mem_usage *
                       static_cast<double>(list.size()) / static_cast<double>(bytes_per_entry) /
                       5.0 / static_cast<double>(n_pt_batch);
      n_target = static_cast<size_t>(t);
      if (n_target >= cap) n_target = cap;
    }
    // draws until the target of unique dets is met (solver.h:990-1000)
    std::fill(seen.begin(), seen.end(), 0);
    size_t n_unique = 0;
    while (n_unique < n_target) {
      const size_t id = std::lower_bound(cum.begin(), cum.end(), ur(gen)) - cum.begin();
      if (id >= n_var)
        throw ArgError("coefficient weights do not sum to 1 (empty or non-finite wavefunction)");
      if (!seen[id]) {
        seen[id] = 1;
        n_unique++;
      }
      n_dets_in_sample++;
    }
  }
  std::vector<uint32_t> dtm_list;
  if (semisto) {
    // the top n_target / 4 weights by a min-heap quantile (solver.h:1009-1036)
    const size_t n_heap = n_target / 4;
    if (n_heap == 0)
      throw ArgError("semistochastic PT2 needs a sample-size target of at least 4 (the "
                     "reference's quantile heap would be empty)");
    std::priority_queue<double, std::vector<double>, std::greater<double>> heap;
    for (size_t i = 0; i < n_heap; i++) heap.push(probs[i]);
    for (size_t i = n_heap; i < n_var; i++)
      if (heap.top() < probs[i]) {
        heap.pop();
        heap.push(probs[i]);
      }
    const double C = heap.top();
    double s2 = 0.0;
    for (size_t i = 0; i < n_var; i++) {
      if (probs[i] > C) {
        probs[i] = 0.;
        dtm_list.push_back(static_cast<uint32_t>(i));
      } else {
        s2 += probs[i];
      }
    }
    for (auto& p : probs) p /= s2;
  }
  const size_t n_dtm = dtm_list.size();
  if (n_dets_in_sample < n_dtm + 2)
    throw ArgError("stochastic PT2 sample too small for its deterministic part");
  if (info) {
    info[0] = n_dets_in_sample;
    info[1] = n_dtm;
    info[2] = n_target;
  }
  std::uniform_int_distribution<size_t> ui_var(0, n_var - 1);
  std::uniform_int_distribution<size_t> ui_batch(0, n_batches - 1);
  const double factor = 1. / (n_dets_in_sample - n_dtm - 1.);
  // Iterations per device pass: the first pass runs the 6 iterations before which the
  // stopping rules cannot fire, later passes 2 (results past the stop are discarded).
  const uint32_t kFirstChunk = 6, kNextChunk = 2;
  // A pass's random numbers in the reference's order (per iteration: its draws, then its
  // batch, solver.h:1048-1072).  They depend on nothing but the generator, so a helper thread
  // draws each pass ahead of it: the first while the alias tables are built, the next during
  // the current pass's device work (a pass that turns out not to be needed only advanced the
  // generator, which nothing uses afterwards).
  const size_t n_draw = n_dets_in_sample - n_dtm;
  struct PassDraws {
    std::vector<std::vector<size_t>> r1;
    std::vector<std::vector<double>> r2;
    std::vector<size_t> batch;
  };
  auto draw_pass = [&gen, &ur, &ui_var, &ui_batch, n_draw](uint32_t n_it) {
    PassDraws d;
    d.r1.assign(n_it, std::vector<size_t>(n_draw));
    d.r2.assign(n_it, std::vector<double>(n_draw));
    d.batch.resize(n_it);
    for (uint32_t it = 0; it < n_it; it++) {
      for (size_t k = 0; k < n_draw; k++) {
        d.r1[it][k] = ui_var(gen);
        d.r2[it][k] = ur(gen);
      }
      d.batch[it] = ui_batch(gen);
    }
    return d;
  };
  // one helper thread draws ahead unless the calling thread may use only one host thread
  const unsigned n_host = host_threads();
  const auto draw_policy = n_host > 1 ? std::launch::async : std::launch::deferred;
  std::future<PassDraws> next_draws;
  if (max_iterations > 0)
    next_draws = std::async(draw_policy, draw_pass,
                            static_cast<uint32_t>(std::min<size_t>(kFirstChunk, max_iterations)));
  // per-iteration sample counts, one array per iteration of a pass (zero between uses; set up
  // on a helper thread while the alias tables are built); which iterations of a pass drew
  // each det (zero between uses); the deterministic dets
  std::vector<std::vector<uint32_t>> cnts;
  std::vector<uint8_t> pass_mask, is_dtm;
  auto zeroed = std::async(n_host > 1 ? std::launch::async : std::launch::deferred, [&]() {
    const size_t k = std::min<size_t>(std::max<size_t>(kFirstChunk, kNextChunk), max_iterations);
    for (size_t it = 0; it < k; it++) cnts.emplace_back(n_var, 0u);
    pass_mask.assign(n_var, 0);
    is_dtm.assign(n_var, 0);
  });
  std::vector<double> aprob;
  std::vector<size_t> alias;
  alias_tables(probs, aprob, alias);
  zeroed.get();
  for (uint32_t i : dtm_list) is_dtm[i] = 1;
  static_assert(kFirstChunk <= 8 && kNextChunk <= 8, "iteration masks are 8 bits");
  if (c->prof.on)
    c->prof.host("pt2_host_setup", std::chrono::duration<double, std::milli>(
                                       std::chrono::steady_clock::now() - t_setup).count());
  Pt2Out out;
  std::vector<double> loop_vals;
  bool done = false;
  size_t iteration = 0;
  uint64_t parts = 1;
  while (!done && iteration < max_iterations) {
    // draw the samples of the next chunk of iterations (solver.h:1048-1072)
    const uint32_t chunk = iteration == 0 ? kFirstChunk : kNextChunk;
    const uint32_t n_it = static_cast<uint32_t>(std::min<size_t>(chunk, max_iterations - iteration));
    std::vector<uint32_t> h_det, h_iter, h_batch, h_off;
    std::vector<double> h_count, h_weight;
    std::vector<uint8_t> h_dtm;
    {
      HostScope hs(c->prof, "pt2_host_sample");
      // the pass's random numbers (drawn ahead), then the next pass's, ahead of it
      HostScope hs_rng(c->prof, "pt2_host_sample_rng");
      PassDraws draws = next_draws.get();
      hs_rng.stop();
      const size_t it_next = iteration + n_it;
      if (it_next < max_iterations)
        next_draws = std::async(
            draw_policy, draw_pass,
            static_cast<uint32_t>(std::min<size_t>(kNextChunk, max_iterations - it_next)));
      const auto& r1s = draws.r1;
      const auto& r2s = draws.r2;
      const auto& batch_ids = draws.batch;
      // Per iteration and on a host thread of its own: the alias lookups (independent of one
      // another: one loop whose cache misses overlap, the table entries of a later draw
      // prefetched; the tables are far larger than the host caches), the sample counts per det
      // and the dets in order of first draw (the reference's unordered_map counts and
      // insertion-ordered list).
      while (cnts.size() < n_it) cnts.emplace_back(n_var, 0u);
      std::vector<std::vector<uint32_t>> lists(n_it);
      auto sample_one = [&](uint32_t it) {
        constexpr size_t kAhead = 32;
        const auto& r1 = r1s[it];
        const auto& r2 = r2s[it];
        auto& cnt = cnts[it];
        std::vector<uint32_t> ids(n_draw);
        for (size_t k = 0; k < n_draw; k++) {
          if (k + kAhead < n_draw) {
            __builtin_prefetch(&aprob[r1[k + kAhead]]);
            __builtin_prefetch(&alias[r1[k + kAhead]]);
          }
          ids[k] = static_cast<uint32_t>(r2[k] < aprob[r1[k]] ? r1[k] : alias[r1[k]]);
        }
        auto& list = lists[it];
        for (size_t k = 0; k < n_draw; k++) {
          if (k + kAhead < n_draw) __builtin_prefetch(&cnt[ids[k + kAhead]], 1);
          const uint32_t id = ids[k];
          if (cnt[id]++ == 0) list.push_back(id);
        }
      };
      {
        HostScope hs_look(c->prof, "pt2_host_sample_lookup");
        std::atomic<uint32_t> next_it{0};
        auto run = [&]() {
          for (uint32_t it; (it = next_it.fetch_add(1)) < n_it;) sample_one(it);
        };
        std::vector<std::thread> th;
        for (uint32_t t = 1; t < std::min<uint32_t>(n_it, n_host); t++) th.emplace_back(run);
        run();
        for (auto& t : th) t.join();
      }
      HostScope hs_group(c->prof, "pt2_host_sample_group");
      // The pass's entries grouped by det, dets in increasing order and a det's iterations in
      // order: a det drawn in several iterations is walked once (the heaviest dets, with the
      // widest windows, are drawn in nearly every iteration).  A bit mask per det marks the
      // iterations that drew it (all of them for a deterministic det: count and weight 1); one
      // scan of the masks in det order lays the entries out.
      const uint8_t all_it = static_cast<uint8_t>((1u << n_it) - 1u);
      size_t n_ent_pass = n_dtm * n_it;
      for (uint32_t it = 0; it < n_it; it++) {
        n_ent_pass += lists[it].size();
        for (uint32_t i : lists[it]) pass_mask[i] |= static_cast<uint8_t>(1u << it);
      }
      for (uint32_t i : dtm_list) pass_mask[i] = all_it;
      h_det.resize(n_ent_pass);
      h_iter.resize(n_ent_pass);
      h_batch.resize(n_ent_pass);
      h_count.resize(n_ent_pass);
      h_weight.resize(n_ent_pass);
      h_dtm.resize(n_ent_pass);
      h_off.clear();
      size_t k = 0;
      for (size_t i = 0; i < n_var; i++) {
        const uint32_t m = pass_mask[i];
        if (!m) continue;
        pass_mask[i] = 0;
        h_off.push_back(static_cast<uint32_t>(k));
        const bool dt = is_dtm[i] != 0;
        for (uint32_t it = 0; it < n_it; it++) {
          if (!(m >> it & 1u)) continue;
          h_det[k] = static_cast<uint32_t>(i);
          h_iter[k] = it;
          h_batch[k] = static_cast<uint32_t>(batch_ids[it]);
          if (dt) {
            h_count[k] = 1.0;
            h_weight[k] = 1.0;
            h_dtm[k] = 1;
          } else {
            h_count[k] = static_cast<double>(cnts[it][i]);
            cnts[it][i] = 0;
            h_weight[k] = (n_dets_in_sample - n_dtm) * probs[i];
            h_dtm[k] = 0;
          }
          k++;
        }
      }
      h_off.push_back(static_cast<uint32_t>(k));
    }
    const uint32_t n_ent = static_cast<uint32_t>(h_det.size());
    const uint32_t n_src = static_cast<uint32_t>(h_off.size() - 1);  // dets of the pass
    DevBuf<uint32_t> d_det, d_iter, d_batch;
    DevBuf<double> d_count, d_weight;
    DevBuf<uint8_t> d_dtm;
    DevBuf<uint32_t> d_off;
    d_det.mt = d_iter.mt = d_batch.mt = d_count.mt = d_weight.mt = d_dtm.mt = &c->mem;
    d_off.mt = &c->mem;
    d_off.resize(n_src + 1);
    SHCI_CUDA(cudaMemcpyAsync(d_off.p, h_off.data(), (n_src + 1) * 4, cudaMemcpyHostToDevice, s));
    d_det.resize(n_ent);
    d_iter.resize(n_ent);
    d_batch.resize(n_ent);
    d_count.resize(n_ent);
    d_weight.resize(n_ent);
    d_dtm.resize(n_ent);
    SHCI_CUDA(cudaMemcpyAsync(d_det.p, h_det.data(), n_ent * 4, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_iter.p, h_iter.data(), n_ent * 4, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_batch.p, h_batch.data(), n_ent * 4, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_count.p, h_count.data(), n_ent * 8, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_weight.p, h_weight.data(), n_ent * 8, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_dtm.p, h_dtm.data(), n_ent, cudaMemcpyHostToDevice, s));
    StoSources S{d_det.p, d_iter.p, d_count.p, d_weight.p, d_batch.p, d_dtm.p, d_off.p};
    PtParams Q{};
    Q.eps = eps_pt;
    Q.eps_psto = eps_pt_psto;
    Q.factor = factor;
    Q.iter_shift = shift;
    size_t bn = 0;
    std::vector<double> it_sum;  // per-iteration sums of the contributions
    pt_in_parts(c, n_batches, &parts, [&]() {
      set_batches(Q, n_batches * parts);
      DevBuf<uint64_t> entries;
      pt_counts<kSto>(c, st, Q, S, n_src, entries);
      PieceList pieces(c);
      make_pt_pieces(c, entries, n_src, n_batches * parts, d_off.p, pieces);
      DevBuf<PtRec<5>> rec;
      rec.mt = &c->mem;
      bn = 0;
      it_sum.assign(n_it, 0.0);
      for (uint64_t j = 0; j < parts; j++) {
        std::vector<uint32_t> b;
        if (parts > 1) {
          for (uint32_t x : h_batch) b.push_back(static_cast<uint32_t>(x + n_batches * j));
          SHCI_CUDA(cudaMemcpyAsync(d_batch.p, b.data(), n_ent * 4, cudaMemcpyHostToDevice, s));
        }
        const size_t m = pt_emit_reduce<kSto>(c, st, Q, S, pieces, rec, 5);
        if (!m) continue;
        DevBuf<double> x, o;
        DevBuf<uint64_t> starts;
        x.mt = o.mt = starts.mt = &c->mem;
        x.resize(m);
        o.resize(2 * n_it);
        starts.resize(n_it + 1);
        const uint64_t mask = shift == 64 ? ~0ull : ((1ull << shift) - 1ull);
        {
          ProfScope ps(c->prof, s, "pt2_contrib");
          k_pt_x<kSto><<<grid_for(m, 256), 256, 0, s>>>(diag_fix(c), rec.p, m, energy_var,
                                                        static_cast<double>(n_batches), mask, x.p);
          SHCI_LAUNCH_CHECK();
          k_iter_starts<<<1, 128, 0, s>>>(rec.p, m, shift, n_it, starts.p);
          SHCI_LAUNCH_CHECK();
          seg_reduce2(c, x.p, starts.p, n_it, m, o.p);
        }
        std::vector<double> h(2 * n_it);
        SHCI_CUDA(cudaMemcpyAsync(h.data(), o.p, h.size() * 8, cudaMemcpyDeviceToHost, s));
        SHCI_CUDA(cudaStreamSynchronize(s));
        for (uint32_t it = 0; it < n_it; it++) it_sum[it] += h[2 * it];
        bn += m;
        c->launches += 3;
      }
    });
    out.n_pt_dets += bn;
    // statistics and stopping rules, iteration by iteration (solver.h:1126-1147)
    for (uint32_t it = 0; it < n_it && !done; it++) {
      loop_vals.push_back(it_sum[it]);
      const double n = static_cast<double>(loop_vals.size());
      double sm = 0.0, sq = 0.0;
      for (double v : loop_vals) {
        sm += v;
        sq += v * v;
      }
      out.value = sm / n;
      out.uncert = std::sqrt((sq - sm * sm / n) / (n - 1)) / std::sqrt(n);
      iteration++;
      if (iteration >= 6 && out.uncert <= target_error * 0.7) done = true;
      if (iteration >= 10 &&
          std::sqrt(out.uncert * out.uncert + psto_uncert * psto_uncert) <= target_error)
        done = true;
    }
  }
  out.n_batches_done = iteration;
  if (loops) *loops = loop_vals;
  c->prof.flush();
  return out;
}

}  // namespace shci
