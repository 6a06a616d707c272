// Heat-bath selection (K6): one step of Solver<S>::run_variation's "get next det list".
//
// Reference: src/solver/solver.h:435-495 driving ChemSystem::find_connected_dets
// (src/chem/chem_system.cc:289-402).  For each pass j = 0..4 over var dets i = j (mod 5):
//   eps_min = eps_var / |c_i| (0 for i = 0 with var_sd), skipped when eps_min >=
//   eps_tried_prev[i]; singles from singles_queue[p] with S >= eps_min whose |H_ai| >= eps_min,
//   doubles from hci_queue[pq] with eps_min <= H < eps_tried_prev[i]; dets already in the
//   variational set are dropped; eps_tried_prev[i] = 1.000000001 * eps_min.
// New dets of a pass are appended in ascending Det order and belong to the variational set from the
// next pass on, so a new det belongs to the first pass that finds it: all sources are emitted
// at once, each candidate with its source's pass, and of equal candidates the lowest pass counts.
//   k_sel_count : a warp per source det -> window entries (walk.cuh),
//   k_sel_emit  : a warp per piece of a window builds the candidates 32 at a time, tests membership
//                 in the hash set of the variational dets and (singles) the |H_ai| >= eps_min rule,
//                 and appends what is left, unordered,
//   one radix sort by (det, pass), first of each det, stable sort by pass -> the new dets in order.
// (The passes used to run one after the other: five times the launches and synchronisations, with
// the first sources' long windows as each launch's tail.  n = 26, seven selections to 80,351 dets:
// 4.0 -> 0.9 ms of emission; the whole variational stage 38.7 -> 27.8 ms, n = 16 14.5 -> 9.7 ms.)
// With second rejection (off by default) the emission also drops window entries whose
// |H|^2 / (one-body energy difference to HF) is below factor * eps_min^2 and records, per
// source, the largest |H| it dropped; eps_tried_prev then becomes 1.000000001 * max(that,
// eps_min) (solver.h:461-465, chem_system.cc:300-308, 318-324, 364-370, 401).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "ctx.h"
#include "kernels.h"
#include "walk.cuh"

namespace shci {

namespace {

// Window entries per source det i (none where eps_min >= eps_tried_prev, solver.h:448) and eps_min.
__global__ void __launch_bounds__(kSelWarps * 32)
    k_sel_count(SelParams P, uint32_t n, uint64_t* cnt_out, double* eps_min_out) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t wpg = gridDim.x * kSelWarps;
  for (uint32_t i = blockIdx.x * kSelWarps + (threadIdx.x >> 5); i < n; i += wpg) {
    const double eps_min = src_eps_min(P, i);
    const double eps_max = P.eps_tried[i];
    uint64_t tot = 0;
    if (eps_min < eps_max) {
      const uint64_t up = P.up[i], dn = P.dn[i];
      const int n_slots = P.n_elecs + P.n_pairs;
      for (int s0 = 0; s0 < n_slots; s0 += 32) {
        uint32_t lo = 0, c = 0;
        if (s0 + (int)lane < n_slots) slot_range(P, up, dn, s0 + lane, eps_min, eps_max, &lo, &c);
        uint64_t cc = c;
#pragma unroll
        for (int o = 16; o; o >>= 1) cc += __shfl_xor_sync(kFull, cc, o);
        tot += cc;
      }
    }
    if (lane == 0) {
      cnt_out[i] = tot;
      eps_min_out[i] = eps_min;
    }
  }
}

// eps_tried_prev of the processed sources (solver.h:468).  rej_max (second rejection only): the
// largest rejected |H| of each source, else null.  As find_connected_dets returns it: max(largest
// rejected, eps_min), except that a det whose eps_min is above every double's |H|, or a system
// without double excitations, returns eps_min before the doubles (chem_system.cc:339-340, 345),
// dropping what its singles rejected.
__global__ void k_sel_mark(SelParams P, uint32_t n, const double* eps_min_in,
                           const double* rej_max) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double eps_min = eps_min_in[i];
    if (eps_min < P.eps_tried[i]) {
      const bool rej = rej_max && !P.no_doubles && !(eps_min > P.max_hci);
      P.eps_tried[i] = 1.000000001 * (rej ? fmax(rej_max[i], eps_min) : eps_min);
    }
  }
}

// One-body energy difference of det (up, dn) from HF, accumulated in the reference's order
// (chem_system.cc:300-308): -e_hf_1b, then h_pp over the alpha electrons, then the beta ones.
__device__ __forceinline__ double diff_from_hf(const SelParams& P, uint64_t up, uint64_t dn) {
  const int n = P.n_orbs;
  double d = -P.e_hf_1b;
  for (uint64_t m = up; m; m &= m - 1) d += P.I.h1[ctz64(m) * (n + 1)];
  for (uint64_t m = dn; m; m &= m - 1) d += P.I.h1[ctz64(m) * (n + 1)];
  return d;
}

// Second-rejection test of entry e with slot code and targets x (chem_system.cc:318-324, 364-370):
// true when the entry is dropped; *h is its |H| (the queue's S or H).
__device__ __forceinline__ bool second_rejected(const SelParams& P, uint32_t x, uint32_t e,
                                                double diff, double eps_min, double* h) {
  const int n1 = P.n_orbs + 1;
  const double* d1 = P.I.h1;
  const int p = x >> kPBit & 63u, q = x >> kQBit & 63u;
  int r = x >> kRBit & 63u, s = x >> kSBit & 63u;
  double den;
  if (x & kOne) {
    *h = P.s_S[e];
    den = diff - d1[p * n1] + d1[r * n1];
  } else {
    if ((x & kADn) && !(x & kBDn)) {  // the reference swaps r and s here (:357-361)
      const int t = r;
      r = s;
      s = t;
    }
    *h = P.d_H[e];
    den = diff - d1[p * n1] - d1[q * n1] + d1[r * n1] + d1[s * n1];
  }
  const double hv = *h;
  return den > 0. && __ddiv_rn(__dmul_rn(hv, hv), den) <
                         __dmul_rn(__dmul_rn(P.rej_factor, eps_min), eps_min);
}

struct SelWarp {
  WalkWarp w;
  uint2 a[64];  // entries to be built: slot code with targets, source det
};

struct SelPieces {
  const uint32_t* src;
  const uint32_t* begin;
  const uint32_t* len;
  uint32_t n;
};

// Candidates of the pieces, unordered: cand[k] = (up, dn), pass[k] = the pass (source det mod 5);
// *count may pass cap (nothing is written past it).
__global__ void __launch_bounds__(kSelWarps * 32, 4)
    k_sel_emit(SelParams P, SelPieces pc, const double* __restrict__ eps_min_in,
               ulonglong2* __restrict__ cand, uint8_t* __restrict__ pass,
               unsigned long long* __restrict__ count, uint64_t cap, double* rej_max) {
  __shared__ SelWarp ws[kSelWarps];
  SelWarp& W = ws[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t ah = 0, an = 0;
  auto drain = [&](uint32_t m) {  // the m oldest entries
    __syncwarp();
    const uint2 en = W.a[(ah + lane) & 63u];
    __syncwarp();
    ah += m;
    an -= m;
    bool ok = false;
    uint64_t ru = 0, rd = 0;
    if (lane < m) {
      const uint64_t up = P.up[en.y], dn = P.dn[en.y];
      uint64_t cu = up, cd = dn;
      apply_entry(en.x, &cu, &cd);
      // time_sym: the stored form has up <= dn (solver.h:452-454)
      const bool flip = P.time_sym && cu > cd;
      ru = flip ? cd : cu;
      rd = flip ? cu : cd;
      ok = !in_set(P, ru, rd);
      // small single excitations are filtered (solver.h:456-459)
      if (ok && (en.x & kOne)) ok = !(fabs(h_one(P.I, up, dn, cu, cd)) < eps_min_in[en.y]);
    }
    const unsigned bal = __ballot_sync(kFull, ok);
    if (!bal) return;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(count, static_cast<unsigned long long>(__popc(bal)));
    at = __shfl_sync(kFull, at, 0) + __popc(bal & lt);
    if (ok && at < cap) {
      cand[at] = make_ulonglong2(ru, rd);
      pass[at] = static_cast<uint8_t>(en.y % 5u);
    }
  };
  const uint32_t wpg = gridDim.x * kSelWarps;
  for (uint32_t p = blockIdx.x * kSelWarps + (threadIdx.x >> 5); p < pc.n; p += wpg) {
    const uint32_t i = pc.src[p];
    const double eps_min = eps_min_in[i];
    const uint64_t up = P.up[i], dn = P.dn[i];
    const double diff = P.rej_on ? diff_from_hf(P, up, dn) : 0.0;
    double rmax = 0.0;  // largest rejected |H| seen by this lane
    walk_window(P, W.w, up, dn, eps_min, P.eps_tried[i], pc.begin[p], pc.len[p],
                [&](bool valid, bool free, uint32_t x, uint32_t e) {
                  double h;
                  if (P.rej_on && valid && second_rejected(P, x, e, diff, eps_min, &h)) {
                    rmax = fmax(rmax, h);
                    free = false;
                  }
                  const unsigned bal = __ballot_sync(kFull, free);
                  if (!bal) return;
                  if (free) W.a[(ah + an + __popc(bal & lt)) & 63u] = make_uint2(x, i);
                  an += __popc(bal);
                  if (an >= 32u) drain(32u);
                });
    if (P.rej_on) {
#pragma unroll
      for (int o = 16; o; o >>= 1) rmax = fmax(rmax, __shfl_xor_sync(kFull, rmax, o));
      // (non-negative doubles order like their bits)
      if (lane == 0 && rmax > 0.0)
        atomicMax(reinterpret_cast<unsigned long long*>(rej_max + i),
                  static_cast<unsigned long long>(__double_as_longlong(rmax)));
    }
  }
  while (an) drain(an < 32u ? an : 32u);
}

// Rank of string s among the strings with its number of electrons, in numeric order: the sum of
// C(position of the k-th electron, k).
__device__ __forceinline__ uint64_t string_rank(const uint64_t* __restrict__ binom, uint64_t s) {
  uint64_t r = 0;
  int k = 1;
  for (uint64_t m = s; m; m &= m - 1, k++) r += binom[k * 64 + ctz64(m)];
  return r;
}

// key = (rank(up) * n_dn_strings + rank(dn)) * 8 + pass: (det, pass) order in one integer.
__global__ void k_cand_keys(const ulonglong2* __restrict__ cand, const uint8_t* __restrict__ pass,
                            size_t m, const uint64_t* __restrict__ binom, uint64_t n_dn_strings,
                            uint64_t* __restrict__ key, uint32_t* __restrict__ idx) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    const ulonglong2 c = cand[k];
    key[k] = (string_rank(binom, c.x) * n_dn_strings + string_rank(binom, c.y)) * 8u + pass[k];
    idx[k] = static_cast<uint32_t>(k);
  }
}

// One component of the candidates in the order idx: 0 pass, 1 dn, 2 up.
__global__ void k_cand_component(const ulonglong2* __restrict__ cand,
                                 const uint8_t* __restrict__ pass, const uint32_t* __restrict__ idx,
                                 size_t m, int which, uint64_t* __restrict__ key) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    const uint32_t i = idx[k];
    key[k] = which == 0 ? pass[i] : which == 1 ? cand[i].y : cand[i].x;
  }
}

// flag[k] = 1 for the first candidate of each det in the order idx.
__global__ void k_cand_first(const ulonglong2* __restrict__ cand, const uint32_t* __restrict__ idx,
                             const uint64_t* __restrict__ key, bool ranked, size_t m,
                             uint32_t* __restrict__ flag) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    bool first = k == 0;
    if (!first && ranked) {
      first = key[k] >> 3 != key[k - 1] >> 3;
    } else if (!first) {
      const ulonglong2 a = cand[idx[k]], b = cand[idx[k - 1]];
      first = a.x != b.x || a.y != b.y;
    }
    flag[k] = first ? 1u : 0u;
  }
}

__global__ void k_cand_take(const ulonglong2* __restrict__ cand, const uint8_t* __restrict__ pass,
                            const uint32_t* __restrict__ idx, const uint32_t* __restrict__ flag,
                            const uint32_t* __restrict__ pos, size_t m,
                            ulonglong2* __restrict__ out, uint8_t* __restrict__ out_pass) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x)
    if (flag[k]) {
      const uint32_t i = idx[k];
      out[pos[k]] = cand[i];
      out_pass[pos[k]] = pass[i];
    }
}

__global__ void k_pass_keys(const uint8_t* __restrict__ pass, size_t m, uint32_t* __restrict__ key,
                            uint32_t* __restrict__ idx) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    key[k] = pass[k];
    idx[k] = static_cast<uint32_t>(k);
  }
}

__global__ void k_append(const ulonglong2* __restrict__ cand, const uint32_t* __restrict__ idx,
                         size_t m, uint64_t* __restrict__ up, uint64_t* __restrict__ dn,
                         double* __restrict__ coef) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    const ulonglong2 c = cand[idx[k]];
    up[k] = c.x;
    dn[k] = c.y;
    coef[k] = 1e-16;
  }
}

__global__ void k_valid_flags(const uint64_t* up, size_t n, uint32_t* flags) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    flags[i] = up[i] != kInvalid ? 1u : 0u;
}

__global__ void k_compact2(const uint64_t* a, const uint64_t* b, const uint32_t* flags,
                           const uint32_t* pos, size_t n, uint64_t* oa, uint64_t* ob) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    if (flags[i]) {
      oa[pos[i]] = a[i];
      ob[pos[i]] = b[i];
    }
}

// flags[k] = 1 where (su, sd)[k] differs from its predecessor
__global__ void k_unique_flags(const uint64_t* su, const uint64_t* sd, size_t n, uint32_t* flags) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x)
    flags[k] = (k == 0 || su[k] != su[k - 1] || sd[k] != sd[k - 1]) ? 1u : 0u;
}

__global__ void k_fill_coef(double* c, size_t from, size_t to, double v) {
  for (size_t i = from + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < to;
       i += (size_t)gridDim.x * blockDim.x)
    c[i] = v;
}

// Several states: the coefficient of largest magnitude over the states, the first one on
// ties (solver.h:440-444).
struct StatePtrs {
  const double* p[kMaxStates - 1];
};
__global__ void k_max_coef(const double* c0, StatePtrs xs, int n_extra, size_t n, double* out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    double m = c0[i];
    for (int k = 0; k < n_extra; k++) {
      const double v = xs.p[k][i];
      if (fabs(v) > fabs(m)) m = v;
    }
    out[i] = m;
  }
}

}  // namespace

// Sorts (up, dn) pairs held in a / b (length m) into ascending (a, b) order and removes
// duplicates; returns the unique count (left in a / b).  a_bits = bits of the a key (0: n_orbs);
// b keys always have n_orbs bits.
size_t sort_unique_pairs(shci_ctx* c, DevBuf<uint64_t>& a, DevBuf<uint64_t>& b, size_t m,
                         int a_bits) {
  if (m == 0) return 0;
  cudaStream_t s = c->stream;
  const int nb = c->I.n;
  c->u0.reserve(m, 1.25);
  c->u1.reserve(m, 1.25);
  c->u2.reserve(m, 1.25);
  c->k2.reserve(m, 1.25);
  // LSD over (dn, then up): sort indices by dn, gather up, sort by up
  DevBuf<uint64_t>& key = c->k2;
  SHCI_CUDA(cudaMemcpyAsync(key.p, b.p, m * 8, cudaMemcpyDeviceToDevice, s));
  iota_u32(c->u0.p, m, s);
  radix_sort_pairs(key, c->u0, m, 0, nb, s, c->sort);
  gather_u64(a.p, c->u0.p, key.p, m, s);
  radix_sort_pairs(key, c->u0, m, 0, a_bits > 0 ? a_bits : nb, s, c->sort);
  // key = sorted ups; gather dns
  DevBuf<uint64_t> sd;
  sd.mt = &c->mem;
  sd.resize(m);
  gather_u64(b.p, c->u0.p, sd.p, m, s);
  k_unique_flags<<<grid_for(m, 256), 256, 0, s>>>(key.p, sd.p, m, c->u1.p);
  SHCI_LAUNCH_CHECK();
  const uint32_t nu = exclusive_scan_u32(c->u1.p, c->u2.p, m, s, c->sort);
  k_compact2<<<grid_for(m, 256), 256, 0, s>>>(key.p, sd.p, c->u1.p, c->u2.p, m, a.p, b.p);
  SHCI_LAUNCH_CHECK();
  c->launches += 8;
  return nu;
}

// Appends the entries of (a, b) whose a != kInvalid to (oa, ob) after *n_out (growing them);
// *n_out is advanced by the number appended.
void compact_valid(shci_ctx* c, const uint64_t* a, const uint64_t* b, size_t m,
                   DevBuf<uint64_t>& oa, DevBuf<uint64_t>& ob, size_t* n_out) {
  if (m == 0) return;
  cudaStream_t s = c->stream;
  c->u1.reserve(m, 1.25);
  c->u2.reserve(m, 1.25);
  k_valid_flags<<<grid_for(m, 256), 256, 0, s>>>(a, m, c->u1.p);
  SHCI_LAUNCH_CHECK();
  const uint32_t nv = exclusive_scan_u32(c->u1.p, c->u2.p, m, s, c->sort);
  c->launches += 3;
  if (!nv) return;
  const size_t at = *n_out;
  oa.n = ob.n = at;
  oa.grow_keep(at + nv, s);
  ob.grow_keep(at + nv, s);
  k_compact2<<<grid_for(m, 256), 256, 0, s>>>(a, b, c->u1.p, c->u2.p, m, oa.p + at, ob.p + at);
  SHCI_LAUNCH_CHECK();
  *n_out = at + nv;
}

// Inserts the det ids into the variational hash set (slot = fingerprint << 32 | id + 1,
// linear probing; the table is at most half full, so every insertion finds an empty slot).  Equal
// dets probe the same slots and slots are never emptied, so of two equal dets the one inserted
// later meets the other on its way: *dup is set.
__global__ void k_hash_insert(const uint64_t* __restrict__ up, const uint64_t* __restrict__ dn,
                              size_t n, unsigned long long* table, uint64_t mask,
                              unsigned* dup) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t u = up[i], d = dn[i];
    const uint64_t h = set_slot_hash(u, d);
    const unsigned long long v = ((h >> 32) << 32) | (static_cast<unsigned long long>(i) + 1ull);
    uint64_t p = h & mask;
    for (uint64_t probe = 0; probe <= mask; probe++) {
      const unsigned long long old = atomicCAS(&table[p], 0ull, v);
      if (old == 0ull) break;
      if ((old >> 32) == (v >> 32)) {
        const uint32_t id = static_cast<uint32_t>(old) - 1u;
        if (up[id] == u && dn[id] == d) {
          atomicOr(dup, 1u);
          atomicMin(&table[p], v);  // (the same fingerprint: the lower id stays)
          break;
        }
      }
      p = (p + 1) & mask;
    }
  }
}

// The membership set used by selection, PT2, S^2 and the 1-RDM: a hash set of the det list, a power
// of two >= 2n slots.  allow_dup: the set holds the first of each group of equal dets instead of
// refusing the list; returns whether there are such.  (The set used to come with a sorted copy of the
// list that only the duplicate check read: two radix sorts per call.)
const unsigned* build_det_set(shci_ctx* c) {
  const size_t n = c->up.size();
  cudaStream_t s = c->stream;
  c->err_word.resize(8);
  unsigned* dup = c->err_word.p;
  SHCI_CUDA(cudaMemsetAsync(dup, 0, sizeof(unsigned), s));
  size_t slots = 1024;
  while (slots < 2 * n) slots <<= 1;
  c->set_hash.mt = &c->mem;
  c->set_hash.resize(slots, 1.0);
  c->set_hash_mask = slots - 1;
  SHCI_CUDA(cudaMemsetAsync(c->set_hash.p, 0, slots * 8, s));
  k_hash_insert<<<grid_for(n, 256), 256, 0, s>>>(c->d_up.p, c->d_dn.p, n, c->set_hash.p,
                                                 c->set_hash_mask, dup);
  SHCI_LAUNCH_CHECK();
  c->launches += 1;
  return dup;
}

void check_det_set(unsigned flag) {
  if (flag) throw ArgError("the det list contains duplicates");
}

bool rebuild_det_set(shci_ctx* c, bool allow_dup) {
  const unsigned* dup = build_det_set(c);
  unsigned flag = 0;
  SHCI_CUDA(cudaMemcpyAsync(&flag, dup, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream));
  SHCI_CUDA(cudaStreamSynchronize(c->stream));
  if (!allow_dup) check_det_set(flag);
  return flag != 0;
}

namespace {

struct Candidates {
  DevBuf<ulonglong2> det;
  DevBuf<uint8_t> pass;
  size_t n = 0;
  explicit Candidates(shci_ctx* c) {
    det.mt = &c->mem;
    pass.mt = &c->mem;
  }
};

// Leaves each det once, with its lowest pass, in ascending Det order.
//
// A det is ranked among all dets of its electron counts where that rank and the pass fit 64 bits
// (2^62.3 for 10 alpha + 10 beta electrons in 40 orbitals), so that one radix sort of as few
// digits as the space has gives the order; larger spaces, or SHCI_SELECT_KEYS=strings, sort by pass,
// beta string and alpha string in turn.
void unique_candidates(shci_ctx* c, Candidates& C) {
  if (C.n == 0) return;
  if (C.n >= 0xffffffffull) throw ArgError("2^32 or more selection candidates");
  cudaStream_t s = c->stream;
  const size_t m = C.n;
  const unsigned n = c->I.n;
  std::vector<uint64_t> binom(65 * 64, 0);  // [k][pos] = C(pos, k)
  for (int pos = 0; pos < 64; pos++) {
    binom[pos] = 1;
    for (int k = 1; k <= pos; k++)
      binom[k * 64 + pos] = binom[k * 64 + pos - 1] + binom[(k - 1) * 64 + pos - 1];
  }
  auto strings = [&](unsigned ne) {  // C(n, ne)
    return ne > n ? 0ull : ne == 0 ? 1ull
                                   : binom[ne * 64 + n - 1] + binom[(ne - 1) * 64 + n - 1];
  };
  const uint64_t su = strings(c->I.n_up), sd = strings(c->I.n_dn);
  const unsigned __int128 all = static_cast<unsigned __int128>(su) * sd * 8u;
  const char* env = std::getenv("SHCI_SELECT_KEYS");
  const bool ranked = all <= (static_cast<unsigned __int128>(1) << 64) &&
                      !(env && std::strcmp(env, "strings") == 0);
  DevBuf<uint64_t>& key = c->k2;
  key.reserve(m, 1.25);
  c->u0.reserve(m, 1.25);
  c->u1.reserve(m, 1.25);
  c->u2.reserve(m, 1.25);
  if (ranked) {
    DevBuf<uint64_t> tab;
    tab.mt = &c->mem;
    tab.resize(binom.size());
    SHCI_CUDA(cudaMemcpyAsync(tab.p, binom.data(), binom.size() * 8, cudaMemcpyHostToDevice, s));
    int bits = 1;
    while (bits < 64 && (all - 1) >> bits) bits++;
    k_cand_keys<<<grid_for(m, 256), 256, 0, s>>>(C.det.p, C.pass.p, m, tab.p, sd, key.p, c->u0.p);
    SHCI_LAUNCH_CHECK();
    radix_sort_pairs(key, c->u0, m, 0, bits, s, c->sort, false);
  } else {
    iota_u32(c->u0.p, m, s);
    for (int which = 0; which < 3; which++) {
      k_cand_component<<<grid_for(m, 256), 256, 0, s>>>(C.det.p, C.pass.p, c->u0.p, m, which, key.p);
      SHCI_LAUNCH_CHECK();
      radix_sort_pairs(key, c->u0, m, 0, which == 0 ? 3 : static_cast<int>(n), s, c->sort);
    }
  }
  k_cand_first<<<grid_for(m, 256), 256, 0, s>>>(C.det.p, c->u0.p, key.p, ranked, m, c->u1.p);
  SHCI_LAUNCH_CHECK();
  const uint32_t nu = exclusive_scan_u32(c->u1.p, c->u2.p, m, s, c->sort);
  Candidates U(c);
  U.det.resize(nu);
  U.pass.resize(nu);
  k_cand_take<<<grid_for(m, 256), 256, 0, s>>>(C.det.p, C.pass.p, c->u0.p, c->u1.p, c->u2.p, m,
                                               U.det.p, U.pass.p);
  SHCI_LAUNCH_CHECK();
  C.det.swap(U.det);
  C.pass.swap(U.pass);
  C.n = nu;
  c->launches += 5;
}

}  // namespace

size_t select_dets(shci_ctx* c, double eps_var, bool var_sd) {
  if (!c->Q.built) throw ArgError("heat-bath queues not built (call shci_build_queues)");
  sync_dets(c);
  cudaStream_t s = c->stream;
  const size_t n_dets = c->up.size();
  const int n = c->I.n;
  const int n_elecs = static_cast<int>(c->I.n_up + c->I.n_dn);
  // eps_tried_prev grows with INF for new dets (solver.h:431)
  c->eps_tried.resize(n_dets, 1.0e100);
  DevBuf<double> d_eps;
  d_eps.mt = &c->mem;
  d_eps.resize(n_dets);
  SHCI_CUDA(cudaMemcpyAsync(d_eps.p, c->eps_tried.data(), n_dets * 8, cudaMemcpyHostToDevice, s));
  std::vector<uint32_t> pairs;
  for (int a = 0; a < n_elecs; a++)
    for (int b = a + 1; b < n_elecs; b++) pairs.push_back(a | (b << 16));
  DevBuf<uint32_t> d_pairs;
  d_pairs.mt = &c->mem;
  d_pairs.resize(pairs.empty() ? 1 : pairs.size());
  if (!pairs.empty())
    SHCI_CUDA(cudaMemcpyAsync(d_pairs.p, pairs.data(), pairs.size() * 4, cudaMemcpyHostToDevice, s));
  const unsigned* dup = build_det_set(c);

  SelParams P{};
  P.I = c->dI;
  P.coef = c->d_coef.p;
  P.eps_tried = d_eps.p;
  P.d_off = c->Q.d_off.p;
  P.d_H = c->Q.d_H.p;
  P.d_rs = c->Q.d_rs.p;
  P.s_off = c->Q.s_off.p;
  P.s_S = c->Q.s_S.p;
  P.s_r = c->Q.s_r.p;
  P.pair_tab = d_pairs.p;
  P.eps_var = eps_var;
  P.max_hci = c->Q.max_hci;
  P.max_singles = c->Q.max_singles;
  P.n_orbs = n;
  P.n_up = static_cast<int>(c->I.n_up);
  P.n_elecs = n_elecs;
  P.n_pairs = static_cast<int>(pairs.size());
  P.var_sd = var_sd ? 1 : 0;
  P.rej_on = c->second_rejection ? 1 : 0;
  P.rej_factor = c->second_rejection_factor;
  P.time_sym = c->time_sym ? 1 : 0;
  P.no_doubles = c->has_doubles ? 0 : 1;
  P.inactive = c->inactive_orbs;
  P.e_hf_1b = 0.0;
  if (c->second_rejection) {
    // ChemSystem::get_e_hf_1b (chem_system.cc:812-823) on dets[0]: alpha, then beta (doubled
    // alpha under time_sym)
    for (uint64_t m = c->up[0]; m; m &= m - 1) P.e_hf_1b += c->I.h(__builtin_ctzll(m), __builtin_ctzll(m));
    if (c->time_sym) {
      P.e_hf_1b *= 2.;
    } else {
      for (uint64_t m = c->dn[0]; m; m &= m - 1)
        P.e_hf_1b += c->I.h(__builtin_ctzll(m), __builtin_ctzll(m));
    }
  }

  // several states: the sources' thresholds use the largest |c| over the states
  DevBuf<double> d_selc;
  if (c->n_states > 1) {
    d_selc.mt = &c->mem;
    d_selc.resize(n_dets);
    StatePtrs xs{};
    for (unsigned k = 1; k < c->n_states; k++) xs.p[k - 1] = c->d_xcoef[k - 1].p;
    k_max_coef<<<grid_for(n_dets, 256), 256, 0, s>>>(c->d_coef.p, xs,
                                                     static_cast<int>(c->n_states - 1), n_dets,
                                                     d_selc.p);
    SHCI_LAUNCH_CHECK();
    c->launches += 1;
  }
  P.up = c->d_up.p;
  P.dn = c->d_dn.p;
  P.coef = c->n_states > 1 ? d_selc.p : c->d_coef.p;
  P.set_hash = c->set_hash.p;
  P.set_hash_mask = c->set_hash_mask;
  int sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  const unsigned grid = static_cast<unsigned>(sms) * 8u;
  const uint32_t n_src = static_cast<uint32_t>(n_dets);
  DevBuf<uint64_t> cnt;
  DevBuf<double> epsm, rejm;
  DevBuf<unsigned long long> found;
  cnt.mt = &c->mem;
  epsm.mt = rejm.mt = &c->mem;
  found.mt = &c->mem;
  cnt.resize(n_src);
  epsm.resize(n_src);
  found.resize(1);
  if (P.rej_on) {
    rejm.resize(n_src);
    SHCI_CUDA(cudaMemsetAsync(rejm.p, 0, n_src * 8ull, s));
  }
  k_sel_count<<<grid_for((size_t)n_src * 32, kSelWarps * 32, grid), kSelWarps * 32, 0, s>>>(
      P, n_src, cnt.p, epsm.p);
  SHCI_LAUNCH_CHECK();
  PieceList L(c);
  check_det_set(make_pieces(c, cnt, n_src, 1, 0.0, 0.0, nullptr, L, dup));
  Candidates C(c);
  const uint64_t kCap = 1ull << 27;  // window entries per launch, and candidates held before a sort
  uint64_t base = 0;
  for (size_t k0 = 0; k0 < L.n;) {
    uint64_t end = 0;
    const size_t k1 = piece_run(c, L, k0, base, kCap, &end);
    const uint32_t np = static_cast<uint32_t>(k1 - k0);
    // room for a third of the entries (most go to occupied orbitals or to dets of the list);
    // a launch that finds more runs again
    uint64_t room = std::min<uint64_t>(end - base, (end - base) / 3 + 4096);
    for (;;) {
      C.det.n = C.pass.n = C.n;
      C.det.grow_keep(C.n + room, s);
      C.pass.grow_keep(C.n + room, s);
      SHCI_CUDA(cudaMemsetAsync(found.p, 0, 8, s));
      {
        ProfScope ps(c->prof, s, "select_emit");
        k_sel_emit<<<grid_for((size_t)np * 32, kSelWarps * 32, grid), kSelWarps * 32, 0, s>>>(
            P, SelPieces{L.src.p + k0, L.begin.p + k0, L.len.p + k0, np}, epsm.p, C.det.p + C.n,
            C.pass.p + C.n, found.p, room, P.rej_on ? rejm.p : nullptr);
        SHCI_LAUNCH_CHECK();
      }
      unsigned long long got = 0;
      SHCI_CUDA(cudaMemcpyAsync(&got, found.p, 8, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaStreamSynchronize(s));
      c->launches += 1;
      if (got <= room) {
        C.n += got;
        break;
      }
      room = got;
    }
    if (C.n > kCap) unique_candidates(c, C);
    k0 = k1;
    base = end;
  }
  k_sel_mark<<<grid_for(n_src, 256), 256, 0, s>>>(P, n_src, epsm.p, P.rej_on ? rejm.p : nullptr);
  SHCI_LAUNCH_CHECK();
  c->launches += 2;
  unique_candidates(c, C);
  const size_t n_new_total = C.n;
  if (n_new_total) {
    // pass order, ascending Det order within a pass
    DevBuf<uint32_t> pk;
    pk.mt = &c->mem;
    pk.resize(n_new_total);
    c->u0.reserve(n_new_total, 1.25);
    k_pass_keys<<<grid_for(n_new_total, 256), 256, 0, s>>>(C.pass.p, n_new_total, pk.p, c->u0.p);
    SHCI_LAUNCH_CHECK();
    radix_sort_pairs32(pk, c->u0, n_new_total, 0, 3, s, c->sort, false);
    const size_t old = c->up.size();
    c->up.resize(old + n_new_total);
    c->dn.resize(old + n_new_total);
    c->coefs.resize(old + n_new_total, 1e-16);
    c->d_up.grow_keep(old + n_new_total, s);
    c->d_dn.grow_keep(old + n_new_total, s);
    c->d_coef.grow_keep(old + n_new_total, s);
    k_append<<<grid_for(n_new_total, 256), 256, 0, s>>>(C.det.p, c->u0.p, n_new_total,
                                                        c->d_up.p + old, c->d_dn.p + old,
                                                        c->d_coef.p + old);
    SHCI_LAUNCH_CHECK();
    SHCI_CUDA(cudaMemcpyAsync(c->up.data() + old, c->d_up.p + old, n_new_total * 8, cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaMemcpyAsync(c->dn.data() + old, c->d_dn.p + old, n_new_total * 8, cudaMemcpyDeviceToHost, s));
    // states 1..: 1e-16, except that while the list is small (<= 50 dets when this step began)
    // det k starts as state k's unit vector (solver.h:479-486)
    for (unsigned k = 1; k < c->n_states; k++) {
      auto& xc = c->d_xcoef[k - 1];
      xc.grow_keep(old + n_new_total, s);
      k_fill_coef<<<grid_for(n_new_total, 256), 256, 0, s>>>(xc.p, old, old + n_new_total, 1e-16);
      SHCI_LAUNCH_CHECK();
      if (n_dets <= 50 && k >= old && k < old + n_new_total)
        k_fill_coef<<<1, 32, 0, s>>>(xc.p, k, k + 1, 1.0);
    }
    c->launches += 5;
  }
  // eps_tried_prev back to the host mirror (only the sources of this step changed)
  SHCI_CUDA(cudaMemcpyAsync(c->eps_tried.data(), d_eps.p, n_dets * 8, cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  c->eps_tried.resize(c->up.size(), 1.0e100);
  c->prof.flush();
  return n_new_total;
}

}  // namespace shci
