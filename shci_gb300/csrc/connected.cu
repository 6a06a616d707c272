// Batched connected-determinant enumeration: BaseSystem::find_connected_dets
// (src/base_system.h:57-62) as ChemSystem implements it (src/chem/chem_system.cc:289-402),
// with second rejection off, for many dets in one call.
//
// A det has a heat-bath slot per electron for single excitations and one per electron pair for
// doubles, each with its window of its queue in the reference's order.  The candidates that pass the
// occupancy checks are the dets the reference's handler would receive; a det's slots follow one
// another, so its list is in the handler's order.  A warp per unit counts (and later writes) the
// valid entries, and a scan of the counts gives every unit its offset.
//
// Few dets: the unit is one slot, its window found by a kernel before (with a warp per det, 16 dets
// of an n = 26 system kept 16 warps of the chip busy for 785 rounds per walk: 2.06 -> 0.39 ms for the
// two calls, 85 us of kernels).  Many dets: most slots' windows are empty, and a warp for each costs
// more than the walk, so the unit is 32 slots of a det or more, whose windows the lanes find and
// whose entries are flattened over them.
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "ctx.h"
#include "heatbath.cuh"
#include "kernels.h"

namespace shci {

namespace {

constexpr int kConnWarps = 8;
constexpr uint64_t kSlotUnits = 3u << 18;  // (slots_per_unit gives the reasons of these)
constexpr uint64_t kGroup32Units = 1u << 18, kGroup64Units = 1u << 20;
constexpr uint64_t kConnOut = 1u << 27;  // candidates written before they are copied out (2.3 GB)

// Window of det k: the reference returns before any handler call when eps_max < eps_min
// (chem_system.cc:295).
__device__ __forceinline__ bool conn_window(const double* eps_max, const double* eps_min,
                                            uint32_t k, double* lo, double* hi) {
  *lo = eps_min[k];
  *hi = eps_max[k];
  return !(*hi < *lo);
}

// Window of each (det, slot): {first entry, entries, slot code, 0}.
__global__ void k_conn_windows(SelParams P, const uint64_t* __restrict__ up,
                               const uint64_t* __restrict__ dn,
                               const double* __restrict__ eps_max,
                               const double* __restrict__ eps_min, uint32_t n_units, int n_slots,
                               uint4* __restrict__ win) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n_units;
       t += gridDim.x * blockDim.x) {
    const uint32_t k = t / n_slots;
    double lo, hi;
    uint32_t first = 0, cnt = 0, code = 0;
    if (conn_window(eps_max, eps_min, k, &lo, &hi))
      code = slot_range(P, up[k], dn[k], static_cast<int>(t % n_slots), lo, hi, &first, &cnt);
    win[t] = make_uint4(first, cnt, code, 0u);
  }
}

// Where the entries of the units [first, end) go: those of unit t to off[t] - base.
struct ConnOut {
  uint64_t first, end, base;
  uint64_t* up;
  uint64_t* dn;
  uint8_t* nx;
};

// Entry x of det (u, d) to place q.
__device__ __forceinline__ void conn_put(const ConnOut& out, uint64_t q, uint32_t x, uint64_t u,
                                         uint64_t d) {
  apply_entry(x, &u, &d);
  out.up[q] = u;
  out.dn[q] = d;
  out.nx[q] = x & kOne ? 1 : 2;
}

// Units of one slot.  EMIT: writes the unit's valid entries at off[unit]; else counts them into
// off[unit].
template <bool EMIT>
__global__ void __launch_bounds__(kConnWarps * 32)
    k_conn_slots(SelParams P, const uint64_t* __restrict__ up, const uint64_t* __restrict__ dn,
                 const uint4* __restrict__ win, int n_slots, uint64_t* __restrict__ off,
                 ConnOut out) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t warps = gridDim.x * kConnWarps;
  const uint32_t end = static_cast<uint32_t>(out.end);
  for (uint32_t t = static_cast<uint32_t>(out.first) + blockIdx.x * kConnWarps + (threadIdx.x >> 5);
       t < end; t += warps) {
    const uint4 w = win[t];
    const uint32_t k = t / n_slots;
    uint64_t pos = EMIT ? off[t] - out.base : 0;
    if (w.y) {
      const uint64_t u = up[k], d = dn[k];
      for (uint32_t e0 = 0; e0 < w.y; e0 += 32) {
        uint32_t x = 0;
        const bool ok = e0 + lane < w.y && entry_code(P, w.z, w.x + e0 + lane, u | P.inactive,
                                                      d | P.inactive, &x);
        const unsigned bal = __ballot_sync(kFull, ok);
        if (EMIT && ok) conn_put(out, pos + __popc(bal & lt), x, u, d);
        pos += __popc(bal);
      }
    }
    if (!EMIT && lane == 0) off[t] = pos;
  }
}

// The same for units of `per` slots (a multiple of 32, or all of a det's).
template <bool EMIT>
__global__ void __launch_bounds__(kConnWarps * 32)
    k_conn_groups(SelParams P, const uint64_t* __restrict__ up, const uint64_t* __restrict__ dn,
                  const double* __restrict__ eps_max, const double* __restrict__ eps_min,
                  int n_slots, int per, uint32_t units_per_det, uint64_t* __restrict__ off,
                  ConnOut out) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t warps = gridDim.x * kConnWarps;
  const uint32_t end = static_cast<uint32_t>(out.end);
  for (uint32_t t = static_cast<uint32_t>(out.first) + blockIdx.x * kConnWarps + (threadIdx.x >> 5);
       t < end; t += warps) {
    const uint32_t k = t / units_per_det;
    const int first = static_cast<int>(t % units_per_det) * per;
    const int last = min(n_slots, first + per);
    uint64_t pos = EMIT ? off[t] : 0;
    if (EMIT && off[t + 1] == pos) continue;
    pos -= out.base;
    double lo, hi;
    if (conn_window(eps_max, eps_min, k, &lo, &hi) &&
        !(lo > P.max_singles && lo > P.max_hci)) {  // (narrow windows of light dets are empty)
      const uint64_t u = up[k], d = dn[k];
      for (int s0 = first; s0 < last; s0 += 32) {
        uint32_t b = 0, c = 0, code = 0;
        if (s0 + (int)lane < last) code = slot_range(P, u, d, s0 + lane, lo, hi, &b, &c);
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t x = __shfl_up_sync(kFull, inc, o);
          if (lane >= (unsigned)o) inc += x;
        }
        const uint32_t total = __shfl_sync(kFull, inc, 31);
        for (uint32_t e0 = 0; e0 < total; e0 += 32) {
          const uint32_t e = e0 + lane;
          uint32_t ol = 0;  // owner: the number of slots that end at or before e
#pragma unroll
          for (uint32_t step = 16; step; step >>= 1) {
            const uint32_t v = __shfl_sync(kFull, inc, ol + step - 1);
            if (v <= e) ol += step;
          }
          const uint32_t at = e - __shfl_sync(kFull, inc - c, ol) + __shfl_sync(kFull, b, ol);
          const uint32_t o_code = __shfl_sync(kFull, code, ol);
          uint32_t x = 0;
          const bool ok = e < total && entry_code(P, o_code, at, u | P.inactive, d | P.inactive, &x);
          const unsigned bal = __ballot_sync(kFull, ok);
          if (EMIT && ok) conn_put(out, pos + __popc(bal & lt), x, u, d);
          pos += __popc(bal);
        }
      }
    }
    if (!EMIT && lane == 0) off[t] = pos;
  }
}

// Slots of a unit.  A slot each while that makes few units; then 32 of a det's slots, and more where
// even these are so many that mostly empty ones cost more than a long walk.  Both calls, for windows
// [eps / |c|, inf) of the n dets, eps = 1e-3, 1e-4, 1e-5:
//   n = 26, 14 electrons, 3,000 dets: 0.34, 0.38, 0.83 ms by slots, 0.31, 0.56, 1.12 by 32;
//   n = 40, 20 electrons, 3,000 dets (630,000 slots): 0.36, 0.56, 1.28 and 0.31, 0.71, 1.70;
//   10,000 (2.1 million): 0.67, 1.03, 3.8 and 0.43, 0.94, 4.3; 300,000: 15.3, 16.4, 43.5 by slots,
//   2.9, 4.2, 36.7 by 32 (2.1 million units), 2.5, 3.6, 37.3 by 64, 2.1, 3.4, 36.5 by 128;
//   60,000: 0.88, 1.81 by 32 (420,000 units), 0.77, 1.85 by 64, 0.77, 2.07 by 128.
int slots_per_unit(uint64_t n, uint64_t n_slots) {
  // SHCI_CONNECTED_SLOTS sets them.
  if (const char* env = std::getenv("SHCI_CONNECTED_SLOTS"))
    return std::min(1 << 20, std::max(1, std::atoi(env)));
  if (n * n_slots <= kSlotUnits) return 1;
  const uint64_t units = n * ((n_slots + 31) / 32);
  return units <= kGroup32Units ? 32 : units <= kGroup64Units ? 64 : 128;
}

// cnt[k] = entries of det k, from the scanned unit offsets.
__global__ void k_conn_totals(const uint64_t* __restrict__ off, const uint64_t* __restrict__ total,
                              uint32_t n, uint32_t units_per_det, uint64_t* __restrict__ cnt) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const uint64_t a = off[(size_t)k * units_per_det];
    cnt[k] = (k + 1 < n ? off[(size_t)(k + 1) * units_per_det] : *total) - a;
  }
}

SelParams conn_params(shci_ctx* c, DevBuf<uint32_t>& pairs) {
  if (!c->Q.built) upload_queues(c);
  const int n_elecs = static_cast<int>(c->I.n_up + c->I.n_dn);
  std::vector<uint32_t> pr;
  for (int a = 0; a < n_elecs; a++)
    for (int b = a + 1; b < n_elecs; b++) pr.push_back(a | (b << 16));
  pairs.mt = &c->mem;
  pairs.resize(pr.empty() ? 1 : pr.size());
  if (!pr.empty())
    SHCI_CUDA(cudaMemcpyAsync(pairs.p, pr.data(), pr.size() * 4, cudaMemcpyHostToDevice,
                              c->stream));
  SelParams P{};
  P.I = c->dI;
  P.d_off = c->Q.d_off.p;
  P.d_H = c->Q.d_H.p;
  P.d_rs = c->Q.d_rs.p;
  P.s_off = c->Q.s_off.p;
  P.s_S = c->Q.s_S.p;
  P.s_r = c->Q.s_r.p;
  P.pair_tab = pairs.p;
  P.max_hci = c->Q.max_hci;
  P.max_singles = c->Q.max_singles;
  P.n_orbs = c->I.n;
  P.n_up = static_cast<int>(c->I.n_up);
  P.n_elecs = n_elecs;
  P.n_pairs = static_cast<int>(pr.size());
  P.no_doubles = c->has_doubles ? 0 : 1;
  P.inactive = c->inactive_orbs;
  return P;
}

}  // namespace

void find_connected(shci_ctx* c, const uint64_t* up, const uint64_t* dn, const double* eps_max,
                    const double* eps_min, size_t n, uint64_t* offsets, uint64_t* out_up,
                    uint64_t* out_dn, uint8_t* n_excite) {
  if (n == 0) {
    if (offsets) offsets[0] = 0;
    return;
  }
  if (n >= 0xffffffffull) throw ArgError("more than 2^32-1 dets in one call");
  if (!up || !dn || !eps_max || !eps_min || !offsets) throw ArgError("null input pointer");
  const bool emit = out_up != nullptr;
  if (emit && (!out_dn || !n_excite)) throw ArgError("null output pointer");
  const int n_up = static_cast<int>(c->I.n_up), n_dn = static_cast<int>(c->I.n_dn);
  for (size_t k = 0; k < n; k++)
    if (__builtin_popcountll(up[k]) != n_up || __builtin_popcountll(dn[k]) != n_dn)
      throw ArgError("det " + std::to_string(k) + " does not have the system's electron counts");
  cudaStream_t s = c->stream;
  DevBuf<uint32_t> pairs;
  const SelParams P = conn_params(c, pairs);
  const int n_slots = P.n_elecs + P.n_pairs;
  int per = slots_per_unit(n, n_slots);
  // (units are counted in 32 bits)
  if (n_slots == 0 || n * (uint64_t)((n_slots + per - 1) / per) > 1u << 31) per = std::max(2, n_slots);
  bool by_slot = per == 1;
  // One pass over all dets where their arrays fit, else whole dets as units, then passes.
  size_t step = n, m_max = n;
  uint32_t units_per_det = 0;
  DevBuf<uint64_t> d_up, d_dn, d_cnt, d_off;
  DevBuf<double> d_hi, d_lo;
  DevBuf<uint4> d_win;
  d_up.mt = d_dn.mt = d_cnt.mt = d_off.mt = &c->mem;
  d_hi.mt = d_lo.mt = &c->mem;
  d_win.mt = &c->mem;
  for (;;) {
    units_per_det = static_cast<uint32_t>(std::max(1, (n_slots + per - 1) / per));
    try {
      d_up.resize(m_max);
      d_dn.resize(m_max);
      d_hi.resize(m_max);
      d_lo.resize(m_max);
      d_cnt.resize(m_max);
      if (by_slot) d_win.resize(m_max * n_slots);
      d_off.resize(m_max * units_per_det + 1);
      break;
    } catch (const OomError&) {
      for (auto* b : {&d_up, &d_dn, &d_cnt, &d_off}) b->release();
      d_hi.release();
      d_lo.release();
      d_win.release();
      if (by_slot || units_per_det > 1) {
        by_slot = false;
        per = std::max(2, n_slots);
      } else if (m_max == 1) {
        throw;
      } else {
        m_max = step = (m_max + 7) / 8;
      }
    }
  }
  DevBuf<uint64_t> o_up, o_dn;
  DevBuf<uint8_t> o_nx;
  o_up.mt = o_dn.mt = &c->mem;
  o_nx.mt = &c->mem;
  int sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  if (emit && offsets[0] != 0)
    throw ArgError("offsets[0] must be 0 (pass the count call's offsets)");
  if (!emit) offsets[0] = 0;
  std::vector<uint64_t> cnt(m_max);
  auto walk = [&](bool write, const ConnOut& o) {
    const unsigned grid =
        grid_for((size_t)(o.end - o.first) * 32, kConnWarps * 32, (unsigned)sms * 8u);
    if (by_slot) {
      const auto k = write ? k_conn_slots<true> : k_conn_slots<false>;
      k<<<grid, kConnWarps * 32, 0, s>>>(P, d_up.p, d_dn.p, d_win.p, n_slots, d_off.p, o);
    } else {
      const auto k = write ? k_conn_groups<true> : k_conn_groups<false>;
      k<<<grid, kConnWarps * 32, 0, s>>>(P, d_up.p, d_dn.p, d_hi.p, d_lo.p, n_slots, per,
                                         units_per_det, d_off.p, o);
    }
    SHCI_LAUNCH_CHECK();
    c->launches += 1;
  };
  // Counts of the dets [b, b + m): into offsets, or (emit) compared with them.
  auto count = [&](size_t b, uint32_t m) {
    const uint64_t units = m * (uint64_t)units_per_det;
    SHCI_CUDA(cudaMemcpyAsync(d_up.p, up + b, m * 8ull, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_dn.p, dn + b, m * 8ull, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_hi.p, eps_max + b, m * 8ull, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_lo.p, eps_min + b, m * 8ull, cudaMemcpyHostToDevice, s));
    if (by_slot) {
      k_conn_windows<<<grid_for(units, 256), 256, 0, s>>>(
          P, d_up.p, d_dn.p, d_hi.p, d_lo.p, static_cast<uint32_t>(units), n_slots, d_win.p);
      SHCI_LAUNCH_CHECK();
      c->launches += 1;
    }
    walk(false, ConnOut{0, units, 0, nullptr, nullptr, nullptr});
    exclusive_scan_u64_async(d_off.p, d_off.p, units, s, c->sort, d_off.p + units);
    k_conn_totals<<<grid_for(m, 256), 256, 0, s>>>(d_off.p, d_off.p + units, m, units_per_det,
                                                   d_cnt.p);
    SHCI_LAUNCH_CHECK();
    SHCI_CUDA(cudaMemcpyAsync(cnt.data(), d_cnt.p, m * 8ull, cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
    c->launches += 3;
    const uint64_t* cn = cnt.data();
    uint64_t* o = offsets + b;
    if (!emit) {
      uint64_t sum = o[0];
      for (uint32_t k = 0; k < m; k++) o[k + 1] = sum += cn[k];
      return;
    }
    bool same = true;
    for (uint32_t k = 0; k < m; k++) same &= o[k + 1] >= o[k] && o[k + 1] - o[k] == cn[k];
    if (!same)
      throw ArgError("offsets do not match the connected-det counts (pass the count call's "
                     "offsets)");
  };
  // The lists go to the caller's offsets, which must be the count call's (a region too small would
  // be overrun): all of them are compared before anything is written.
  for (size_t b = 0; b < n; b += step) count(b, static_cast<uint32_t>(std::min(step, n - b)));
  if (!emit) return;
  uint64_t cap = kConnOut;
  for (size_t b = 0; b < n; b += step) {
    const size_t end = std::min(n, b + step);
    if (n > step) count(b, static_cast<uint32_t>(end - b));  // (one pass has its offsets at hand)
    for (size_t k = b; k < end;) {  // whole dets of at most `cap` candidates (one at least)
      const size_t k1 =
          std::max<size_t>(k + 1, std::upper_bound(offsets + k, offsets + end + 1, offsets[k] + cap) -
                                      offsets - 1);
      const uint64_t at = offsets[k], total = offsets[k1] - at;
      try {
        o_up.resize(total);
        o_dn.resize(total);
        o_nx.resize(total);
      } catch (const OomError&) {
        if (k1 == k + 1) throw;
        o_up.release();
        o_dn.release();
        o_nx.release();
        cap = total / 8;
        continue;
      }
      if (total) {
        walk(true, ConnOut{(k - b) * (uint64_t)units_per_det, (k1 - b) * (uint64_t)units_per_det,
                           at - offsets[b], o_up.p, o_dn.p, o_nx.p});
        SHCI_CUDA(cudaMemcpyAsync(out_up + at, o_up.p, total * 8, cudaMemcpyDeviceToHost, s));
        SHCI_CUDA(cudaMemcpyAsync(out_dn + at, o_dn.p, total * 8, cudaMemcpyDeviceToHost, s));
        SHCI_CUDA(cudaMemcpyAsync(n_excite + at, o_nx.p, total, cudaMemcpyDeviceToHost, s));
        SHCI_CUDA(cudaStreamSynchronize(s));
      }
      k = k1;
    }
  }
}

}  // namespace shci
