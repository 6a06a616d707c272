// Batched connected-determinant enumeration: BaseSystem::find_connected_dets
// (src/base_system.h:57-62) as ChemSystem implements it (src/chem/chem_system.cc:289-402),
// with second rejection off, for many dets in one call.
//
// The work unit is one heat-bath slot of one det: a slot per electron for single excitations, one
// per electron pair for doubles, each with its window of its queue in the reference's order.  The
// candidates that pass the occupancy checks are the dets the reference's handler would receive; a
// det's slots follow one another, so its list is in the handler's order.  One kernel finds the
// windows, a warp per unit counts (and later writes) the valid entries, and a scan of the counts
// gives every unit its offset.  With a warp per det, 16 dets of the n = 26 workload kept 16 warps
// of the chip busy for 785 rounds per walk: 2.06 -> 0.39 ms for the two calls (98 us of kernels).
#include <algorithm>
#include <vector>

#include "ctx.h"
#include "heatbath.cuh"
#include "kernels.h"

namespace shci {

namespace {

constexpr int kConnWarps = 8;

// Window of det k: the reference returns before any handler call when eps_max < eps_min
// (chem_system.cc:295).
__device__ __forceinline__ bool conn_window(const double* eps_max, const double* eps_min,
                                            uint32_t k, double* lo, double* hi) {
  *lo = eps_min[k];
  *hi = eps_max[k];
  return !(*hi < *lo);
}

// Window of each (det, slot): {first entry, entries, electron orbitals (make_candidate_at), 0}.
__global__ void k_conn_windows(SelParams P, const uint64_t* __restrict__ up,
                               const uint64_t* __restrict__ dn,
                               const double* __restrict__ eps_max,
                               const double* __restrict__ eps_min, uint32_t n_units, int n_slots,
                               uint4* __restrict__ win) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n_units;
       t += gridDim.x * blockDim.x) {
    const uint32_t k = t / n_slots;
    double lo, hi;
    uint32_t first = 0, cnt = 0, orbs = 0;
    if (conn_window(eps_max, eps_min, k, &lo, &hi))
      slot_range(P, up[k], dn[k], static_cast<int>(t % n_slots), lo, hi, &first, &cnt, &orbs);
    win[t] = make_uint4(first, cnt, orbs, 0u);
  }
}

// EMIT: writes the unit's valid entries at off[unit]; else counts them into off[unit].
template <bool EMIT>
__global__ void __launch_bounds__(kConnWarps * 32)
    k_conn_walk(SelParams P, const uint64_t* __restrict__ up, const uint64_t* __restrict__ dn,
                const uint4* __restrict__ win, uint32_t n_units, int n_slots,
                uint64_t* __restrict__ off, uint64_t* __restrict__ out_up,
                uint64_t* __restrict__ out_dn, uint8_t* __restrict__ out_nx) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t warps = gridDim.x * kConnWarps;
  for (uint32_t t = blockIdx.x * kConnWarps + (threadIdx.x >> 5); t < n_units; t += warps) {
    const uint4 w = win[t];
    const uint32_t k = t / n_slots;
    const int slot = static_cast<int>(t % n_slots);
    uint64_t pos = EMIT ? off[t] : 0;
    if (w.y) {
      const uint64_t u = up[k], d = dn[k];
      for (uint32_t e0 = 0; e0 < w.y; e0 += 32) {
        uint64_t cu = 0, cd = 0;
        const bool ok = e0 + lane < w.y &&
                        make_candidate_at(P, u, d, slot, w.z, w.x + e0 + lane, &cu, &cd);
        const unsigned bal = __ballot_sync(kFull, ok);
        if (EMIT && ok) {
          const uint64_t q = pos + __popc(bal & lt);
          out_up[q] = cu;
          out_dn[q] = cd;
          out_nx[q] = slot < P.n_elecs ? 1 : 2;
        }
        pos += __popc(bal);
      }
    }
    if (!EMIT && lane == 0) off[t] = pos;
  }
}

// cnt[k] = entries of det k, from the scanned unit offsets.
__global__ void k_conn_totals(const uint64_t* __restrict__ off, const uint64_t* __restrict__ total,
                              uint32_t n, int n_slots, uint64_t* __restrict__ cnt) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const uint64_t a = off[(size_t)k * n_slots];
    cnt[k] = (k + 1 < n ? off[(size_t)(k + 1) * n_slots] : *total) - a;
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
  if (n_slots == 0) {  // no electrons
    for (size_t k = 0; k <= n; k++) {
      if (emit && offsets[k] != 0) throw ArgError("offsets do not match the connected-det counts");
      offsets[k] = 0;
    }
    return;
  }
  // dets per pass: the units' windows and offsets (24 bytes each) stay within 100 MB, or what
  // there is room for
  size_t step = std::max<size_t>(1, (size_t{1} << 22) / n_slots);
  size_t m_max = std::min(n, step);
  DevBuf<uint64_t> d_up, d_dn, d_cnt, d_off;
  DevBuf<double> d_hi, d_lo;
  DevBuf<uint4> d_win;
  d_up.mt = d_dn.mt = d_cnt.mt = d_off.mt = &c->mem;
  d_hi.mt = d_lo.mt = &c->mem;
  d_win.mt = &c->mem;
  for (;;) {
    try {
      d_up.resize(m_max);
      d_dn.resize(m_max);
      d_hi.resize(m_max);
      d_lo.resize(m_max);
      d_cnt.resize(m_max);
      d_win.resize(m_max * n_slots);
      d_off.resize(m_max * n_slots + 1);
      break;
    } catch (const OomError&) {
      if (m_max == 1) throw;
      d_win.release();
      d_off.release();
      m_max = step = (m_max + 7) / 8;
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
  unsigned grid = 0;
  // Counts of the dets [b, b + m): into offsets, or (emit) compared with them.
  auto count = [&](size_t b, uint32_t m) {
    const uint32_t units = m * static_cast<uint32_t>(n_slots);
    SHCI_CUDA(cudaMemcpyAsync(d_up.p, up + b, m * 8ull, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_dn.p, dn + b, m * 8ull, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_hi.p, eps_max + b, m * 8ull, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(d_lo.p, eps_min + b, m * 8ull, cudaMemcpyHostToDevice, s));
    k_conn_windows<<<grid_for(units, 256), 256, 0, s>>>(P, d_up.p, d_dn.p, d_hi.p, d_lo.p, units,
                                                        n_slots, d_win.p);
    SHCI_LAUNCH_CHECK();
    grid = grid_for((size_t)units * 32, kConnWarps * 32, (unsigned)sms * 8u);
    k_conn_walk<false><<<grid, kConnWarps * 32, 0, s>>>(P, d_up.p, d_dn.p, d_win.p, units, n_slots,
                                                        d_off.p, nullptr, nullptr, nullptr);
    SHCI_LAUNCH_CHECK();
    exclusive_scan_u64_async(d_off.p, d_off.p, units, s, c->sort, d_off.p + units);
    k_conn_totals<<<grid_for(m, 256), 256, 0, s>>>(d_off.p, d_off.p + units, m, n_slots, d_cnt.p);
    SHCI_LAUNCH_CHECK();
    SHCI_CUDA(cudaMemcpyAsync(cnt.data(), d_cnt.p, m * 8ull, cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
    c->launches += 5;
    for (uint32_t k = 0; k < m; k++)
      if (!emit)
        offsets[b + k + 1] = offsets[b + k] + cnt[k];
      else if (offsets[b + k + 1] < offsets[b + k] || offsets[b + k + 1] - offsets[b + k] != cnt[k])
        throw ArgError("offsets do not match the connected-det counts (pass the count call's "
                       "offsets)");
  };
  // The lists go to the caller's offsets, which must be the count call's (a region too small would
  // be overrun): all of them are compared before anything is written.
  for (size_t b = 0; b < n; b += step) count(b, static_cast<uint32_t>(std::min(step, n - b)));
  if (!emit) return;
  for (size_t b = 0; b < n; b += step) {
    const uint32_t m = static_cast<uint32_t>(std::min(step, n - b));
    const uint32_t units = m * static_cast<uint32_t>(n_slots);
    if (n > step) count(b, m);  // (a single pass has its unit offsets at hand)
    const uint64_t at = offsets[b], total = offsets[b + m] - at;
    if (!total) continue;
    o_up.resize(total);
    o_dn.resize(total);
    o_nx.resize(total);
    k_conn_walk<true><<<grid, kConnWarps * 32, 0, s>>>(P, d_up.p, d_dn.p, d_win.p, units, n_slots,
                                                       d_off.p, o_up.p, o_dn.p, o_nx.p);
    SHCI_LAUNCH_CHECK();
    c->launches += 1;
    SHCI_CUDA(cudaMemcpyAsync(out_up + at, o_up.p, total * 8, cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaMemcpyAsync(out_dn + at, o_dn.p, total * 8, cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaMemcpyAsync(n_excite + at, o_nx.p, total, cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
  }
}

}  // namespace shci
