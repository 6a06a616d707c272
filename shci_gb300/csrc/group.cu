// Reduce by determinant of the PT2 stages' (det, values) records.
//
// The reference accumulates the pairs in a hash map (solver.h:700-722).  Here the records are grouped
// by a hash of the determinant of at most 32 bits: a stable radix sort of (hash, index) brings equal
// determinants together, in emission order, the records are gathered into that order once, and
// every record compares its determinant with its neighbours of the same hash, so two determinants
// with one hash (about m^2 / 2^33 pairs of m) stay apart.  The sums are formed in an order that the
// records fix.  An order by determinant is not needed (the contributions are summed afterwards, in a
// compensated fixed order).  The sort by determinant that this replaces took a radix sort for each
// string, ten passes over 12-byte items and a gather per array: 13.4 -> 7.6 ms over the three stages
// of an n = 40 run (40,000 dets, 50M records in the first), 1.89 -> 1.20 ms at n = 26 (20M records).
#include <algorithm>

#include "group.cuh"
#include "heatbath.cuh"
#include "kernels.h"

namespace shci {

namespace {

constexpr int kGroupWarps = 8;

// Key: the iteration tag (bits tag_shift .. of u) above the top bits of the hash; idx = k.
template <int NV>
__global__ void k_group_keys(const PtRec<NV>* __restrict__ rec, size_t m, int tag_shift,
                             int tag_bits, int bits, uint32_t* __restrict__ key,
                             uint32_t* __restrict__ idx) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    const uint64_t u = rec[k].u;
    const uint32_t h =
        static_cast<uint32_t>(set_slot_hash(u, rec[k].d) >> 32) >> (32 - bits + tag_bits);
    key[k] = tag_bits ? h | (static_cast<uint32_t>(u >> tag_shift) << (bits - tag_bits)) : h;
    idx[k] = static_cast<uint32_t>(k);
  }
}

// out[k] = rec[idx[k]], and heads: bit k % 32 of mask[k / 32] is set when no earlier record of the
// same key holds the same determinant; cnt[k / 32] is the number of these.  A warp per 32 records,
// two (four) lanes a record, 16 bytes each; their determinants pass through shared memory to be
// compared with the one before.
template <int NV>
__global__ void __launch_bounds__(kGroupWarps * 32)
    k_group_gather(const PtRec<NV>* __restrict__ rec, const uint32_t* __restrict__ idx,
                   const uint32_t* __restrict__ key, size_t m, PtRec<NV>* __restrict__ out,
                   uint32_t* __restrict__ mask, uint32_t* __restrict__ cnt) {
  constexpr int W = sizeof(PtRec<NV>) / sizeof(uint4);
  __shared__ uint4 s_det[kGroupWarps][33];  // determinants of the record before and the warp's 32
  const int lane = threadIdx.x & 31;
  uint4* det = s_det[threadIdx.x >> 5];
  const uint4* __restrict__ in = reinterpret_cast<const uint4*>(rec);
  uint4* __restrict__ o = reinterpret_cast<uint4*>(out);
  const size_t n_words = (m + 31) / 32;
  for (size_t w = blockIdx.x * (size_t)kGroupWarps + (threadIdx.x >> 5); w < n_words;
       w += (size_t)gridDim.x * kGroupWarps) {
    const size_t k0 = w * 32, k = k0 + lane;
    const uint32_t at = k < m ? idx[k] : 0u;
    const uint32_t x = k < m ? key[k] : 0u;
    const uint32_t x0 = k && k < m ? key[k - 1] : ~x;
    uint4 a[W], before;
    if (lane == 0 && k0) before = in[(size_t)idx[k0 - 1] * W];
#pragma unroll
    for (int t = 0; t < W; t++) {
      const int r = (t * 32 + lane) / W;
      const uint32_t src = __shfl_sync(kFull, at, r);
      if (k0 + r < m) a[t] = in[(size_t)src * W + lane % W];
    }
    if (lane == 0 && k0) det[0] = before;
#pragma unroll
    for (int t = 0; t < W; t++) {
      const int r = (t * 32 + lane) / W;
      if (k0 + r >= m) continue;
      o[(k0 + r) * W + lane % W] = a[t];
      if (lane % W == 0) det[1 + r] = a[t];
    }
    __syncwarp();
    bool head = k < m;
    if (head && x == x0) {
      const uint4 p = det[1 + lane], q = det[lane];
      head = (p.x ^ q.x) | (p.y ^ q.y) | (p.z ^ q.z) | (p.w ^ q.w);
      for (size_t j = k - 1; head && j-- > 0 && key[j] == x;) {  // (determinants of one hash)
        const uint4 e = in[(size_t)idx[j] * W];
        head = (p.x ^ e.x) | (p.y ^ e.y) | (p.z ^ e.z) | (p.w ^ e.w);
      }
    }
    const unsigned heads = __ballot_sync(kFull, head);
    if (lane == 0) {
      mask[w] = heads;
      cnt[w] = __popc(heads);
    }
    __syncwarp();  // every lane has read det
  }
}

// The sums, to out[pos[k / 32] + heads before k in its word] for every head k.  A warp per 32
// records: a run of one determinant is summed by halving distances among its lanes; the run that
// goes on behind the warp's records is followed by all lanes, and a determinant that shares its
// key with others by its head's lane.  Bound by the FP64 pipe (a warp's addition takes 16 cycles
// however few lanes need it), so no step is taken that no head needs.  Over the stages of an n = 40
// run (50M, 2 x 10M and 14M records): 0.67 + 0.64 + 0.88 ms (0.94 + 0.83 + 1.25 when every run was
// summed over five steps), against 1.04 + 1.11 + 1.40 for a thread per determinant, which waits in
// each warp for the longest run of 32, and another 1.1 ms of passes for its list of heads.
template <int NV>
__global__ void __launch_bounds__(kGroupWarps * 32)
    k_group_sum(const uint32_t* __restrict__ key, const PtRec<NV>* __restrict__ rec,
                const uint32_t* __restrict__ mask, const uint32_t* __restrict__ pos, size_t m,
                PtRec<NV>* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const size_t n_words = (m + 31) / 32;
  for (size_t w = blockIdx.x * (size_t)kGroupWarps + (threadIdx.x >> 5); w < n_words;
       w += (size_t)gridDim.x * kGroupWarps) {
    const size_t k = w * 32 + lane;
    PtRec<NV> r = rec[k < m ? k : m - 1];
    const uint32_t x = key[k < m ? k : m - 1];
    const unsigned heads = mask[w];
    const uint32_t at = pos[w];
    if (!heads) continue;
    const uint64_t pu = __shfl_up_sync(kFull, r.u, 1), pd = __shfl_up_sync(kFull, r.d, 1);
    const uint32_t px = __shfl_up_sync(kFull, x, 1);
    const bool starts = lane == 0 || k >= m || x != px || r.u != pu || r.d != pd;
    const unsigned runs = __ballot_sync(kFull, starts);
    const unsigned later = lane == 31 ? 0u : runs >> (lane + 1);
    const int end = later ? lane + __ffs(later) : 32;  // the lane behind this one's run
    const int begin = 31 - __clz(runs & (0xffffffffu >> (31 - lane)));
    const int stop = (heads >> begin) & 1u ? end : 0;  // (runs that began before are not summed here)
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) {
      const bool take = lane + h < stop;
      if (!__any_sync(kFull, take)) break;
#pragma unroll
      for (int v = 0; v < NV; v++) {
        const double t = __shfl_down_sync(kFull, r.v[v], h);
        if (take) r.v[v] += t;
      }
    }
    const bool head = (heads >> lane) & 1u;
    size_t q = w * 32 + end;  // the record behind the run
    const int last = 31 - __clz(runs);
    if ((heads >> last & 1u) && w * 32 + 32 < m) {  // the last run goes on?
      const uint32_t lx = __shfl_sync(kFull, x, last);
      const uint64_t lu = __shfl_sync(kFull, r.u, last), ld = __shfl_sync(kFull, r.d, last);
      double acc[NV];
      size_t p0 = w * 32 + 32;
      int more, width = 0;  // lanes that hold a sum
      do {
        const size_t p = p0 + lane;
        const bool in = p < m && key[p] == lx && rec[p].u == lu && rec[p].d == ld;
        const unsigned out_of = ~__ballot_sync(kFull, in);
        more = out_of ? __ffs(out_of) - 1 : 32;
        if (lane < more) {
#pragma unroll
          for (int v = 0; v < NV; v++) acc[v] = width ? acc[v] + rec[p].v[v] : rec[p].v[v];
        }
        width = max(width, more);
        p0 += more;
      } while (more == 32);
      if (width) {
        for (int h = 1; h < width; h <<= 1) {
#pragma unroll
          for (int v = 0; v < NV; v++) {
            const double t = __shfl_down_sync(kFull, acc[v], h);
            if (lane + h < width) acc[v] += t;
          }
        }
#pragma unroll
        for (int v = 0; v < NV; v++) {
          const double t = __shfl_sync(kFull, acc[v], 0);
          if (lane == last) r.v[v] += t;
        }
      }
      if (lane == last) q = p0;
    }
    const uint32_t qx = __shfl_sync(kFull, x, end & 31);
    if (!head) continue;
    // other determinants of its key follow?
    for (bool more = end < 32 ? qx == x && q < m : q < m && key[q] == x; more;
         q++, more = q < m && key[q] == x) {
      if (rec[q].u != r.u || rec[q].d != r.d) continue;
#pragma unroll
      for (int v = 0; v < NV; v++) r.v[v] += rec[q].v[v];
    }
#pragma unroll
    for (int v = 0; v < NV; v++)
      if (static_cast<uint64_t>(__double_as_longlong(r.v[v])) == 1ull << 63) r.v[v] = 0.0;
    out[at + __popc(heads & ((1u << lane) - 1u))] = r;
  }
}

}  // namespace

template <int NV>
size_t group_records(shci_ctx* c, DevBuf<PtRec<NV>>& rec, size_t m, int tag_shift, int tag_bits) {
  if (m == 0) return 0;
  if (m >= 0xffffffffull) throw ArgError("2^32 or more PT records");
  cudaStream_t s = c->stream;
  // hash bits: six more than it takes to count the records, in whole digits
  int bits = 8;
  while (bits < 32 && (static_cast<uint64_t>(m) << (6 + tag_bits)) >> bits) bits += 8;
  DevBuf<uint32_t> key, mask, pos;
  DevBuf<PtRec<NV>> sorted;
  key.mt = mask.mt = pos.mt = &c->mem;
  sorted.mt = &c->mem;
  key.resize(m);
  c->u0.resize(m, 1.25);
  k_group_keys<NV><<<grid_for(m, 256), 256, 0, s>>>(rec.p, m, tag_shift, tag_bits, bits, key.p,
                                                    c->u0.p);
  SHCI_LAUNCH_CHECK();
  radix_sort_pairs32(key, c->u0, m, 0, bits, s, c->sort, false);
  sorted.resize(m);
  const size_t words = (m + 31) / 32;
  mask.resize(words);
  pos.resize(words);
  const unsigned grid = grid_for(m, kGroupWarps * 32);
  k_group_gather<NV><<<grid, kGroupWarps * 32, 0, s>>>(rec.p, c->u0.p, key.p, m, sorted.p, mask.p,
                                                       pos.p);
  SHCI_LAUNCH_CHECK();
  const uint32_t nu = exclusive_scan_u32(pos.p, pos.p, words, s, c->sort);
  k_group_sum<NV><<<grid, kGroupWarps * 32, 0, s>>>(key.p, sorted.p, mask.p, pos.p, m, rec.p);
  SHCI_LAUNCH_CHECK();
  rec.n = nu;
  c->launches += 6;
  return nu;
}

template size_t group_records<1>(shci_ctx*, DevBuf<PtRec<1>>&, size_t, int, int);
template size_t group_records<2>(shci_ctx*, DevBuf<PtRec<2>>&, size_t, int, int);
template size_t group_records<5>(shci_ctx*, DevBuf<PtRec<5>>&, size_t, int, int);

}  // namespace shci
