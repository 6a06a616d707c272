// Reduce by determinant of the PT2 stages' (det, values) records.
//
// The reference accumulates the pairs in a hash map (solver.h:700-722).  Here the records are grouped
// by a hash of the determinant of at most 32 bits: a stable radix sort of (hash, index) brings equal
// determinants together, in emission order, the records are gathered into that order once, and
// every record compares its determinant with its neighbours of the same hash, so two determinants
// with one hash (about m^2 / 2^33 pairs of m) stay apart.  The sums are formed in emission order.  An
// order by determinant is not needed (the contributions are summed afterwards, in a compensated
// fixed order).  The sort by determinant that this replaces took a radix sort for each string: at
// n = 40, 46M records, ten passes over 12-byte items and a gather per array; 13.4 -> 10.1 ms over
// the three stages of an n = 40 run (40,000 dets), 1.89 -> 1.51 ms at n = 26 (20M records).
#include <algorithm>

#include "group.cuh"
#include "heatbath.cuh"
#include "kernels.h"

namespace shci {

namespace {

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

// out[k] = rec[idx[k]]: two (four) lanes a record, 16 bytes each.
template <int NV>
__global__ void k_group_gather(const PtRec<NV>* __restrict__ rec, const uint32_t* __restrict__ idx,
                               size_t m, PtRec<NV>* __restrict__ out) {
  constexpr size_t W = sizeof(PtRec<NV>) / sizeof(uint4);
  const uint4* __restrict__ in = reinterpret_cast<const uint4*>(rec);
  uint4* __restrict__ o = reinterpret_cast<uint4*>(out);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < m * W;
       t += (size_t)gridDim.x * blockDim.x)
    o[t] = in[idx[t / W] * W + t % W];
}

// head[k] = 1 when no earlier record of the same key holds the same determinant.
template <int NV>
__global__ void k_group_heads(const uint32_t* __restrict__ key, const PtRec<NV>* __restrict__ rec,
                              size_t m, uint32_t* head) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x) {
    const uint32_t x = key[k];
    const uint64_t u = rec[k].u, d = rec[k].d;
    uint32_t first = 1;
    for (size_t j = k; j-- > 0 && key[j] == x;)
      if (rec[j].u == u && rec[j].d == d) {
        first = 0;
        break;
      }
    head[k] = first;
  }
}

__global__ void k_group_starts(const uint32_t* __restrict__ head, const uint32_t* __restrict__ pos,
                               size_t m, uint32_t* __restrict__ start) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < m;
       k += (size_t)gridDim.x * blockDim.x)
    if (head[k]) start[pos[k]] = static_cast<uint32_t>(k);
}

// Determinant g, whose first record is at start[g]: the sums run over the records of the same key
// and determinant, in order.
template <int NV>
__global__ void k_group_sum(const uint32_t* __restrict__ key, const PtRec<NV>* __restrict__ rec,
                            const uint32_t* __restrict__ start, uint32_t n, size_t m,
                            PtRec<NV>* __restrict__ out) {
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
    const size_t k = start[g];
    const uint32_t x = key[k];
    PtRec<NV> r = rec[k];
#pragma unroll
    for (int v = 0; v < NV; v++) r.v[v] += 0.0;
    for (size_t j = k + 1; j < m && key[j] == x; j++) {
      if (rec[j].u != r.u || rec[j].d != r.d) continue;
#pragma unroll
      for (int v = 0; v < NV; v++) r.v[v] += rec[j].v[v];
    }
    out[g] = r;
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
  DevBuf<uint32_t> key, start;
  DevBuf<PtRec<NV>> sorted;
  key.mt = start.mt = &c->mem;
  sorted.mt = &c->mem;
  key.resize(m);
  c->u0.resize(m, 1.25);
  k_group_keys<NV><<<grid_for(m, 256), 256, 0, s>>>(rec.p, m, tag_shift, tag_bits, bits, key.p,
                                                    c->u0.p);
  SHCI_LAUNCH_CHECK();
  radix_sort_pairs32(key, c->u0, m, 0, bits, s, c->sort, false);
  sorted.resize(m);
  k_group_gather<NV><<<grid_for(m * (sizeof(PtRec<NV>) / 16), 256), 256, 0, s>>>(rec.p, c->u0.p, m,
                                                                                 sorted.p);
  SHCI_LAUNCH_CHECK();
  c->u1.reserve(m, 1.25);
  c->u2.reserve(m, 1.25);
  k_group_heads<NV><<<grid_for(m, 256), 256, 0, s>>>(key.p, sorted.p, m, c->u1.p);
  SHCI_LAUNCH_CHECK();
  const uint32_t nu = exclusive_scan_u32(c->u1.p, c->u2.p, m, s, c->sort);
  start.resize(nu);
  k_group_starts<<<grid_for(m, 256), 256, 0, s>>>(c->u1.p, c->u2.p, m, start.p);
  SHCI_LAUNCH_CHECK();
  k_group_sum<NV><<<grid_for(nu, 256), 256, 0, s>>>(key.p, sorted.p, start.p, nu, m, rec.p);
  SHCI_LAUNCH_CHECK();
  rec.n = nu;
  c->launches += 8;
  return nu;
}

template size_t group_records<1>(shci_ctx*, DevBuf<PtRec<1>>&, size_t, int, int);
template size_t group_records<2>(shci_ctx*, DevBuf<PtRec<2>>&, size_t, int, int);
template size_t group_records<5>(shci_ctx*, DevBuf<PtRec<5>>&, size_t, int, int);

}  // namespace shci
