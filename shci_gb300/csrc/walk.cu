// Pieces of the heat-bath windows (walk.cuh).
#include "walk.cuh"

#include <algorithm>
#include <cstdlib>

#include "kernels.h"

namespace shci {

namespace {

// Region of a piece of l entries of a source that stands for `mult` of them.
__device__ __forceinline__ uint64_t piece_region(uint64_t l, uint64_t mult, uint64_t n_batches,
                                                 double slack, double pad) {
  uint64_t r = l * mult;
  if (n_batches > 1) {
    const double est = ceil(static_cast<double>(r) / static_cast<double>(n_batches) * slack + pad);
    if (est < static_cast<double>(r)) r = est > 0.0 ? static_cast<uint64_t>(est) : 0ull;
  }
  return r;
}

// Entries of a piece: eight pieces a resident warp, within kPieceMin and kPieceLen.  (A piece costs a
// warp the search of its source's slots, about as long as a few hundred entries take.)
__device__ __forceinline__ uint32_t piece_len(unsigned long long total, uint32_t warps,
                                              uint32_t fixed) {
  if (fixed) return fixed;
  const unsigned long long len = total / (8ull * warps);
  return len <= kPieceMin ? kPieceMin : len >= kPieceLen ? kPieceLen : static_cast<uint32_t>(len);
}

__global__ void k_window_total(const uint64_t* __restrict__ entries, uint32_t n_src,
                               unsigned long long* __restrict__ total) {
  unsigned long long sum = 0;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_src; k += gridDim.x * blockDim.x)
    sum += entries[k];
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(total, sum);
}

// Pieces of every source; back[0] = the regions of all, back[2] = *flag.
__global__ void k_piece_count(const uint64_t* __restrict__ entries, uint32_t n_src,
                              uint64_t n_batches, double slack, double pad,
                              const uint32_t* __restrict__ ent_off, uint32_t warps,
                              uint32_t fixed, uint32_t* __restrict__ np, const unsigned* __restrict__ flag,
                              unsigned long long* __restrict__ back) {
  unsigned long long sum = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) back[2] = flag ? *flag : 0u;
  const uint32_t plen = piece_len(back[3], warps, fixed);
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_src;
       k += gridDim.x * blockDim.x) {
    const uint64_t m = entries[k], whole = m / plen, rest = m % plen;
    const uint64_t mult = ent_off ? ent_off[k + 1] - ent_off[k] : 1u;
    np[k] = static_cast<uint32_t>(whole + (rest != 0));
    sum += whole * piece_region(plen, mult, n_batches, slack, pad);
    if (rest) sum += piece_region(rest, mult, n_batches, slack, pad);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(back, sum);
}

// Region sizes go into off[p], to be scanned.
__global__ void k_piece_fill(const uint64_t* __restrict__ entries, const uint32_t* __restrict__ first,
                             uint32_t n_src, uint64_t n_batches, double slack, double pad,
                             const uint32_t* __restrict__ ent_off, uint32_t warps, uint32_t fixed,
                             const unsigned long long* __restrict__ total, uint32_t* __restrict__ src,
                             uint32_t* __restrict__ begin, uint32_t* __restrict__ len,
                             uint64_t* __restrict__ off) {
  const uint32_t plen = piece_len(*total, warps, fixed);
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_src;
       k += gridDim.x * blockDim.x) {
    const uint64_t m = entries[k];
    const uint64_t mult = ent_off ? ent_off[k + 1] - ent_off[k] : 1u;
    uint32_t p = first[k];
    for (uint64_t b = 0; b < m; b += plen, p++) {
      const uint64_t l = min(static_cast<unsigned long long>(plen),
                             static_cast<unsigned long long>(m - b));
      src[p] = k;
      begin[p] = static_cast<uint32_t>(b);  // (a source's windows hold fewer than 2^32 entries)
      len[p] = static_cast<uint32_t>(l);
      off[p] = piece_region(l, mult, n_batches, slack, pad);
    }
  }
}

}  // namespace

unsigned make_pieces(shci_ctx* c, const DevBuf<uint64_t>& entries, uint32_t n_src,
                     uint64_t n_batches, double slack, double pad, const uint32_t* ent_off,
                     PieceList& L, const unsigned* flag) {
  cudaStream_t s = c->stream;
  L.n = 0;
  L.tot = 0;
  if (n_src == 0) return 0;
  DevBuf<uint32_t> first;
  first.mt = &c->mem;
  first.resize(n_src);
  int sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  const uint32_t warps = static_cast<uint32_t>(sms) * kWalkWarps;
  // SHCI_WALK_PIECE sets the entries of a piece.
  const char* env = std::getenv("SHCI_WALK_PIECE");
  const uint32_t fixed = env ? static_cast<uint32_t>(std::max(1, std::atoi(env))) : 0u;
  // total of the regions, pieces, flag (one wait for these); total of the windows
  DevBuf<unsigned long long> back;
  back.mt = &c->mem;
  back.resize(4);
  SHCI_CUDA(cudaMemsetAsync(back.p, 0, 32, s));
  k_window_total<<<grid_for(n_src, 256, 152), 256, 0, s>>>(entries.p, n_src, back.p + 3);
  SHCI_LAUNCH_CHECK();
  k_piece_count<<<grid_for(n_src, 256), 256, 0, s>>>(
      entries.p, n_src, n_batches, slack, pad, ent_off, warps, fixed, first.p, flag, back.p);
  SHCI_LAUNCH_CHECK();
  exclusive_scan_u32_async(first.p, first.p, n_src, s, c->sort,
                           reinterpret_cast<uint32_t*>(back.p + 1));
  unsigned long long h[3];
  SHCI_CUDA(cudaMemcpyAsync(h, back.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  L.tot = h[0];
  L.n = static_cast<uint32_t>(h[1]);
  c->launches += 5;
  if (L.n == 0) return static_cast<unsigned>(h[2]);
  L.src.resize(L.n);
  L.begin.resize(L.n);
  L.len.resize(L.n);
  L.off.resize(L.n + 1);
  k_piece_fill<<<grid_for(n_src, 256), 256, 0, s>>>(
      entries.p, first.p, n_src, n_batches, slack, pad, ent_off, warps, fixed, back.p + 3, L.src.p,
      L.begin.p, L.len.p, L.off.p);
  SHCI_LAUNCH_CHECK();
  exclusive_scan_u64_async(L.off.p, L.off.p, L.n, s, c->sort, L.off.p + L.n);
  return static_cast<unsigned>(h[2]);
}

size_t piece_run(shci_ctx* c, const PieceList& L, size_t k0, uint64_t base, uint64_t cap,
                 uint64_t* end) {
  *end = L.tot;
  if (L.tot - base <= cap) return L.n;
  auto off_at = [&](size_t k) {
    uint64_t v = 0;
    SHCI_CUDA(cudaMemcpyAsync(&v, L.off.p + k, 8, cudaMemcpyDeviceToHost, c->stream));
    SHCI_CUDA(cudaStreamSynchronize(c->stream));
    return v;
  };
  size_t lo = k0 + 1, hi = L.n;  // off[lo] is taken in any case; off[hi] - base > cap
  while (lo + 1 < hi) {
    const size_t mid = lo + (hi - lo) / 2;
    if (off_at(mid) - base <= cap) lo = mid;
    else hi = mid;
  }
  *end = off_at(lo);
  return lo;
}

}  // namespace shci
