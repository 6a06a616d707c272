// Work items of the row kernels: a warp per piece of a row.
//
// A warp per row makes the longest row the kernel's time when the matrix is small: the first
// determinants connect to most of the list (100,000 elements at 400,000 dets, n = 40), and one
// warp walks 32 elements per round of dependent loads (about 1.2 us).  Rows are therefore cut
// into pieces of kItemLen elements, listed once per build, and the warps of a grid take the pieces
// of all segments in turn.
#pragma once

#include "ctx.h"

namespace shci {

// 512 elements are 16 rounds of a warp (about 20 us): the tail a launch can have.  Shorter pieces pay
// the row's reduction and atomic more often, longer ones lengthen the tail: 48 products of an n = 26
// variation 8.0 ms, 8.5 with pieces of 1,024, 8.3 with 256; 1.25 G elements 6.96, 6.99 and 7.01 ms.
constexpr uint32_t kItemLen = 512;

struct ItemSeg {
  const uint4* items;       // null: whole rows
  const uint32_t* n_items;  // device
  const uint64_t* row_ptr;
  const uint32_t* row_cnt;
  uint32_t n;               // rows
  uint64_t base;            // first output index of the segment's items
  const uint32_t* col;
  const double* v64;
  const float* v32;
  const float* r32;
};

struct ItemTab {
  int n;
  ItemSeg s[kMaxSegments];
};

// The items of all segments of H; *len = bound on their number.
inline ItemTab item_tab(const DevHamiltonian& H, size_t* len = nullptr) {
  ItemTab t{};
  uint64_t base = 0;
  for (const SegView& g : segments(H)) {
    const bool ok = g.items->ok;
    t.s[t.n++] = ItemSeg{ok ? g.items->it.p : nullptr, ok ? g.items->off.p + g.n : nullptr,
                         g.row_ptr, g.row_cnt, static_cast<uint32_t>(g.n), base, g.col,
                         g.val64, g.val32, g.res32};
    base += ok ? g.items->cap : g.n;
  }
  if (len) *len = base;
  return t;
}

// f(segment, output index, row, start, length) for the calling warp's share of the items.
template <class F>
__device__ __forceinline__ void for_items(const ItemTab& T, F&& f) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (int g = 0; g < T.n; g++) {
    const ItemSeg& S = T.s[g];
    const uint32_t m = S.items ? *S.n_items : S.n;
    for (; t < m; t += warps) {
      if (S.items) {
        const uint4 v = __ldg(S.items + t);
        f(S, S.base + t, v.x, v.z | (static_cast<uint64_t>(v.w) << 32), v.y);
      } else {
        f(S, S.base + t, t, S.row_ptr[t], S.row_cnt[t]);
      }
    }
    t -= m;
  }
}

}  // namespace shci
