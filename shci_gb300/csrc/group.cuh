// Records of the PT2 stages: a determinant (alpha string, with an iteration tag above the orbital
// bits in the stochastic stage, and beta string) and its NV values, in one or two 32-byte sectors, so
// that the reduction's random read of a record costs one or two sectors instead of one per array.
#pragma once

#include "ctx.h"

namespace shci {

template <int NV>
struct alignas(32) PtRec {
  uint64_t u, d;
  double v[NV];
};
static_assert(sizeof(PtRec<1>) == 32 && sizeof(PtRec<2>) == 32 && sizeof(PtRec<5>) == 64,
              "records are whole sectors");

// group.cu: sums the values of equal determinants of the first m records in input order.  The
// distinct determinants (the tag, tag_bits bits from tag_shift up, is the outermost order; otherwise
// unordered) and their sums are left in rec; returns their number.
template <int NV>
size_t group_records(shci_ctx* c, DevBuf<PtRec<NV>>& rec, size_t m, int tag_shift, int tag_bits);

}  // namespace shci
