// The fixed-point scale of the mixed H*v (spmv.cu), shared with the kernels that read its sums.
#pragma once

#include "ctx.h"

namespace shci {

// Scale exponent s with B * 2^s < 2^61 (B > 0), from the bound's binary exponent.
__device__ __forceinline__ int fix_scale(double B) {
  if (!(B > 0.0)) return 0;
  const int e = static_cast<int>((__double_as_longlong(B) >> 52) & 0x7ff) - 1022;  // B < 2^e
  return 61 - e;
}

// The same from scal = {bound on the row abs sums, bits of max |x|}.
__device__ __forceinline__ int fix_scale_of(const double* __restrict__ scal) {
  return fix_scale(scal[0] * __longlong_as_double(static_cast<long long>(
                                 reinterpret_cast<const unsigned long long*>(scal)[1])));
}

}  // namespace shci
