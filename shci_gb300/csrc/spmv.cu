// Symmetric sparse H*v over the upper-triangle store (K4).
//
// Replaces SparseMatrix::mul (src/solver/sparse_matrix.cc:28-56): y = H x with H stored as
// its strict upper triangle plus an FP64 diagonal.  A warp takes a piece of a row i at a time
// (items.cuh) and streams its (col, val) pairs once: the row part y_i += H_ij x_j is reduced in registers and the
// transpose part y_j += H_ij x_i goes out as atomics (y is L2 resident).
//
// FP64 storage: FP64 products and FP64 atomics (the exact path).
//
// Mixed storage (FP32 value, optional FP32 residual): GB300 runs FP64 at 1/64 of the FP32
// rate, and one FP64 multiply-add per stored element already made this kernel FP64-bound, so
// the mixed kernel uses no FP64 per element:
//   * x is split into float pairs x = xh + xl (relative error 2^-48);
//   * products v * (xh + xl) are formed as float pairs with an exact FMA error term, so each
//     is accurate to about 2^-47 relative (far below the FP32 rounding of the stored value);
//   * the row part is accumulated as a float pair; each transpose contribution, and each
//     row's total, is converted to a 64-bit fixed-point integer with round-to-nearest and
//     added with an integer atomic.  The fixed-point scale 2^s is chosen per call from the
//     bound B = max_i sum_j |H_ij| * max_i |x_i| >= max_i |y_i| >= any single term, so that
//     B * 2^s < 2^61: every converted term and every final y_i fits, and integer additions
//     (modulo 2^64) are exact and order-independent.  The result does not depend on the
//     order of the atomics, so mixed H*v is bit-reproducible.  The absolute resolution of
//     y is 2^-s ~ B * 2^-61.
// The row abs-sum bound is computed once per matrix (float atomics; inflated by 5% against
// their rounding).
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "ctx.h"
#include "items.cuh"
#include "kernels.h"
#include "spmv.cuh"

namespace shci {

namespace {

__global__ void k_item_counts(const uint32_t* __restrict__ row_cnt, uint32_t n, uint32_t* cnt) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    cnt[i] = (row_cnt[i] + kItemLen - 1) / kItemLen;
}

__global__ void k_item_fill(const uint64_t* __restrict__ row_ptr,
                            const uint32_t* __restrict__ row_cnt,
                            const uint32_t* __restrict__ off, uint32_t n, uint4* it) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t len = row_cnt[i];
    uint32_t k = off[i];
    for (uint32_t b = 0; b < len; b += kItemLen) {
      const uint64_t st = row_ptr[i] + b;
      it[k++] = make_uint4(i, min(len - b, kItemLen), static_cast<uint32_t>(st),
                           static_cast<uint32_t>(st >> 32));
    }
  }
}

// y = diag * x
__global__ void k_diag_mul(const double* __restrict__ diag, const double* __restrict__ x,
                           double* __restrict__ y, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = diag[i] * x[i];
}

// FP64 store: FP64 products, FP64 atomics (y holds diag * x).
__global__ void __launch_bounds__(256)
    k_spmv(const __grid_constant__ ItemTab T, const double* __restrict__ x,
           double* __restrict__ y) {
  const unsigned lane = threadIdx.x & 31;
  for_items(T, [&](const ItemSeg& S, uint64_t, uint32_t i, uint64_t rs, uint32_t len) {
    const double xi = x[i];
    double acc = 0.0;
    const uint32_t* __restrict__ col = S.col + rs;
    const double* __restrict__ v64 = S.v64 + rs;
    for (uint32_t k = lane; k < len; k += 32) {
      const uint32_t j = col[k];
      const double v = v64[k];
      acc += v * x[j];
      atomicAdd(&y[j], v * xi);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (lane == 0) atomicAdd(&y[i], acc);
  });
}

// ---------------------------------------------------------------- mixed: fixed point
// f * 2^s rounded to the nearest integer (ties away from zero), for |f| * 2^s < 2^63.
// Subnormal floats (< 1.2e-38) count as zero.
__device__ __forceinline__ long long f2fix(float f, int s) {
  const unsigned b = __float_as_uint(f);
  const int ex = static_cast<int>((b >> 23) & 0xffu);
  const unsigned m = ex ? ((b & 0x7fffffu) | 0x800000u) : 0u;  // value = m * 2^(ex - 150)
  const int sh = ex - 150 + s;
  const int rs = min(max(-sh, 1), 30);
  const long long left = static_cast<long long>(m) << max(sh, 0);
  const long long right = static_cast<long long>((m + (1u << (rs - 1))) >> rs);
  const long long r = sh >= 0 ? left : right;
  return (b >> 31) ? -r : r;
}

// Exact float-pair sum (a + b = s + e): Knuth's two-sum.
__device__ __forceinline__ void two_sum(float a, float b, float* s, float* e) {
  const float t = a + b;
  const float z = t - a;
  *e = (a - (t - z)) + (b - z);
  *s = t;
}

// v * (xh + xl) (+ r * xh) as a float pair p + e.
template <bool RES>
__device__ __forceinline__ void prod2(float v, float r, float xh, float xl, float* p, float* e) {
  const float q = v * xh;
  float t = fmaf(v, xh, -q);
  t = fmaf(v, xl, t);
  if (RES) t = fmaf(r, xh, t);
  *p = q;
  *e = t;
}

// x -> float pairs; max |x| (as ordered bits of a non-negative double) into *xmax_bits; the
// fixed-point accumulators (when given) cleared.  norm2 (when given): x is divided by its root first,
// in place.
template <bool NORM>
__global__ void k_split_x(const double* __restrict__ x, uint32_t n, float2* xs,
                          unsigned long long* xmax_bits, unsigned long long* yfix,
                          const double* __restrict__ norm2, double* __restrict__ x_out) {
  unsigned long long mx = 0;
  const double nrm = NORM ? sqrt(*norm2) : 1.0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = NORM ? x_out[i] / nrm : x[i];
    if (NORM) x_out[i] = v;
    const float h = static_cast<float>(v);
    const float l = static_cast<float>(v - static_cast<double>(h));
    xs[i] = make_float2(h, l);
    if (yfix) yfix[i] = 0ull;
    const unsigned long long a = static_cast<unsigned long long>(__double_as_longlong(fabs(v)));
    mx = a > mx ? a : mx;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(kFull, mx, o);
    mx = t > mx ? t : mx;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(xmax_bits, mx);
}

// v /= sqrt(*norm2), y = diag * v
__global__ void k_normalize_diag(double* __restrict__ v, const double* __restrict__ norm2,
                                 const double* __restrict__ diag, double* __restrict__ y,
                                 uint32_t n) {
  const double s = sqrt(*norm2);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = v[i] / s;
    v[i] = x;
    y[i] = diag[i] * x;
  }
}

// Off-diagonal row abs sums of the full symmetric matrix, in float.
template <bool RES>
__global__ void __launch_bounds__(256)
    k_rowabs(const uint64_t* __restrict__ row_ptr, const uint32_t* __restrict__ row_len,
             const uint32_t* __restrict__ col,
             const float* __restrict__ v32, const float* __restrict__ r32,
             const double* __restrict__ diag, float* rowabs, uint32_t n) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const uint64_t rs = row_ptr[i], re = rs + row_len[i];
    float acc = 0.0f;
    for (uint64_t k = rs + lane; k < re; k += 32) {
      const float a = fabsf(v32[k]) + (RES ? fabsf(r32[k]) : 0.0f);
      acc += a;
      atomicAdd(&rowabs[col[k]], a);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (lane == 0) atomicAdd(&rowabs[i], acc);
  }
}

// max_i (rowabs_i + |diag_i|), as the bits of a non-negative float.
__global__ void k_max_bound(const float* __restrict__ a, const double* __restrict__ diag,
                            uint32_t n, unsigned* max_bits) {
  unsigned mx = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    mx = max(mx, __float_as_uint(a[i] + __double2float_ru(fabs(diag[i]))));
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
  if ((threadIdx.x & 31) == 0) atomicMax(max_bits, mx);
}

// Float sums of positive terms are within n_terms * 2^-24 relative; 5% covers that.
__global__ void k_scale_bound(double* scal) {
  const float fm = __uint_as_float(*reinterpret_cast<const unsigned*>(scal + 2));
  scal[0] = 1.05 * static_cast<double>(fm) + 1e-300;
}

// Mixed H*v: float-pair products, fixed-point accumulation (off-diagonal part only).
template <bool RES>
__global__ void __launch_bounds__(256)
    k_spmv_fix(const __grid_constant__ ItemTab T, const float2* __restrict__ xs,
               const double* __restrict__ scal, unsigned long long* __restrict__ yfix) {
  const int s = fix_scale_of(scal);
  const unsigned lane = threadIdx.x & 31;
  for_items(T, [&](const ItemSeg& S, uint64_t, uint32_t i, uint64_t rs, uint32_t len) {
    const float2 xi = xs[i];
    float ah = 0.0f, al = 0.0f;
    const uint32_t* __restrict__ col = S.col + rs;
    const float* __restrict__ v32 = S.v32 + rs;
    const float* __restrict__ r32 = RES ? S.r32 + rs : nullptr;
    for (uint32_t k = lane; k < len; k += 32) {
      const uint32_t j = col[k];
      const float v = v32[k];
      const float r = RES ? r32[k] : 0.0f;
      const float2 xj = xs[j];
      float p, e, t, te;
      prod2<RES>(v, r, xj.x, xj.y, &p, &e);
      two_sum(ah, p, &t, &te);
      ah = t;
      al += te + e;
      prod2<RES>(v, r, xi.x, xi.y, &p, &e);
      atomicAdd(&yfix[j], static_cast<unsigned long long>(f2fix(p, s) + f2fix(e, s)));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float bh = __shfl_xor_sync(kFull, ah, o), bl = __shfl_xor_sync(kFull, al, o);
      float t, te;
      two_sum(ah, bh, &t, &te);
      ah = t;
      al = al + bl + te;
    }
    if (lane == 0)
      atomicAdd(&yfix[i], static_cast<unsigned long long>(f2fix(ah, s) + f2fix(al, s)));
  });
}

// y = yfix * 2^-s + diag * x
__global__ void k_fix_out(const unsigned long long* __restrict__ yfix,
                          const double* __restrict__ diag, const double* __restrict__ x,
                          const double* __restrict__ scal, double* __restrict__ y, uint32_t n) {
  const int s = fix_scale_of(scal);
  const double inv = ldexp(1.0, -s);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = static_cast<double>(static_cast<long long>(yfix[i])) * inv + diag[i] * x[i];
}

}  // namespace

// H.scal[0] = bound on max_i sum_j |H_ij| from the off-diagonal sums in H.rowabs and the
// diagonal; H.rowabs stays (an incremental update adds to it).
void finish_mixed_bound(shci_ctx* c) {
  auto& H = c->H;
  cudaStream_t s = c->stream;
  const uint32_t n = static_cast<uint32_t>(H.n);
  H.scal.resize(4);
  SHCI_CUDA(cudaMemsetAsync(H.scal.p, 0, 4 * 8, s));
  unsigned* mb = reinterpret_cast<unsigned*>(H.scal.p + 2);
  k_max_bound<<<grid_for(n, 256), 256, 0, s>>>(H.rowabs.p, H.diag.p, n, mb);
  SHCI_LAUNCH_CHECK();
  k_scale_bound<<<1, 1, 0, s>>>(H.scal.p);
  SHCI_LAUNCH_CHECK();
  H.bound_valid = true;
  c->launches += 2;
}

namespace {

// Row abs-sum bound of a mixed store that was not built with one (a pass over the store).
void mixed_bound(shci_ctx* c, unsigned grid) {
  auto& H = c->H;
  cudaStream_t s = c->stream;
  const uint32_t n = static_cast<uint32_t>(H.n);
  H.rowabs.resize(n, 1.1);
  H.rowabs_hb = false;
  SHCI_CUDA(cudaMemsetAsync(H.rowabs.p, 0, (size_t)n * 4, s));
  for (const SegView& g : segments(H)) {
    k_rowabs<true><<<grid, 256, 0, s>>>(g.row_ptr, g.row_cnt, g.col, g.val32, g.res32, H.diag.p,
                                        H.rowabs.p, static_cast<uint32_t>(g.n));
    SHCI_LAUNCH_CHECK();
    c->launches += 1;
  }
  finish_mixed_bound(c);
}

// out[item] = w_i * sum over the item's elements of residual_ij * w_j (no atomics: the FP64
// energy correction needs only w^T R w = 2 sum_i w_i sum_j R_ij w_j of the residual store R).  w
// comes split into float pairs and the products and sums are float pairs, as in the mixed H*v
// (about 2^-44 relative): the FP64 form spent two FP64 operations per element (conversion and
// FMA), more than the gathers cost on GB300.
__global__ void __launch_bounds__(256)
    k_res_rows(const __grid_constant__ ItemTab T, const float2* __restrict__ ws,
               const double* __restrict__ w, double* __restrict__ out) {
  const unsigned lane = threadIdx.x & 31;
  for_items(T, [&](const ItemSeg& S, uint64_t at, uint32_t i, uint64_t rs, uint32_t len) {
    float ah = 0.0f, al = 0.0f;
    const uint32_t* __restrict__ col = S.col + rs;
    const float* __restrict__ r32 = S.r32 + rs;
    for (uint32_t k = lane; k < len; k += 32) {
      const float2 wj = ws[col[k]];
      float p, e, s2, se;
      prod2<false>(r32[k], 0.0f, wj.x, wj.y, &p, &e);
      two_sum(ah, p, &s2, &se);
      ah = s2;
      al += se + e;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float bh = __shfl_xor_sync(kFull, ah, o), bl = __shfl_xor_sync(kFull, al, o);
      float s2, se;
      two_sum(ah, bh, &s2, &se);
      ah = s2;
      al = al + bl + se;
    }
    if (lane == 0) out[at] = w[i] * (static_cast<double>(ah) + static_cast<double>(al));
  });
}

// Grid of the item kernels: eight CTAs of eight warps per SM, fewer when the matrix is small.
unsigned item_grid(shci_ctx* c, size_t items) {
  int sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  return grid_for(items * 32, 256, (unsigned)sms * 8u);
}

}  // namespace

void build_items(shci_ctx* c) {
  auto& H = c->H;
  auto& R = H.items;
  cudaStream_t s = c->stream;
  const uint32_t n = static_cast<uint32_t>(H.n);
  R.ok = false;
  if (n == 0) return;
  R.cap = H.nnz_current / kItemLen + n;  // sum of ceil(len / kItemLen) over n rows
  if (R.cap >= 0xffffffffull) return;
  // SHCI_ROW_ITEMS=0: whole rows, as without room for the list.
  const char* env = std::getenv("SHCI_ROW_ITEMS");
  if (env && std::strcmp(env, "0") == 0) return;
  try {
    R.off.resize((size_t)n + 1, 1.1);
    R.it.resize(R.cap, 1.1);
    k_item_counts<<<grid_for(n, 256), 256, 0, s>>>(H.row_cnt.p, n, R.off.p);
    SHCI_LAUNCH_CHECK();
    exclusive_scan_u32_async(R.off.p, R.off.p, n, s, c->sort, R.off.p + n);
  } catch (const OomError&) {  // no room: the kernels take whole rows
    R.off.release();
    R.it.release();
    return;
  }
  k_item_fill<<<grid_for(n, 256), 256, 0, s>>>(H.row_ptr.p, H.row_cnt.p, R.off.p, n, R.it.p);
  SHCI_LAUNCH_CHECK();
  R.ok = true;
  c->launches += 4;
}

size_t residual_rows(shci_ctx* c, const double* w, DevBuf<double>& out) {
  auto& H = c->H;
  if (!H.valid || H.precision == SHCI_PREC_FP64) throw ArgError("no mixed Hamiltonian built");
  const uint32_t n = static_cast<uint32_t>(H.n);
  cudaStream_t s = c->stream;
  size_t len = 0;
  const ItemTab T = item_tab(H, &len);
  out.resize(len, 1.1);
  ProfScope ps(c->prof, s, "spmv_res_rows");
  H.xs.resize(2 * (size_t)n, 1.1);
  float2* ws = reinterpret_cast<float2*>(H.xs.p);
  SHCI_CUDA(cudaMemsetAsync(H.scal.p + 1, 0, 8, s));
  k_split_x<false><<<grid_for(n, 256), 256, 0, s>>>(
      w, n, ws, reinterpret_cast<unsigned long long*>(H.scal.p + 1), nullptr, nullptr, nullptr);
  SHCI_LAUNCH_CHECK();
  SHCI_CUDA(cudaMemsetAsync(out.p, 0, len * 8, s));
  k_res_rows<<<item_grid(c, len), 256, 0, s>>>(T, ws, w, out.p);
  SHCI_LAUNCH_CHECK();
  c->launches += 2;
  return len;
}

void spmv(shci_ctx* c, const double* x, double* y, bool residual) {
  auto& H = c->H;
  if (!H.valid) throw ArgError("no Hamiltonian built");
  cudaStream_t s = c->stream;
  const uint32_t n = static_cast<uint32_t>(H.n);
  size_t len = 0;
  const ItemTab T = item_tab(H, &len);
  const unsigned grid = item_grid(c, len);
  if (H.precision == SHCI_PREC_FP64) {
    ProfScope ps(c->prof, s, "spmv");
    k_diag_mul<<<grid_for(n, 256), 256, 0, s>>>(H.diag.p, x, y, n);
    SHCI_LAUNCH_CHECK();
    k_spmv<<<grid, 256, 0, s>>>(T, x, y);
    SHCI_LAUNCH_CHECK();
    c->launches += 2;
    return;
  }
  if (!H.bound_valid) mixed_bound(c, grid);
  H.xs.resize(2 * (size_t)n, 1.1);
  H.yfix.resize(n, 1.1);
  ProfScope ps(c->prof, s, "spmv");
  SHCI_CUDA(cudaMemsetAsync(H.scal.p + 1, 0, 8, s));
  float2* xs = reinterpret_cast<float2*>(H.xs.p);
  k_split_x<false><<<grid_for(n, 256), 256, 0, s>>>(
      x, n, xs, reinterpret_cast<unsigned long long*>(H.scal.p + 1), H.yfix.p, nullptr, nullptr);
  SHCI_LAUNCH_CHECK();
  if (residual) k_spmv_fix<true><<<grid, 256, 0, s>>>(T, xs, H.scal.p, H.yfix.p);
  else k_spmv_fix<false><<<grid, 256, 0, s>>>(T, xs, H.scal.p, H.yfix.p);
  SHCI_LAUNCH_CHECK();
  k_fix_out<<<grid_for(n, 256), 256, 0, s>>>(H.yfix.p, H.diag.p, x, H.scal.p, y, n);
  SHCI_LAUNCH_CHECK();
  c->launches += 3;
}

double* spmv_xmax(shci_ctx* c) {
  auto& H = c->H;
  if (H.precision == SHCI_PREC_FP64) return nullptr;
  if (!H.bound_valid) mixed_bound(c, item_grid(c, H.n));
  return H.scal.p + 1;
}

void spmv_normalized(shci_ctx* c, double* v, const double* norm2, double* y) {
  auto& H = c->H;
  cudaStream_t s = c->stream;
  const uint32_t n = static_cast<uint32_t>(H.n);
  size_t len = 0;
  const ItemTab T = item_tab(H, &len);
  const unsigned grid = item_grid(c, len);
  ProfScope ps(c->prof, s, "spmv");
  if (H.precision == SHCI_PREC_FP64) {
    k_normalize_diag<<<grid_for(n, 256), 256, 0, s>>>(v, norm2, H.diag.p, y, n);
    SHCI_LAUNCH_CHECK();
    k_spmv<<<grid, 256, 0, s>>>(T, v, y);
  } else {
    H.xs.resize(2 * (size_t)n, 1.1);
    H.yfix.resize(n, 1.1);
    float2* xs = reinterpret_cast<float2*>(H.xs.p);
    k_split_x<true><<<grid_for(n, 256), 256, 0, s>>>(
        nullptr, n, xs, reinterpret_cast<unsigned long long*>(H.scal.p + 1), H.yfix.p, norm2, v);
    SHCI_LAUNCH_CHECK();
    k_spmv_fix<false><<<grid, 256, 0, s>>>(T, xs, H.scal.p, H.yfix.p);
  }
  SHCI_LAUNCH_CHECK();
  c->launches += 2;
}

}  // namespace shci
