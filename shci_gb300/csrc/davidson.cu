// Davidson eigensolver on the device (K5).
//
// Follows Davidson::diagonalize (src/solver/davidson.cc:8-196).  davidson(): n_states = 1, at
// most five stored vectors, a restart that collapses onto the current Ritz vector, the
// diagonal preconditioner with the 1e-8 cut, Gram-Schmidt, the <= 5x5 subspace eigenproblem
// (solved on the host in FP64 by cyclic Jacobi) with the Ritz vector's first component made
// non-negative, and convergence |lambda - lambda_prev| <= tol.  davidson_states(): the same
// for n_states > 1 (5 n_states stored vectors, one preconditioned vector per step for the
// states in turn, a subspace solve after the last state's vector, convergence state by state).
// All vector work is FP64 on the device; dot products reduce in a fixed order so results do
// not depend on timing.
#include <algorithm>
#include <cmath>
#include <numeric>

#include "ctx.h"
#include "kernels.h"
#include "spmv.cuh"

namespace shci {

namespace {

constexpr int kDotBlocks = 304;
constexpr int kDotThreads = 256;

// dst[k * stride] = sum of acc[k] over the block, k < m <= M: the sums' shuffles side by side, then a
// warp a sum.
template <int M>
__device__ __forceinline__ void block_sums(double (&acc)[M], int m, double* __restrict__ dst,
                                           int stride) {
  constexpr int kWarps = kDotThreads / 32;
  static_assert(M <= kWarps, "a warp a sum");
  __shared__ double s[M][kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1)
#pragma unroll
    for (int k = 0; k < M; k++)
      if (k < m) acc[k] += __shfl_xor_sync(kFull, acc[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < M; k++) s[k][warp] = acc[k];
  __syncthreads();
  if (warp < m) {
    double t = lane < kWarps ? s[warp][lane] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
    if (lane == 0) dst[warp * stride] = t;
  }
}

struct Ptrs6 {
  const double* p[6];
};

// Ends a reduction over the grid: every block leaves its m partial sums, and the block that arrives
// last adds them up in block order into out[0, m) (so the result does not depend on timing) and
// resets the counter.  A second launch for that sum cost as much as the sum itself.  Bound by the
// latency of its chains of shuffles and FP64 additions at the vector lengths of small systems: five
// dots of 14,000 elements 11 us, 15 with one sum after the other.
template <int M>
__device__ __forceinline__ void grid_sums(double (&acc)[M], int m, double* __restrict__ partial,
                                          unsigned* __restrict__ counter,
                                          double* __restrict__ out) {
  __shared__ bool last;
  block_sums(acc, m, partial + blockIdx.x, kDotBlocks);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) + 1u == gridDim.x;
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < M; k++) acc[k] = 0.0;
  for (int b = threadIdx.x; b < static_cast<int>(gridDim.x); b += blockDim.x)
#pragma unroll
    for (int k = 0; k < M; k++)
      if (k < m) acc[k] += __ldcg(partial + k * kDotBlocks + b);
  block_sums(acc, m, out, 1);
  if (threadIdx.x == 0) *counter = 0u;
}

// out[k] = <x, ys[k]> (ys[k] null: sum of x), k < m <= 6
__global__ void __launch_bounds__(kDotThreads)
    k_mdot(const double* __restrict__ x, Ptrs6 ys, int m, size_t n, double* __restrict__ partial,
           unsigned* __restrict__ counter, double* __restrict__ out) {
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double xi = x[i];
#pragma unroll
    for (int k = 0; k < 6; k++)
      if (k < m) acc[k] += ys.p[k] ? xi * ys.p[k][i] : xi;
  }
  grid_sums(acc, m, partial, counter, out);
}

// v -= (*coef) * u
__global__ void k_axpy_dev(double* __restrict__ v, const double* __restrict__ u,
                           const double* __restrict__ coef, size_t n) {
  const double a = *coef;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    v[i] -= a * u[i];
}

__global__ void k_normalize(double* __restrict__ v, const double* __restrict__ norm2, size_t n) {
  const double s = sqrt(*norm2);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    v[i] = v[i] / s;
}

__global__ void k_scale(double* __restrict__ v, double s, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    v[i] = v[i] / s;
}

// v = (Hw - lambda w) / (lambda - d), 0 where |lambda - d| < 1e-8  (davidson.cc:135-143)
__global__ void k_precond(double* __restrict__ v, const double* __restrict__ Hw,
                          const double* __restrict__ w, const double* __restrict__ diag,
                          double lambda, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double d = lambda - diag[i];
    v[i] = fabs(d) < 1.0e-8 ? 0.0 : (Hw[i] - lambda * w[i]) / d;
  }
}

// w = sum_k e_k v_k, Hw = sum_k e_k Hv_k  (davidson.cc:184-194)
struct Comb {
  const double* v[5];
  const double* hv[5];
  double e[5];
  int k;
};
__global__ void k_combine(double* __restrict__ w, double* __restrict__ hw, Comb cb, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    double a = 0.0, b = 0.0;
    for (int k = 0; k < cb.k; k++) {
      a += cb.v[k][i] * cb.e[k];
      b += cb.hv[k][i] * cb.e[k];
    }
    w[i] = a;
    hw[i] = b;
  }
}

// w = sum_k e_k v_k, Hw = sum_k e_k Hv_k over up to 5 * kMaxStates vectors
struct CombN {
  const double* v[5 * kMaxStates];
  const double* hv[5 * kMaxStates];
  double e[5 * kMaxStates];
  int k;
};
__global__ void k_combine_n(double* __restrict__ w, double* __restrict__ hw, CombN cb, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    double a = 0.0, b = 0.0;
    for (int k = 0; k < cb.k; k++) {
      a += cb.v[k][i] * cb.e[k];
      b += cb.hv[k][i] * cb.e[k];
    }
    w[i] = a;
    hw[i] = b;
  }
}

// One step of davidson() up to the product: the Ritz vector of the last subspace solve (cb.k > 0), the
// preconditioned residual (davidson.cc:135-143), Gram-Schmidt (:146-152) and the norm, each sum in
// the pass that forms its vector.  A step was 9 to 11 + 3 ic launches and two synchronisations around
// the product; now 4 + ic and one (n = 16 FP64 variation, 33 products: 9.7 -> 7.7 ms; n = 26 mixed, 48
// products: 27.8 -> 25.3 ms).
//
// w = sum_k e_k v_k, hw = sum_k e_k hv_k; v = (hw - lambda w) / (lambda - d), 0 where |lambda - d| <
// 1e-8; out[0] = <v, next> (next null: <v, v>).  *xmax (mixed products) is cleared.
__global__ void __launch_bounds__(kDotThreads)
    k_ritz_precond(double* __restrict__ w, double* __restrict__ hw, Comb cb,
                   double* __restrict__ v, const double* __restrict__ diag, double lambda,
                   const double* __restrict__ next, size_t n, double* __restrict__ partial,
                   unsigned* __restrict__ counter, double* __restrict__ out,
                   double* __restrict__ xmax) {
  if (xmax && blockIdx.x == 0 && threadIdx.x == 0) *xmax = 0.0;
  double acc[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    double a, b;
    if (cb.k) {
      a = b = 0.0;
      for (int k = 0; k < cb.k; k++) {
        a += cb.v[k][i] * cb.e[k];
        b += cb.hv[k][i] * cb.e[k];
      }
      w[i] = a;
      hw[i] = b;
    } else {
      a = w[i];
      b = hw[i];
    }
    const double d = lambda - diag[i];
    const double x = fabs(d) < 1.0e-8 ? 0.0 : (b - lambda * a) / d;
    v[i] = x;
    acc[0] += x * (next ? next[i] : x);
  }
  grid_sums(acc, 1, partial, counter, out);
}

// v -= (*coef) * u; out[0] = <v, next> (next null: <v, v>)
__global__ void __launch_bounds__(kDotThreads)
    k_axpy_dot(double* __restrict__ v, const double* __restrict__ u,
               const double* __restrict__ coef, const double* __restrict__ next, size_t n,
               double* __restrict__ partial, unsigned* __restrict__ counter,
               double* __restrict__ out) {
  const double a = *coef;
  double acc[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double x = v[i] - a * u[i];
    v[i] = x;
    acc[0] += x * (next ? next[i] : x);
  }
  grid_sums(acc, 1, partial, counter, out);
}

// The mixed product's end (spmv.cu, k_fix_out) and its dots: hv = yfix * 2^-s + diag * v, out[k] =
// <hv, ys[k]>.
__global__ void __launch_bounds__(kDotThreads)
    k_fix_rows(const unsigned long long* __restrict__ yfix, const double* __restrict__ scal,
               const double* __restrict__ diag, const double* __restrict__ v,
               double* __restrict__ hv, Ptrs6 ys, int m, size_t n, double* __restrict__ partial,
               unsigned* __restrict__ counter, double* __restrict__ out) {
  const double inv = ldexp(1.0, -fix_scale_of(scal));
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double x = static_cast<double>(static_cast<long long>(yfix[i])) * inv + diag[i] * v[i];
    hv[i] = x;
#pragma unroll
    for (int k = 0; k < 6; k++)
      if (k < m) acc[k] += x * ys.p[k][i];
  }
  grid_sums(acc, m, partial, counter, out);
}

class Dots {
 public:
  Dots(shci_ctx* c) : c_(c) {
    c->dav.partial.reserve(6 * kDotBlocks);
    c->dav.scal.reserve(kScal + 1);
    counter = reinterpret_cast<unsigned*>(c->dav.scal.p + kScal);
    SHCI_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned), c->stream));
  }
  static constexpr int kScal = 32;  // scalars, then the reductions' block counter
  unsigned* counter;
  // out_dev[k] = <x, ys[k]>, k < m (stays on the device)
  void mdot(const double* x, std::initializer_list<const double*> ys, size_t n, double* out_dev) {
    Ptrs6 p{};
    int m = 0;
    for (auto y : ys) p.p[m++] = y;
    mdot(x, p, m, n, out_dev);
  }
  void mdot(const double* x, const Ptrs6& p, int m, size_t n, double* out_dev) {
    k_mdot<<<grid(n), kDotThreads, 0, c_->stream>>>(x, p, m, n, c_->dav.partial.p, counter,
                                                    out_dev);
    SHCI_LAUNCH_CHECK();
    c_->launches += 1;
  }
  // (a fixed function of n: the order of a sum follows from the length alone)
  static unsigned grid(size_t n) { return grid_for(n, kDotThreads, kDotBlocks); }
  double dot_host(const double* a, const double* b, size_t n) {
    mdot(a, {b}, n, c_->dav.scal.p);
    double r = 0.0;
    SHCI_CUDA(cudaMemcpyAsync(&r, c_->dav.scal.p, 8, cudaMemcpyDeviceToHost, c_->stream));
    SHCI_CUDA(cudaStreamSynchronize(c_->stream));
    return r;
  }

 private:
  shci_ctx* c_;
};

}  // namespace

// Cyclic Jacobi on the lower triangle of a k x k matrix: eigenvalues ascending, eigenvectors
// in columns (evecs[r*k + c]).
void jacobi_eig(int k, const double* lower, int ld, double* evals, double* evecs) {
  std::vector<double> a(static_cast<size_t>(k) * k), v(static_cast<size_t>(k) * k);
  for (int i = 0; i < k; i++)
    for (int j = 0; j < k; j++) {
      a[i * k + j] = i >= j ? lower[i * ld + j] : lower[j * ld + i];
      v[i * k + j] = i == j ? 1.0 : 0.0;
    }
  for (int sweep = 0; sweep < 100; sweep++) {
    double off = 0.0, tot = 0.0;
    for (int i = 0; i < k * k; i++) tot += a[i] * a[i];
    for (int i = 0; i < k; i++)
      for (int j = 0; j < k; j++)
        if (i != j) off += a[i * k + j] * a[i * k + j];
    if (off == 0.0 || off <= 1e-30 * tot) break;
    for (int p = 0; p < k; p++)
      for (int q = p + 1; q < k; q++) {
        const double apq = a[p * k + q];
        if (apq == 0.0) continue;
        const double th = (a[q * k + q] - a[p * k + p]) / (2.0 * apq);
        const double t = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1.0));
        const double cs = 1.0 / std::sqrt(t * t + 1.0), sn = t * cs;
        for (int r = 0; r < k; r++) {
          const double x = a[r * k + p], y = a[r * k + q];
          a[r * k + p] = cs * x - sn * y;
          a[r * k + q] = sn * x + cs * y;
        }
        for (int r = 0; r < k; r++) {
          const double x = a[p * k + r], y = a[q * k + r];
          a[p * k + r] = cs * x - sn * y;
          a[q * k + r] = sn * x + cs * y;
        }
        for (int r = 0; r < k; r++) {
          const double x = v[r * k + p], y = v[r * k + q];
          v[r * k + p] = cs * x - sn * y;
          v[r * k + q] = sn * x + cs * y;
        }
      }
  }
  std::vector<int> idx(k);
  std::iota(idx.begin(), idx.end(), 0);
  std::sort(idx.begin(), idx.end(), [&](int x, int y) { return a[x * k + x] < a[y * k + y]; });
  for (int c = 0; c < k; c++) {
    evals[c] = a[idx[c] * k + idx[c]];
    for (int r = 0; r < k; r++) evecs[r * k + c] = v[r * k + idx[c]];
  }
}

__global__ void k_vec_differs(const double* __restrict__ a, const double* __restrict__ b, size_t n,
                              double* flag) {
  bool d = false;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    d |= __double_as_longlong(a[i]) != __double_as_longlong(b[i]);
  if (__any_sync(kFull, d) && (threadIdx.x & 31) == 0) *flag = 1.0;
}

DavidsonOut davidson(shci_ctx* c, double tol) {
  DavidsonOut out;
  auto& D = c->dav;
  D.ritz = false;
  const size_t n = c->H.n;
  cudaStream_t s = c->stream;
  const unsigned g = grid_for(n, 256, 152 * 16);
  Dots dots(c);
  if (n == 1) {
    SHCI_CUDA(cudaMemcpyAsync(&out.eval, c->H.diag.p, 8, cudaMemcpyDeviceToHost, s));
    const double one = 1.0;
    SHCI_CUDA(cudaMemcpyAsync(c->d_coef.p, &one, 8, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
    out.converged = true;
    return out;
  }
  const size_t store = std::min<size_t>(n, 5);
  for (size_t k = 0; k < store; k++) {
    D.v[k].mt = D.Hv[k].mt = &c->mem;
    D.v[k].resize(n, 1.1);
    D.Hv[k].resize(n, 1.1);
  }
  D.w.mt = D.Hw.mt = &c->mem;
  D.w.resize(n, 1.1);
  D.Hw.resize(n, 1.1);
  // v0 = init / |init|
  SHCI_CUDA(cudaMemcpyAsync(D.v[0].p, c->d_coef.p, n * 8, cudaMemcpyDeviceToDevice, s));
  dots.mdot(D.v[0].p, {D.v[0].p}, n, D.scal.p);
  k_normalize<<<g, 256, 0, s>>>(D.v[0].p, D.scal.p, n);
  SHCI_LAUNCH_CHECK();
  spmv(c, D.v[0].p, D.Hv[0].p, false);
  out.n_matvec++;
  double lambda = dots.dot_host(D.v[0].p, D.Hv[0].p, n);
  double hk[5 * 5] = {0};
  hk[0] = lambda;
  // the Ritz vector still to be formed from the stored vectors: at the next step, or at the end
  Comb cb{};
  cb.k = 1;
  cb.v[0] = D.v[0].p;
  cb.hv[0] = D.Hv[0].p;
  cb.e[0] = 1.0;
  auto form_ritz = [&]() {
    if (!cb.k) return;
    k_combine<<<g, 256, 0, s>>>(D.w.p, D.Hw.p, cb, n);
    SHCI_LAUNCH_CHECK();
    c->launches += 1;
    cb.k = 0;
  };
  out.trace.push_back(lambda);
  double lambda_prev = lambda;
  bool converged = false;
  double* scal = D.scal.p;       // [0, ic): <v, v_i>, [ic]: <v, v>
  double* row_dev = scal + 8;    // [0, ic]: <H v, v_i>
  const unsigned gd = Dots::grid(n);
  double* xmax = spmv_xmax(c);
  for (size_t it = 1; it < store * 2; it++) {
    const size_t ic = it % store;
    if (it >= store && ic == 0) {  // restart (davidson.cc:115-131)
      form_ritz();
      SHCI_CUDA(cudaMemcpyAsync(D.v[0].p, D.w.p, n * 8, cudaMemcpyDeviceToDevice, s));
      SHCI_CUDA(cudaMemcpyAsync(D.Hv[0].p, D.Hw.p, n * 8, cudaMemcpyDeviceToDevice, s));
      lambda = dots.dot_host(D.v[0].p, D.Hv[0].p, n);
      hk[0] = lambda;
      continue;
    }
    double* v = D.v[ic].p;
    k_ritz_precond<<<gd, kDotThreads, 0, s>>>(D.w.p, D.Hw.p, cb, v, c->H.diag.p, lambda,
                                              ic ? D.v[0].p : nullptr, n, D.partial.p,
                                              dots.counter, scal, xmax);
    SHCI_LAUNCH_CHECK();
    cb.k = 0;
    for (size_t i = 0; i < ic; i++) {  // Gram-Schmidt (davidson.cc:146-152)
      k_axpy_dot<<<gd, kDotThreads, 0, s>>>(v, D.v[i].p, scal + i,
                                            i + 1 < ic ? D.v[i + 1].p : nullptr, n, D.partial.p,
                                            dots.counter, scal + i + 1);
      SHCI_LAUNCH_CHECK();
    }
    spmv_normalized(c, v, scal + ic, D.Hv[ic].p);
    Ptrs6 p{};
    for (size_t i = 0; i <= ic; i++) p.p[i] = D.v[i].p;
    if (xmax) {
      k_fix_rows<<<gd, kDotThreads, 0, s>>>(c->H.yfix.p, c->H.scal.p, c->H.diag.p, v, D.Hv[ic].p,
                                            p, (int)ic + 1, n, D.partial.p, dots.counter, row_dev);
      SHCI_LAUNCH_CHECK();
    } else {
      dots.mdot(D.Hv[ic].p, p, (int)ic + 1, n, row_dev);
    }
    // the norm comes back with the row: a vector without one has cost a product that is dropped
    double back[16];
    SHCI_CUDA(cudaMemcpyAsync(back, scal, sizeof(back), cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
    if (std::sqrt(back[ic]) < 1e-12) {
      converged = true;
      break;
    }
    out.n_matvec++;
    for (size_t i = 0; i <= ic; i++) hk[ic * 5 + i] = back[8 + i];
    const int k = static_cast<int>(ic + 1);
    double ev[5], evec[25];
    jacobi_eig(k, hk, 5, ev, evec);
    lambda = ev[0];
    const double factor = evec[0] < 0 ? -1.0 : 1.0;
    cb.k = k;
    for (int i = 0; i < k; i++) {
      cb.v[i] = D.v[i].p;
      cb.hv[i] = D.Hv[i].p;
      cb.e[i] = evec[i * k] * factor;
    }
    c->launches += 2 + ic;
    out.trace.push_back(lambda);
    if (std::fabs(lambda - lambda_prev) <= tol) converged = true;
    if (!converged) lambda_prev = lambda;
    if (converged) break;
  }
  form_ritz();
  SHCI_CUDA(cudaMemcpyAsync(c->d_coef.p, D.w.p, n * 8, cudaMemcpyDeviceToDevice, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  D.ritz = true;
  D.ritz_h = c->H.build_id;
  out.eval = lambda;
  out.converged = converged;
  c->prof.flush();
  return out;
}

double* state_coef(shci_ctx* c, unsigned s) {
  return s == 0 ? c->d_coef.p : c->d_xcoef[s - 1].p;
}

// davidson.cc:8-196 for n_states = c->n_states > 1.  The subspace matrix starts with only its
// diagonal set (:62-77); the initial vectors are normalised and orthogonalised in order.
DavidsonStatesOut davidson_states(shci_ctx* c, double tol) {
  DavidsonStatesOut out;
  auto& D = c->dav;
  D.ritz = false;
  const size_t n = c->H.n;
  cudaStream_t s = c->stream;
  const unsigned g = grid_for(n, 256, 152 * 16);
  const unsigned req = c->n_states;
  const unsigned ns = static_cast<unsigned>(std::min<size_t>(n, req));
  out.evals.assign(req, 0.0);
  Dots dots(c);
  if (n == 1) {
    SHCI_CUDA(cudaMemcpyAsync(&out.evals[0], c->H.diag.p, 8, cudaMemcpyDeviceToHost, s));
    const double one = 1.0, zero = 0.0;
    SHCI_CUDA(cudaMemcpyAsync(c->d_coef.p, &one, 8, cudaMemcpyHostToDevice, s));
    for (unsigned k = 1; k < req; k++)
      SHCI_CUDA(cudaMemcpyAsync(state_coef(c, k), &zero, 8, cudaMemcpyHostToDevice, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
    out.converged = true;
    return out;
  }
  const size_t nis = std::min<size_t>(n, 5);
  const size_t m = ns * nis;
  for (size_t k = 0; k < m; k++) {
    D.sv[k].mt = D.sHv[k].mt = &c->mem;
    D.sv[k].resize(n, 1.1);
    D.sHv[k].resize(n, 1.1);
  }
  for (unsigned k = 0; k < ns; k++) {
    D.sw[k].mt = D.sHw[k].mt = &c->mem;
    D.sw[k].resize(n, 1.1);
    D.sHw[k].resize(n, 1.1);
  }
  double* scal = D.scal.p;
  auto host_dots = [&](const double* x, const std::vector<const double*>& ys, double* outv) {
    for (size_t b = 0; b < ys.size(); b += 6) {
      Ptrs6 p{};
      const int mm = static_cast<int>(std::min<size_t>(6, ys.size() - b));
      for (int q = 0; q < mm; q++) p.p[q] = ys[b + q];
      dots.mdot(x, p, mm, n, scal);
      SHCI_CUDA(cudaMemcpyAsync(outv + b, scal, mm * 8, cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaStreamSynchronize(s));
    }
  };
  // initial vectors (:44-60)
  for (unsigned k = 0; k < ns; k++) {
    SHCI_CUDA(cudaMemcpyAsync(D.sv[k].p, state_coef(c, k), n * 8, cudaMemcpyDeviceToDevice, s));
    double nrm = std::sqrt(dots.dot_host(D.sv[k].p, D.sv[k].p, n));
    k_scale<<<g, 256, 0, s>>>(D.sv[k].p, nrm, n);
    SHCI_LAUNCH_CHECK();
    if (k > 0) {
      for (unsigned q = 0; q < k; q++) {
        dots.mdot(D.sv[k].p, {D.sv[q].p}, n, scal);
        k_axpy_dev<<<g, 256, 0, s>>>(D.sv[k].p, D.sv[q].p, scal, n);
        SHCI_LAUNCH_CHECK();
      }
      nrm = std::sqrt(dots.dot_host(D.sv[k].p, D.sv[k].p, n));
      k_scale<<<g, 256, 0, s>>>(D.sv[k].p, nrm, n);
      SHCI_LAUNCH_CHECK();
    }
  }
  std::vector<double> hk(m * m, 0.0), lam(ns), lam_prev(ns);
  for (unsigned k = 0; k < ns; k++) {
    spmv(c, D.sv[k].p, D.sHv[k].p, false);
    out.n_matvec++;
    lam[k] = dots.dot_host(D.sv[k].p, D.sHv[k].p, n);
    hk[k * m + k] = lam[k];
    SHCI_CUDA(cudaMemcpyAsync(D.sw[k].p, D.sv[k].p, n * 8, cudaMemcpyDeviceToDevice, s));
    SHCI_CUDA(cudaMemcpyAsync(D.sHw[k].p, D.sHv[k].p, n * 8, cudaMemcpyDeviceToDevice, s));
  }
  lam_prev = lam;
  bool converged = false;
  size_t n_conv = 0, pre = 0;
  for (size_t it = ns; it < m * 2; it++) {
    const size_t ic = it % m;
    if (it >= m) {  // restart onto the Ritz vectors (:86-103)
      if (ic < ns - 1) continue;
      if (ic == ns - 1) {
        for (unsigned k = 0; k < ns; k++) {
          SHCI_CUDA(cudaMemcpyAsync(D.sv[k].p, D.sw[k].p, n * 8, cudaMemcpyDeviceToDevice, s));
          SHCI_CUDA(cudaMemcpyAsync(D.sHv[k].p, D.sHw[k].p, n * 8, cudaMemcpyDeviceToDevice, s));
        }
        for (unsigned k = 0; k < ns; k++) {
          lam[k] = dots.dot_host(D.sv[k].p, D.sHv[k].p, n);
          hk[k * m + k] = lam[k];
          for (unsigned q = k + 1; q < ns; q++) {
            const double e = dots.dot_host(D.sv[k].p, D.sHv[q].p, n);
            hk[k * m + q] = e;
            hk[q * m + k] = e;
          }
        }
        continue;
      }
    }
    // preconditioned residual of state `pre` (:133-143)
    k_precond<<<g, 256, 0, s>>>(D.sv[ic].p, D.sHw[pre].p, D.sw[pre].p, c->H.diag.p, lam[pre], n);
    SHCI_LAUNCH_CHECK();
    for (size_t i = 0; i < ic; i++) {  // (:145-152)
      dots.mdot(D.sv[ic].p, {D.sv[i].p}, n, scal);
      k_axpy_dev<<<g, 256, 0, s>>>(D.sv[ic].p, D.sv[i].p, scal, n);
      SHCI_LAUNCH_CHECK();
    }
    const double nrm = std::sqrt(dots.dot_host(D.sv[ic].p, D.sv[ic].p, n));
    if (nrm < 1e-12) {
      converged = true;
      break;
    }
    k_scale<<<g, 256, 0, s>>>(D.sv[ic].p, nrm, n);
    SHCI_LAUNCH_CHECK();
    spmv(c, D.sv[ic].p, D.sHv[ic].p, false);
    out.n_matvec++;
    {  // row ic of the subspace matrix (:163-167)
      std::vector<const double*> ys(ic + 1);
      for (size_t i = 0; i <= ic; i++) ys[i] = D.sv[i].p;
      std::vector<double> row(ic + 1);
      host_dots(D.sHv[ic].p, ys, row.data());
      for (size_t i = 0; i <= ic; i++) hk[ic * m + i] = row[i];
    }
    c->launches += 4 + 2 * ic;
    if (pre + 1 == ns) {  // subspace solve (:169-172) and Ritz vectors (:173-194)
      const int k = static_cast<int>(ic + 1);
      std::vector<double> ev(k), evec(static_cast<size_t>(k) * k);
      jacobi_eig(k, hk.data(), static_cast<int>(m), ev.data(), evec.data());
      for (unsigned st = 0; st < ns; st++) {
        lam[st] = ev[st];
        const double factor = evec[st] < 0 ? -1.0 : 1.0;
        CombN cb{};
        cb.k = k;
        for (int i = 0; i < k; i++) {
          cb.v[i] = D.sv[i].p;
          cb.hv[i] = D.sHv[i].p;
          cb.e[i] = evec[i * k + st] * factor;
        }
        k_combine_n<<<g, 256, 0, s>>>(D.sw[st].p, D.sHw[st].p, cb, n);
        SHCI_LAUNCH_CHECK();
        c->launches += 1;
      }
      for (unsigned st = static_cast<unsigned>(n_conv); st < ns; st++) {  // (:180-186)
        if (std::fabs(lam[st] - lam_prev[st]) > tol) break;
        n_conv++;
      }
      if (n_conv == ns) converged = true;
      if (!converged) lam_prev = lam;
      if (converged) break;
    }
    pre++;
    if (pre >= ns) pre = n_conv;
  }
  for (unsigned k = 0; k < ns; k++) {
    SHCI_CUDA(cudaMemcpyAsync(state_coef(c, k), D.sw[k].p, n * 8, cudaMemcpyDeviceToDevice, s));
    out.evals[k] = lam[k];
  }
  SHCI_CUDA(cudaStreamSynchronize(s));
  out.converged = converged;
  c->prof.flush();
  return out;
}

// Rayleigh quotient of d_coef with value + residual.  When d_coef is still the Ritz vector w
// of the last Davidson call on this (mixed) Hamiltonian, w^T H w = w^T Hw + w^T R w with Hw =
// H32 w kept by Davidson (FP32 values, FP64 diagonal), so only the residual store R is read
// (2 w^T R w over its upper triangle: one gather per element, no atomics);
// otherwise H w is formed from value + residual.
double rayleigh_fp64(shci_ctx* c) {
  const size_t n = c->H.n;
  auto& D = c->dav;
  cudaStream_t s = c->stream;
  Dots dots(c);
  if (n > 1 && D.ritz && D.ritz_h == c->H.build_id && c->H.precision != SHCI_PREC_FP64 &&
      D.w.n == n && c->d_coef.n >= n) {
    D.scal.reserve(Dots::kScal + 1);
    SHCI_CUDA(cudaMemsetAsync(D.scal.p, 0, 8, s));
    k_vec_differs<<<grid_for(n, 256, 152 * 8), 256, 0, s>>>(c->d_coef.p, D.w.p, n, D.scal.p);
    SHCI_LAUNCH_CHECK();
    double differs = 0.0;
    SHCI_CUDA(cudaMemcpyAsync(&differs, D.scal.p, 8, cudaMemcpyDeviceToHost, s));
    SHCI_CUDA(cudaStreamSynchronize(s));
    if (differs == 0.0) {
      D.rt.mt = &c->mem;
      const size_t len = residual_rows(c, D.w.p, D.rt);
      double r[3];  // w^T Hw, w^T w, w^T R w / 2
      dots.mdot(D.w.p, {D.Hw.p, D.w.p}, n, D.scal.p);
      dots.mdot(D.rt.p, {nullptr}, len, D.scal.p + 2);
      SHCI_CUDA(cudaMemcpyAsync(r, D.scal.p, sizeof(r), cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaStreamSynchronize(s));
      c->launches += 1;
      return (r[0] + 2.0 * r[2]) / r[1];
    }
  }
  return rayleigh_fp64_of(c, c->d_coef.p);
}

double rayleigh_fp64_of(shci_ctx* c, const double* x) {
  const size_t n = c->H.n;
  auto& D = c->dav;
  Dots dots(c);
  D.ritz = false;  // Hw is overwritten below
  D.Hw.mt = &c->mem;
  D.Hw.resize(n, 1.1);
  spmv(c, x, D.Hw.p, true);
  const double num = dots.dot_host(x, D.Hw.p, n);
  const double den = dots.dot_host(x, x, n);
  return num / den;
}

}  // namespace shci
