// One- and two-body reduced density matrices of the variational wavefunction (K8): the
// adjoint of the energy, dE_var/dh and dE_var/dg.
//
// Reference: RDM::get_1rdm (src/chem/rdm.cc:12-131), RDM::get_2rdm over the Hamiltonian
// connections (:333-371, 397-433), get_2rdm_elements (:435-642), permfac_ccaa (:243-269) and
// the half storage of write_in_2rdm / combine4_2rdm (:233-241, 644-657); time_sym = false.
//  1-RDM: a warp per det; its lanes take the single excitations p -> r of the same symmetry,
//         look the target det up in the hash set of the det list and accumulate c_i c_j sign into
//         a per-block n x n tile in shared memory; the diagonal (p = r) stays in registers.
//  2-RDM: a warp per work item (a piece of a row's stored connections, items.cuh) adds c_i c_j f
//         into the half-stored array (a = p n + s, b = q n + r, kept when a >= b) with FP64
//         atomics (the array is L2 resident for the sizes of interest); single excitations are
//         queued and finished 32 at a time; the diagonal has a kernel of its own.
#include <algorithm>

#include "ctx.h"
#include "heatbath.cuh"
#include "items.cuh"
#include "kernels.h"

namespace shci {

namespace {

constexpr int kRdmWarps = 8;

// A thread per det made every det a chain of n_e n binary searches (17 dependent loads each) with
// half of the chip's threads idle at 80,000 dets: 3.4 ms at n = 26, against 0.27 ms with a warp
// per det and one hash probe per excitation.
__global__ void __launch_bounds__(kRdmWarps * 32)
    k_rdm1(SelParams P, const double* __restrict__ coef, uint32_t n_dets,
           const unsigned* __restrict__ orb_sym, int n, bool dup, double* __restrict__ out) {
  extern __shared__ double tile[];
  __shared__ uint8_t occ[kRdmWarps][64], virt[kRdmWarps][64];
  __shared__ unsigned sym[64];
  const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = threadIdx.x; k < n * n; k += blockDim.x) tile[k] = 0.0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) sym[k] = orb_sym[k];
  __syncthreads();
  double dg0 = 0.0, dg1 = 0.0;  // diagonal elements lane and lane + 32
  const uint32_t warps = gridDim.x * kRdmWarps;
  for (uint32_t i = blockIdx.x * kRdmWarps + w; i < n_dets; i += warps) {
    const uint64_t u = P.up[i], d = P.dn[i];
    const double ci = coef[i];
    // (of equal dets the set holds the first: a det's own partner too)
    const double cc = ci * (dup ? coef[set_index(P, u, d)] : ci);
    for (int spin = 0; spin < 2; spin++) {
      const uint64_t h = spin ? d : u;
      __syncwarp();
      for (int o = lane; o < n; o += 32) {
        const int k = popc64(h & below(o));
        if (h >> o & 1) occ[w][k] = static_cast<uint8_t>(o);
        else virt[w][o - k] = static_cast<uint8_t>(o);
      }
      __syncwarp();
      if (h >> lane & 1) dg0 += cc;
      if (h >> (lane + 32) & 1) dg1 += cc;
      const uint32_t ne = static_cast<uint32_t>(popc64(h)), nv = static_cast<uint32_t>(n) - ne;
      for (uint32_t t = lane; t < ne * nv; t += 32) {
        const int p = occ[w][t / nv], r = virt[w][t % nv];
        if (sym[p] != sym[r]) continue;
        const uint64_t nh = h ^ (1ull << p) ^ (1ull << r);
        const long long j = set_index(P, spin ? u : nh, spin ? nh : d);
        if (j < 0) continue;
        atomicAdd(&tile[p * n + r], flip_sign(ci * coef[j], move_parity(h, p, r)));
      }
    }
  }
  if (dg0 != 0.0) atomicAdd(&tile[lane * (n + 1)], dg0);
  if (dg1 != 0.0) atomicAdd(&tile[(lane + 32) * (n + 1)], dg1);
  __syncthreads();
  for (int k = threadIdx.x; k < n * n; k += blockDim.x)
    if (tile[k] != 0.0) atomicAdd(&out[k], tile[k]);
}

// Half-stored element of pairs x = (p, s) and y = (q, r): the reference writes a term at (x, y)
// and its mirror at (y, x) and keeps the one with a >= b, both when they are equal
// (write_in_2rdm, rdm.cc:233-241).
__device__ __forceinline__ void rdm2_add(double* __restrict__ half, uint32_t x, uint32_t y,
                                         double v) {
  const uint64_t a = x > y ? x : y, b = x > y ? y : x;
  atomicAdd(&half[a * (a + 1) / 2 + b], x == y ? 2.0 * v : v);
}

// Terms of a pair of dets one move apart (get_2rdm_elements, rdm.cc:475-546, 560-590): electron
// b1 -> b2 of string `s` (the other string is `o`), v = c_i c_j times the move's sign.  A
// spectator in the same string passes the move's sign unchanged (permfac_ccaa).
__device__ __forceinline__ void rdm2_single(double* __restrict__ half, int n, uint64_t s,
                                            uint64_t o, int b1, int b2, double v) {
  const uint32_t fwd = b2 * n + b1, rev = b1 * n + b2;
  for (uint64_t m = s & ~(1ull << b1); m; m &= m - 1) {
    const int p = ctz64(m);
    const uint32_t pp = p * (n + 1);
    rdm2_add(half, pp, fwd, v);
    rdm2_add(half, pp, rev, v);
    rdm2_add(half, b2 * n + p, p * n + b1, -v);
    rdm2_add(half, b1 * n + p, p * n + b2, -v);
  }
  for (uint64_t m = o; m; m &= m - 1) {
    const uint32_t pp = ctz64(m) * (n + 1);
    rdm2_add(half, pp, fwd, v);
    rdm2_add(half, pp, rev, v);
  }
}

// Terms of a pair of dets two moves apart (rdm.cc:548-558, 592-640): two or four atomics.
__device__ __forceinline__ void rdm2_double(double* __restrict__ half, int n, uint64_t tu,
                                            uint64_t td, uint64_t cu, uint64_t cd, double cc) {
  const uint64_t xu = tu ^ cu, xd = td ^ cd;
  if (xu && xd) {
    const int a1 = ctz64(tu & xu), a2 = ctz64(cu & xu), b1 = ctz64(td & xd), b2 = ctz64(cd & xd);
    const double v = flip_sign(cc, move_parity(tu, a1, a2) + move_parity(td, b1, b2));
    rdm2_add(half, a2 * n + a1, b2 * n + b1, v);
    rdm2_add(half, a1 * n + a2, b1 * n + b2, v);
    return;
  }
  const uint64_t s = xu ? tu : td, c = xu ? cu : cd, x = xu ? xu : xd;
  const uint64_t from = s & x, to = c & x;
  const int b1 = ctz64(from), b2 = ctz64(from & (from - 1));
  const int b3 = ctz64(to), b4 = ctz64(to & (to - 1));
  const double v = flip_sign(cc, below_count(s, b1) + below_count(s, b2) + below_count(c, b3) +
                                     below_count(c, b4));
  rdm2_add(half, b3 * n + b1, b4 * n + b2, v);
  rdm2_add(half, b3 * n + b2, b4 * n + b1, -v);
  rdm2_add(half, b1 * n + b3, b2 * n + b4, v);
  rdm2_add(half, b1 * n + b4, b2 * n + b3, -v);
}

// Off-diagonal pairs.  A single excitation adds about 4 n_e terms and a double 2 or 4, so a warp
// that finished its lanes' elements in place would run the singles' loop for one or two lanes:
// singles wait in a per-warp queue and are finished 32 at a time.  5.6 -> 1.24 ms at n = 26, 80,000
// dets, 36M elements (a warp per row and the diagonal on one lane of it before); bound by the
// FP64 atomics' L1 and L2 traffic (about 60 % busy each).
__global__ void __launch_bounds__(kRdmWarps * 32)
    k_rdm2(const __grid_constant__ ItemTab T, const uint64_t* __restrict__ up,
           const uint64_t* __restrict__ dn, const double* __restrict__ coef, int n,
           double* __restrict__ half) {
  __shared__ uint2 qs[kRdmWarps][64];
  uint2* q = qs[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t qn = 0;  // waiting (warp-uniform), in q[0, qn)
  auto drain = [&](uint32_t m) {  // the last m entries
    __syncwarp();
    if (lane < m) {
      const uint2 e = q[qn - m + lane];
      const uint64_t tu = up[e.x], td = dn[e.x], cu = up[e.y], cd = dn[e.y];
      const uint64_t xu = tu ^ cu;
      const uint64_t s = xu ? tu : td, c = xu ? cu : cd, o = xu ? td : tu;
      const int b1 = ctz64(s & ~c), b2 = ctz64(c & ~s);
      rdm2_single(half, n, s, o, b1, b2,
                  flip_sign(coef[e.x] * coef[e.y], move_parity(s, b1, b2)));
    }
    __syncwarp();
    qn -= m;
  };
  for_items(T, [&](const ItemSeg& S, uint64_t, uint32_t i, uint64_t rs, uint32_t len) {
    const uint64_t tu = up[i], td = dn[i];
    const double ci = coef[i];
    for (uint32_t k0 = 0; k0 < len; k0 += 32) {
      const uint32_t k = k0 + lane;
      bool single = false;
      uint32_t j = 0;
      if (k < len) {
        j = S.col[rs + k];
        const uint64_t cu = up[j], cd = dn[j];
        const int x2 = popc64(tu ^ cu) + popc64(td ^ cd);
        single = x2 == 2;
        if (x2 == 4) rdm2_double(half, n, tu, td, cu, cd, ci * coef[j]);
      }
      const unsigned bal = __ballot_sync(kFull, single);
      if (bal) {
        if (single) q[qn + __popc(bal & lt)] = make_uint2(i, j);
        qn += __popc(bal);
        if (qn >= 32u) drain(32u);
      }
    }
  });
  if (qn) drain(qn);
}

// Diagonal pairs (rdm.cc:443-473): sum_i c_i^2 over the dets that hold orbitals s and r in the
// same string (s > r), and s in the alpha, r in the beta string.  A warp takes an orbital s at a
// time and its lanes the r; the dets of the block's range pass by as broadcast loads, and a det
// without s in a string costs no FP64 addition.  0.21 ms at n = 26, 80,000 dets (FP64 pipe).
__global__ void __launch_bounds__(kRdmWarps * 32)
    k_rdm2_diag(const uint64_t* __restrict__ up, const uint64_t* __restrict__ dn,
                const double* __restrict__ coef, uint32_t n_dets, uint32_t per_block, int n,
                double* __restrict__ half) {
  const int lane = threadIdx.x & 31;
  const uint32_t b = blockIdx.x * per_block, e = min(n_dets, b + per_block);
  for (int s = threadIdx.x >> 5; s < n; s += kRdmWarps) {
    double same[2] = {0.0, 0.0}, oppo[2] = {0.0, 0.0};
    for (uint32_t i = b; i < e; i++) {
      const uint64_t u = up[i], d = dn[i];
      const bool in_u = u >> s & 1, in_d = d >> s & 1;
      if (!in_u && !in_d) continue;
      const double c = coef[i], c2 = c * c;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int r = lane + 32 * k;
        if (k == 1 && n <= 32) break;
        if (in_u) {
          if (r < s && (u >> r & 1)) same[k] += c2;
          if (d >> r & 1) oppo[k] += c2;
        }
        if (in_d && r < s && (d >> r & 1)) same[k] += c2;
      }
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int r = lane + 32 * k;
      const uint32_t ss = s * (n + 1), rr = r * (n + 1);
      if (same[k] != 0.0) {
        rdm2_add(half, ss, rr, same[k]);
        rdm2_add(half, s * n + r, r * n + s, -same[k]);
      }
      if (oppo[k] != 0.0) rdm2_add(half, ss, rr, oppo[k]);
    }
  }
}

}  // namespace

void rdm1(shci_ctx* c, double* out) {
  const int n = c->I.n;
  DevBuf<double> res;
  res.mt = &c->mem;
  res.resize((size_t)n * n);
  rdm1_dev(c, res.p);
  SHCI_CUDA(cudaMemcpyAsync(out, res.p, (size_t)n * n * 8, cudaMemcpyDeviceToHost, c->stream));
  SHCI_CUDA(cudaStreamSynchronize(c->stream));
}

void rdm1_dev(shci_ctx* c, double* res_dev) {
  sync_dets(c);
  const uint32_t n_dets = static_cast<uint32_t>(c->up.size());
  const int n = c->I.n;
  cudaStream_t s = c->stream;
  const bool dup = rebuild_det_set(c, true);
  SelParams P{};
  P.up = c->d_up.p;
  P.dn = c->d_dn.p;
  P.set_hash = c->set_hash.p;
  P.set_hash_mask = c->set_hash_mask;
  DevBuf<unsigned> sym;
  sym.mt = &c->mem;
  sym.resize(n);
  SHCI_CUDA(cudaMemcpyAsync(sym.p, c->I.orb_sym.data(), n * sizeof(unsigned), cudaMemcpyHostToDevice, s));
  SHCI_CUDA(cudaMemsetAsync(res_dev, 0, (size_t)n * n * 8, s));
  int sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  {
    ProfScope ps(c->prof, s, "rdm1");
    k_rdm1<<<grid_for((size_t)n_dets * 32, kRdmWarps * 32, (unsigned)sms * 6u), kRdmWarps * 32,
             (size_t)n * n * sizeof(double), s>>>(P, c->d_coef.p, n_dets, sym.p, n, dup, res_dev);
    SHCI_LAUNCH_CHECK();
  }
  SHCI_CUDA(cudaStreamSynchronize(s));
  c->prof.flush();
  c->launches += 1;
}

void rdm2(shci_ctx* c, double* out_half) {
  const size_t nn = (size_t)c->I.n * c->I.n, size = nn * (nn + 1) / 2;
  DevBuf<double> half;
  half.mt = &c->mem;
  half.resize(size);
  rdm2_dev(c, half.p);
  SHCI_CUDA(cudaMemcpyAsync(out_half, half.p, size * 8, cudaMemcpyDeviceToHost, c->stream));
  SHCI_CUDA(cudaStreamSynchronize(c->stream));
}

void rdm2_dev(shci_ctx* c, double* half_dev) {
  auto& H = c->H;
  if (!H.valid || H.n != c->up.size()) throw ArgError("the 2-RDM needs the current Hamiltonian");
  sync_dets(c);
  const int n = c->I.n;
  const size_t nn = (size_t)n * n, size = nn * (nn + 1) / 2;
  cudaStream_t s = c->stream;
  SHCI_CUDA(cudaMemsetAsync(half_dev, 0, size * 8, s));
  int sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  const uint32_t n_dets = static_cast<uint32_t>(H.n);
  {
    ProfScope ps(c->prof, s, "rdm2");
    size_t items = 0;
    const ItemTab T = item_tab(H, &items);
    k_rdm2<<<grid_for(items * 32, kRdmWarps * 32, (unsigned)sms * 6u), kRdmWarps * 32, 0, s>>>(
        T, c->d_up.p, c->d_dn.p, c->d_coef.p, n, half_dev);
    SHCI_LAUNCH_CHECK();
    // at least 64 dets a block: each block ends with up to 3 n^2 atomics
    const uint32_t per = std::max<uint32_t>(64u, (n_dets + sms * 8 - 1) / (sms * 8));
    k_rdm2_diag<<<(n_dets + per - 1) / per, kRdmWarps * 32, 0, s>>>(
        c->d_up.p, c->d_dn.p, c->d_coef.p, n_dets, per, n, half_dev);
    SHCI_LAUNCH_CHECK();
  }
  SHCI_CUDA(cudaStreamSynchronize(s));
  c->prof.flush();
  c->launches += 2;
}

}  // namespace shci
