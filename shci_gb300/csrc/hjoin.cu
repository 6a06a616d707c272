// Hamiltonian build by a two-hole core join.
//
// Two determinants with the same electron counts are connected by at most a double
// excitation exactly when they share an (n_e - 2)-electron "core": the det with some pair of
// its electrons removed.  Every det contributes K = C(n_e, 2) entries, one per electron pair
// (alpha-alpha, beta-beta or alpha-beta), keyed by a hash of its core.  After a stable sort by
// key, each bucket of equal keys holds, in det-id order, dets that share a core (plus, rarely,
// dets whose different cores hash alike).  Row i then examines, for each of its K entries,
// only the members after its own entry in that bucket: exactly the dets j > i sharing that
// core.  This finds the same element set as the group scan of the reference's
// Hamiltonian<S>::update_matrix (src/solver/hamiltonian.h:415-598: same-alpha, same-beta and
// alpha-single x beta-single partners) while examining about 1.4 candidates per stored
// element instead of tens.
//
// A pair (i, j) shares one core if it is a double excitation and n_e - 1 cores if it is a
// single; it is taken only from its canonical core: the two electrons of i absent from j
// (double), or the electron of i absent from j plus the lowest electron the two share, alpha
// orbitals before beta ones (single).  The test uses the actual spin strings, so a hash
// collision can only add candidates that fail it; the one collision that could repeat a
// column (two cores of j in one bucket, adjacent by construction) is skipped explicitly.
//
// Used when n_e >= 2, n * K < 2^32 and the index fits in memory; otherwise the scan path
// (hbuild.cu) builds the matrix.
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "ctx.h"
#include "heatbath.cuh"
#include "hrow.cuh"
#include "kernels.h"

namespace shci {

namespace {

constexpr int kJoinWarps = 8, kJoinCtas = 5;
constexpr int kPlaceStretch = 1024;
constexpr const char* kBadCounts = "dets do not all have the electron counts of the first det";
constexpr uint32_t kMinPart = 256;
constexpr int kCloseThreads = 256, kClosePer = 4;
constexpr size_t kSplitEntries = 16u << 20;  // 128 MB of spans

__device__ __forceinline__ uint64_t core_hash(uint64_t cu, uint64_t cd) {
  uint64_t h = cu * 0x9E3779B97F4A7C15ull ^ (cd + 0x632BE59BD9B4E019ull) * 0xC2B2AE3D27D4EB4Full;
  h ^= h >> 29;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 32;
  return h;
}

// Removed-electron masks (alpha, beta) of pair entry k of det (u, d).
__device__ __forceinline__ void pair_masks(uint32_t pr, uint64_t u, uint64_t d, int n_up,
                                           uint64_t* ru, uint64_t* rd) {
  const int r1 = static_cast<int>(pr & 0xffffu), r2 = static_cast<int>(pr >> 16);
  uint64_t a = 0, b = 0;
  if (r1 < n_up) a |= 1ull << nth_bit(u, r1);
  else b |= 1ull << nth_bit(d, r1 - n_up);
  if (r2 < n_up) a |= 1ull << nth_bit(u, r2);
  else b |= 1ull << nth_bit(d, r2 - n_up);
  *ru = a;
  *rd = b;
}

// The electrons of one det over a warp's lanes: lane e holds the orbital of electron e (alpha
// electrons first), so that a pair's masks are two shuffles.  More than 32 electrons: every lane
// looks its pair up in the strings.  Core keys of 1.2 million dets of 20 electrons: 0.70 ms; 1.7
// with two bit searches a pair.
struct LaneElecs {
  uint64_t u, d;
  int n_up;
  bool wide;
  int orb;  // of electron `lane`; beta orbitals + 64
  __device__ __forceinline__ LaneElecs(uint64_t u_, uint64_t d_, int n_up_, int ne)
      : u(u_), d(d_), n_up(n_up_), wide(ne > 32), orb(0) {
    const int e = threadIdx.x & 31;
    if (!wide && e < ne) orb = e < n_up ? nth_bit(u, e) : nth_bit(d, e - n_up) + 64;
  }
  // Masks of pair pr (all lanes call; lanes without a pair pass any valid one).
  __device__ __forceinline__ void masks(uint32_t pr, uint64_t* ru, uint64_t* rd) const {
    if (wide) {
      pair_masks(pr, u, d, n_up, ru, rd);
      return;
    }
    const int a = __shfl_sync(kFull, orb, pr & 0xffffu), b = __shfl_sync(kFull, orb, pr >> 16);
    const uint64_t x = 1ull << (a & 63), y = 1ull << (b & 63);
    *ru = (a < 64 ? x : 0ull) | (b < 64 ? y : 0ull);
    *rd = (a < 64 ? 0ull : x) | (b < 64 ? 0ull : y);
  }
};

__global__ void k_pack_dets(const uint64_t* __restrict__ up, const uint64_t* __restrict__ dn,
                            uint32_t n, ulonglong2* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = make_ulonglong2(up[i], dn[i]);
}

// Entries in det order: key = top `bits` bits of the core hash, value = entry index.
template <class KT>
__global__ void k_core_keys(const uint64_t* __restrict__ up, const uint64_t* __restrict__ dn,
                            uint32_t n, const uint32_t* __restrict__ pairs, uint32_t K, int n_up,
                            int n_dn, int bits, KT* keys, uint32_t* vals, unsigned* err) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = warp0; i < n; i += n_warps) {
    const uint64_t u = up[i], d = dn[i];
    if ((popc64(u) != n_up || popc64(d) != n_dn) && lane == 0) atomicOr(err, (unsigned)kDevCheck);
    const LaneElecs el(u, d, n_up, n_up + n_dn);
    for (uint32_t k0 = 0; k0 < K; k0 += 32) {
      const uint32_t k = k0 + lane;
      uint64_t ru, rd;
      el.masks(pairs[min(k, K - 1u)], &ru, &rd);
      if (k >= K) continue;
      const size_t t = (size_t)i * K + k;
      keys[t] = static_cast<KT>(core_hash(u & ~ru, d & ~rd) >> (64 - bits));
      vals[t] = static_cast<uint32_t>(t);
    }
  }
}

// First position >= q whose key differs from `key` (m if none); all lanes of the warp call with the
// same arguments, keys[q .. ] ascending from `key`.  Probes 32 positions apart 1, 32, 1,024, ...
// until one differs, then narrows by 32 a round.
template <class KT>
__device__ __forceinline__ uint32_t warp_run_end(const KT* __restrict__ keys, KT key, uint32_t q,
                                                 uint32_t m) {
  const unsigned lane = threadIdx.x & 31;
  uint64_t step = 1, lo = q;  // positions q .. lo - 1 hold `key`
  bool narrow = false;
  while (true) {
    const uint64_t t = lo + (uint64_t)lane * step + (step - 1);  // the last of the lane's stretch
    const unsigned past = __ballot_sync(kFull, t >= m || keys[t] != key);
    const int full = past ? __ffs(past) - 1 : 32;  // stretches that hold only `key`
    lo += full * step;
    if (full < 32) {
      narrow = true;
      if (step == 1) return static_cast<uint32_t>(lo);
      step >>= 5;
    } else if (!narrow) {
      step <<= 5;
    }
  }
}

// After the sort every position p of a bucket of equal keys makes a span p | end << 32 and the det
// id of its entry.  A warp per 32 positions: a bucket that ends among them ends at the next lane
// whose successor differs; only the one that runs on is searched for.  ENTRY: the span goes to its
// entry's place, else to position p, and the det ids are left for k_place_spans.
// To entries, this is bound by the scattered 8-byte writes: 228 million entries 9.3 ms, and 11.4
// with flags of the bucket starts, their scan and an array of starts (five launches and a wait
// more: 0.05 against 0.25 ms over the six builds of an n = 16 variation).
template <class KT, bool ENTRY>
__global__ void k_bucket_spans(const KT* __restrict__ keys, const uint32_t* ents, uint32_t m,
                               uint32_t K, uint64_t* span, uint32_t* jdet) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t n_tiles = m / 32u + (m % 32u != 0u);
  for (uint32_t tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile < n_tiles;
       tile += (gridDim.x * blockDim.x) >> 5) {
    const uint64_t p = (uint64_t)tile * 32u + lane;
    const KT key = p < m ? keys[p] : KT(0);
    const bool last = p + 1 >= m || keys[p + 1] != key;
    const unsigned lasts = __ballot_sync(kFull, last);
    uint32_t end = 0;
    if (!(lasts >> 31)) end = warp_run_end(keys, __shfl_sync(kFull, key, 31), (tile + 1) * 32u, m);
    const unsigned mine = lasts >> lane;
    if (mine) end = static_cast<uint32_t>(p) + __ffs(mine);
    if (p < m) {
      const uint32_t v = ents[p];
      span[ENTRY ? v : p] = p | (static_cast<uint64_t>(end) << 32);
      if (ENTRY) jdet[p] = v / K;
    }
  }
}

// out[ents[p]] = span[p], the entries split by their leading bits: the writes of a while fall in a
// window that L2 holds, so that a sector goes to memory once and whole.  A block per stretch of
// positions, in order (a grid that strides over the array writes to every window at once: 8.6 ms
// against 1.7 at 228 million entries).  Beside that, the entries of all positions in jdet become det ids.
__global__ void __launch_bounds__(256)
    k_place_spans(const uint32_t* __restrict__ ents, const uint64_t* __restrict__ span, uint32_t m,
                  uint32_t K, uint64_t* __restrict__ out, uint32_t* __restrict__ jdet) {
  const uint64_t p0 = (uint64_t)blockIdx.x * kPlaceStretch + threadIdx.x;
  uint32_t e[kPlaceStretch / 256];
  uint64_t v[kPlaceStretch / 256];
  uint32_t j[kPlaceStretch / 256];
#pragma unroll
  for (int k = 0; k < kPlaceStretch / 256; k++) {
    const uint64_t p = p0 + k * 256;
    e[k] = p < m ? ents[p] : 0u;
    v[k] = p < m ? span[p] : 0u;
    j[k] = p < m ? jdet[p] : 0u;
  }
#pragma unroll
  for (int k = 0; k < kPlaceStretch / 256; k++)
    if (p0 + k * 256 < m) {
      out[e[k]] = v[k];
      jdet[p0 + k * 256] = j[k] / K;
    }
}

}  // namespace

namespace {

struct JoinView {
  uint32_t K;
  int n_up, n_elecs;
  const ulonglong2* dets;  // (up, dn): one 16-byte read a candidate
  const uint32_t* pairs;
  const uint64_t* span;
  const uint32_t* jdet;
  uint32_t n_prev;  // incremental update: rows < n_prev take only members >= n_prev
  uint32_t part;  // parts of long rows
  const uint32_t* lists;
  const uint2* units;
  uint32_t* unit_cnt;
};

// Members of entry sp = (position p | bucket end << 32) of row i: positions (p', end) with
// p' = p, or, for a row built before (i < n_prev), the last position whose det precedes
// n_prev (a bucket lists its dets in increasing id order, so the members >= n_prev follow).
__device__ __forceinline__ uint32_t member_start(const uint32_t* __restrict__ jdet, uint64_t sp,
                                                 uint32_t i, uint32_t n_prev) {
  uint32_t p = static_cast<uint32_t>(sp);
  if (i < n_prev) {
    uint32_t lo = p + 1u, hi = static_cast<uint32_t>(sp >> 32);
    if (jdet[hi - 1u] < n_prev) return hi - 1u;  // (most buckets have no new member)
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (jdet[mid] < n_prev) lo = mid + 1u;
      else hi = mid;
    }
    p = lo - 1u;
  }
  return p;
}

// Rows of more than two parts of `part` candidates, cut into parts (in the order of the traversal)
// that different warps take: units[slot + k] = (row, part k), lists[0] units and lists[1] rows in
// all, rows[.] = (row, slot).  A part fills its own stretch of the row's storage, which holds one
// place per candidate; k_close_rows closes the gaps.
__global__ void k_long_rows(const uint64_t* __restrict__ row_ptr, uint32_t n, uint32_t part,
                            uint32_t* lists, uint2* __restrict__ units, uint2* __restrict__ rows) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t cand = static_cast<uint32_t>(row_ptr[i + 1] - row_ptr[i]);
    if (cand <= 2u * part) continue;
    const uint32_t parts = (cand - 1u) / part + 1u;
    const uint32_t slot = atomicAdd(&lists[0], parts);
    rows[atomicAdd(&lists[1], 1u)] = make_uint2(i, slot);
    for (uint32_t k = 0; k < parts; k++) units[slot + k] = make_uint2(i, k);
  }
}

// A CTA per long row moves its parts together, a stretch (held in registers between two barriers)
// after the other, and writes the row's length.
template <int MODE>
__global__ void __launch_bounds__(kCloseThreads)
    k_close_rows(const uint64_t* __restrict__ row_ptr, uint32_t part,
                 const uint32_t* __restrict__ lists, const uint2* __restrict__ rows,
                 const uint32_t* __restrict__ unit_cnt, uint32_t* row_cnt, uint32_t* col,
                 double* v64, float* v32, float* r32) {
  __shared__ uint32_t s_cnt[kCloseThreads];
  const uint32_t n_rows = lists[1];
  for (uint32_t r = blockIdx.x; r < n_rows; r += gridDim.x) {
    const uint32_t i = rows[r].x, slot = rows[r].y;
    const uint64_t base = row_ptr[i];
    const uint32_t cand = static_cast<uint32_t>(row_ptr[i + 1] - base);
    const uint32_t parts = (cand - 1u) / part + 1u;
    uint32_t len = 0;
    for (uint32_t k = 0; k < parts; k++) {
      if (k % kCloseThreads == 0) {
        __syncthreads();
        if (k + threadIdx.x < parts) s_cnt[threadIdx.x] = unit_cnt[slot + k + threadIdx.x];
        __syncthreads();
      }
      const uint32_t c = s_cnt[k % kCloseThreads];
      const uint64_t src = base + (uint64_t)k * part, dst = base + len;
      len += c;
      if (src == dst) continue;
      for (uint32_t t0 = 0; t0 < c; t0 += kCloseThreads * kClosePer) {
        uint32_t j[kClosePer];
        double a[kClosePer];
        float b[kClosePer], e[kClosePer];
#pragma unroll
        for (int x = 0; x < kClosePer; x++) {
          const uint32_t t = t0 + threadIdx.x + x * kCloseThreads;
          if (t >= c) continue;
          j[x] = col[src + t];
          if (MODE == 1) a[x] = v64[src + t];
          if (MODE == 2) {
            b[x] = v32[src + t];
            e[x] = r32[src + t];
          }
        }
        __syncthreads();  // (what the stores below write over has been read)
#pragma unroll
        for (int x = 0; x < kClosePer; x++) {
          const uint32_t t = t0 + threadIdx.x + x * kCloseThreads;
          if (t >= c) continue;
          col[dst + t] = j[x];
          if (MODE == 1) v64[dst + t] = a[x];
          if (MODE == 2) {
            v32[dst + t] = b[x];
            r32[dst + t] = e[x];
          }
        }
      }
    }
    if (threadIdx.x == 0) row_cnt[i] = len;
  }
}

// Row kernel of the join (MODE as in RowSink).  A warp per row or, PARTS, part of a long row
// (these first): lanes take the row's entries 32 at a time, the members after each entry are flattened over the
// lanes, and every member that passes the canonical-core test goes to the row's queues.
// Bound by the integer pipe (population counts, compares and shuffles per candidate).  1.2 million
// dets of n = 40 (1.86 G candidates, 1.25 G elements): 25.6 ms; 27.6 with every pair's masks by
// bit searches in the strings and a candidate's two strings from two arrays.  Five CTAs per SM
// (48 registers): 25.6 ms, four (64 registers): 27.1, six (40 registers): 25.8.
template <int MODE, bool PARTS>
__global__ void __launch_bounds__(kJoinWarps * 32, kJoinCtas)
    k_hjoin(DevIntegrals I, uint32_t n, JoinView jv, uint32_t* row_cnt, const uint64_t* row_ptr,
            uint32_t* col, double* v64, float* v32, float* r32, unsigned* work, float* absacc) {
  __shared__ RowQueues qs[kJoinWarps];
  RowQueues& q = qs[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31;
  const uint32_t K = jv.K;
  const uint32_t n_units = PARTS ? jv.lists[0] : 0u;
  while (true) {
    uint32_t w = 0;
    if (lane == 0) w = atomicAdd(work, 1u);
    w = __shfl_sync(kFull, w, 0);
    uint32_t i = w - n_units, t_lo = 0, t_hi = 0xffffffffu;  // the row's candidates [t_lo, t_hi)
    uint64_t base = 0;
    if (PARTS && w < n_units) {
      const uint2 x = jv.units[w];
      i = x.x;
      t_lo = x.y * jv.part;
      t_hi = t_lo + jv.part;
      base = row_ptr[i] + t_lo;
    } else {
      if (i >= n) break;
      if (MODE) {
        base = row_ptr[i];
        const uint64_t places = row_ptr[i + 1] - base;
        if (PARTS && places > 2u * jv.part) continue;
        if (places == 0) {  // most older rows of an incremental update
          if (row_cnt && lane == 0) row_cnt[i] = 0;
          continue;
        }
      }
    }
    const ulonglong2 det_i = __ldg(jv.dets + i);
    const uint64_t ui = det_i.x, di = det_i.y;
    const LaneElecs el(ui, di, jv.n_up, jv.n_elecs);
    RowSink<MODE> sink(q, I, ui, di, base, col, v64, v32, r32);
    if (absacc) sink.track_abs(absacc, i);
    uint32_t n_cand = 0;  // up to the current entries
    for (uint32_t k0 = 0; k0 < K && (!PARTS || n_cand < t_hi); k0 += 32) {
      const uint32_t k = k0 + lane;
      uint32_t p = 0, len = 0;
      if (k < K) {
        const uint64_t sp = jv.span[(size_t)i * K + k];
        p = member_start(jv.jdet, sp, i, jv.n_prev);
        len = static_cast<uint32_t>(sp >> 32) - p - 1u;
      }
      const uint32_t inc = warp_inclusive_u32(len);
      const uint32_t total = __shfl_sync(kFull, inc, 31);
      if (total == 0) continue;
      uint64_t ru, rd;
      el.masks(jv.pairs[min(k, K - 1u)], &ru, &rd);
      const uint32_t first = PARTS && t_lo > n_cand ? t_lo - n_cand : 0u;
      const uint32_t end = PARTS ? min(total, t_hi - n_cand) : total;
      n_cand += total;
      for (uint32_t t0 = first; t0 < end; t0 += 32) {
        const uint32_t t = t0 + lane;
        const uint32_t o = owner_lane(inc, t);
        const uint32_t o_inc = __shfl_sync(kFull, inc, o);
        const uint32_t o_len = __shfl_sync(kFull, len, o);
        const uint32_t o_p = __shfl_sync(kFull, p, o);
        const uint64_t o_ru = __shfl_sync(kFull, ru, o);
        const uint64_t o_rd = __shfl_sync(kFull, rd, o);
        bool cand = false, single = false;
        uint32_t j = 0;
        uint64_t uj = 0, dj = 0;
        if (t < end) {
          const uint32_t pos = o_p + 1u + (t - (o_inc - o_len));
          j = jv.jdet[pos];
          // a second entry of j in this bucket (its two cores hashed alike) sits right after
          // the first; take j once
          const bool repeat = pos > o_p + 1u && jv.jdet[pos - 1u] == j;
          if (!repeat) {
            const ulonglong2 det_j = __ldg(jv.dets + j);
            uj = det_j.x;
            dj = det_j.y;
            const uint64_t xu = ui ^ uj, xd = di ^ dj;
            const int x2 = popc64(xu) + popc64(xd);
            const uint64_t iu = ui & xu, id = di & xd;  // electrons of i absent from j
            if (x2 == 4) {
              cand = o_ru == iu && o_rd == id;
            } else if (x2 == 2) {
              const uint64_t cu = ui & uj, cd = di & dj;
              const uint64_t lu = cu & (~cu + 1ull);
              const uint64_t ld = cu ? 0ull : (cd & (~cd + 1ull));
              cand = o_ru == (iu | lu) && o_rd == (id | ld);
              single = true;
            }
          }
        }
        sink.push(cand, single, j, uj, dj);
      }
    }
    const uint32_t cnt = sink.finish();
    if (lane == 0) {
      if (PARTS && w < n_units) jv.unit_cnt[w] = cnt;
      else if (row_cnt) row_cnt[i] = cnt;
      atomicAdd(reinterpret_cast<unsigned long long*>(work + 2),
                (unsigned long long)(PARTS ? min(n_cand, t_hi) - t_lo : n_cand));
    }
  }
}

// Row capacity of a single-pass build: the candidates of row i (members after each of its
// entries), an upper bound on the elements it keeps.
__global__ void k_join_caps(const uint64_t* __restrict__ span, const uint32_t* __restrict__ jdet,
                            uint32_t n, uint32_t K, uint32_t n_prev, uint64_t* caps,
                            uint32_t* longest) {
  const unsigned lane = threadIdx.x & 31;
  uint32_t most = 0;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    uint64_t c = 0;
    for (uint32_t k = lane; k < K; k += 32) {
      const uint64_t sp = span[(size_t)i * K + k];
      c += static_cast<uint32_t>(sp >> 32) - member_start(jdet, sp, i, n_prev) - 1u;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
    if (lane == 0) caps[i] = c;
    most = max(most, static_cast<uint32_t>(c));
  }
  if (lane == 0 && most > __ldcg(longest)) atomicMax(longest, most);  // (rarely after the first)
}

void release_sort_pingpong(shci_ctx* c) {
  c->sort.kalt.release();
  c->sort.kalt32.release();
  c->sort.valt32.release();
  c->sort.valt64.release();
}

// The sorts' storage goes back before the stored elements are allocated: their digit counts too, which
// for m entries are more than the packed dets.
void release_sort_scratch(shci_ctx* c) {
  release_sort_pingpong(c);
  c->sort.hist.release();
  c->sort.part32.release();
}

void sort_keys(DevBuf<uint32_t>& k, DevBuf<uint32_t>& v, size_t m, int bits, shci_ctx* c) {
  radix_sort_pairs32(k, v, m, 0, bits, c->stream, c->sort, false);
}
void sort_keys(DevBuf<uint64_t>& k, DevBuf<uint32_t>& v, size_t m, int bits, shci_ctx* c) {
  radix_sort_pairs(k, v, m, 0, bits, c->stream, c->sort, false);
}

// Room to sort entries and spans by their entries: the keys' storage, once the buckets are known,
// and 8 or 4 bytes an entry more.
void split_room(shci_ctx* c, const DevBuf<uint32_t>&, size_t m) { c->sort.valt64.resize(m); }
void split_room(shci_ctx* c, const DevBuf<uint64_t>&, size_t m) { c->sort.kalt32.resize(m); }
void split_take(shci_ctx* c, DevBuf<uint32_t>& keys) { swap_storage(keys, c->sort.kalt32); }
void split_take(shci_ctx* c, DevBuf<uint64_t>& keys) { swap_storage(keys, c->sort.valt64); }

// SHCI_JOIN_SPLIT: 0 places spans straight and 1 by their entries' leading bits, at any size; 2 is 1
// with its storage refused.
int split_env() {
  const char* e = std::getenv("SHCI_JOIN_SPLIT");
  return e ? std::atoi(e) : -1;
}

// Entries -> sorted buckets -> spans; keys of type KT hold `bits` hash bits.
template <class KT>
void join_index(shci_ctx* c, DevBuf<KT>& keys, int bits, size_t n, int n_up, int n_dn,
                bool split) {
  auto& J = c->join;
  cudaStream_t s = c->stream;
  const size_t m = J.m;
  keys.resize(m);
  J.jdet.resize(m);
  {
    ProfScope ps(c->prof, s, "join_keys");
    k_core_keys<KT><<<grid_for(n * 32, 256), 256, 0, s>>>(
        c->d_up.p, c->d_dn.p, static_cast<uint32_t>(n), J.pairs.p, J.K, n_up, n_dn, bits,
        keys.p, J.jdet.p, J.lists.p + 3);
    SHCI_LAUNCH_CHECK();
  }
  {
    ProfScope ps(c->prof, s, "join_sort");
    sort_keys(keys, J.jdet, m, bits, c);
  }
  // the sort's ping-pong storage is not needed again for this build
  release_sort_pingpong(c);
  J.span.resize(m);
  {
    ProfScope ps(c->prof, s, "join_buckets");
    const uint32_t m32 = static_cast<uint32_t>(m);
    if (split) {
      try {
        if (split_env() == 2) throw OomError("refused");
        split_room(c, keys, m);
      } catch (const OomError&) {  // straight needs no more storage
        split = false;
      }
    }
    if (!split) {
      k_bucket_spans<KT, true><<<grid_for(m, 256), 256, 0, s>>>(keys.p, J.jdet.p, m32, J.K,
                                                                J.span.p, J.jdet.p);
      SHCI_LAUNCH_CHECK();
    } else {
      // Entries and spans and a sorted copy of both, 24 bytes an entry with the keys': the sort is one
      // digit long, so that the unsorted entries stay for the det ids and the unsorted spans' storage
      // takes the placed ones.
      k_bucket_spans<KT, false><<<grid_for(m, 256), 256, 0, s>>>(keys.p, J.jdet.p, m32, J.K,
                                                                 J.span.p, nullptr);
      SHCI_LAUNCH_CHECK();
      split_take(c, keys);
      int top = 0;  // bits of an entry index
      while (top < 32 && (m32 - 1u) >> top) top++;
      radix_sort_pairs32_64(J.jdet, J.span, m, std::max(0, top - 8), top, s, c->sort, false);
      k_place_spans<<<static_cast<unsigned>((m + kPlaceStretch - 1) / kPlaceStretch), 256, 0, s>>>(
          J.jdet.p, J.span.p, m32, J.K, c->sort.valt64.p, c->sort.kalt32.p);
      SHCI_LAUNCH_CHECK();
      swap_storage(J.jdet, c->sort.kalt32);
      swap_storage(J.span, c->sort.valt64);
      J.jdet.n = J.span.n = m;
      c->launches += 6;
    }
  }
  release_sort_scratch(c);
  keys.release();
  J.key_bytes = sizeof(KT);
  J.bits = bits;
  c->launches += 7;
}

}  // namespace

bool join_prepare(shci_ctx* c) {
  auto& J = c->join;
  const size_t n = c->up.size();
  cudaStream_t s = c->stream;
  if (n == 0) return false;
  const int n_up = __builtin_popcountll(c->up[0]), n_dn = __builtin_popcountll(c->dn[0]);
  const int ne = n_up + n_dn;
  if (ne < 2 || ne > 128) return false;
  const uint64_t K = static_cast<uint64_t>(ne) * (ne - 1) / 2;
  const uint64_t m = n * K;
  if (m >= 0xffffffffull) return false;
  // memory of an entry: key and id with their sorted copies and a quarter to spare (18 B, 27 with
  // 64-bit keys), then id, span and, placed by leading bits, their sorted copies (24 B)
  size_t free_b = 0, total_b = 0;
  SHCI_CUDA(cudaMemGetInfo(&free_b, &total_b));
  size_t avail = free_b + c->mem.cached;  // cached blocks return to the driver on demand
  const size_t live = c->mem.live();
  if (c->mem.budget) avail = std::min(avail, c->mem.budget > live ? c->mem.budget - live : 0);
  if (static_cast<double>(m) * 26.0 > 0.85 * static_cast<double>(avail)) return false;
  J.K = static_cast<uint32_t>(K);
  J.n_up = n_up;
  J.n_elecs = ne;
  J.m = m;
  try {
    J.lists.resize(6);
    SHCI_CUDA(cudaMemsetAsync(J.lists.p, 0, 6 * sizeof(uint32_t), s));
    J.dets.resize(n);
    k_pack_dets<<<grid_for(n, 256), 256, 0, s>>>(c->d_up.p, c->d_dn.p, static_cast<uint32_t>(n),
                                                 J.dets.p);
    SHCI_LAUNCH_CHECK();
    std::vector<uint32_t> pr;
    pr.reserve(K);
    for (int r1 = 0; r1 < ne; r1++)
      for (int r2 = r1 + 1; r2 < ne; r2++) pr.push_back(static_cast<uint32_t>(r1 | (r2 << 16)));
    J.pairs.resize(K);
    SHCI_CUDA(cudaMemcpyAsync(J.pairs.p, pr.data(), K * 4, cudaMemcpyHostToDevice, s));
    // hash bits: 32 while the entries are few enough that merged buckets stay rare.
    // SHCI_JOIN_BITS (4..40) narrows it, so tests can force colliding buckets.
    int bits = m <= (1ull << 30) ? 32 : 40;
    if (const char* e = std::getenv("SHCI_JOIN_BITS")) bits = std::min(40, std::max(4, std::atoi(e)));
    // Spans by way of their entries' leading bits where they outgrow L2.  Straight against by
    // leading bits: 9.5 million entries 0.14 against 0.21 ms, 17 million 0.43 against 0.35, 76
    // million 2.9 against 1.4, 228 million 9.3 against 4.0.  (A single entry goes straight.)
    const int env = split_env();
    const bool split = env < 0 ? m > kSplitEntries : env != 0 && m > 1;
    if (bits <= 32) join_index(c, J.keys32, bits, n, n_up, n_dn, split);
    else join_index(c, J.keys, bits, n, n_up, n_dn, split);
  } catch (const OomError&) {
    join_release(c);
    release_sort_scratch(c);
    return false;
  }
  return true;
}

namespace {

template <bool PARTS>
void launch_hjoin(shci_ctx* c, int mode, uint32_t n, const JoinView& v, uint32_t* row_cnt,
                  const uint64_t* row_ptr, uint32_t* col, double* v64, float* v32, float* r32,
                  unsigned* work, unsigned grid, float* absacc) {
  cudaStream_t s = c->stream;
  if (mode == 1)
    k_hjoin<1, PARTS><<<grid, kJoinWarps * 32, 0, s>>>(c->dI, n, v, row_cnt, row_ptr, col, v64,
                                                        nullptr, nullptr, work, absacc);
  else
    k_hjoin<2, PARTS><<<grid, kJoinWarps * 32, 0, s>>>(c->dI, n, v, row_cnt, row_ptr, col, nullptr,
                                                        v32, r32, work, absacc);
  SHCI_LAUNCH_CHECK();
  c->launches += 1;
}

}  // namespace

void join_rows(shci_ctx* c, int mode, uint32_t* row_cnt, const uint64_t* row_ptr,
               uint32_t* col, double* v64, float* v32, float* r32, unsigned* work,
               unsigned grid, float* absacc, uint32_t n_prev, const JoinCaps& caps) {
  auto& J = c->join;
  const uint32_t n = static_cast<uint32_t>(c->up.size());
  if (!J.dets.p || !J.span.p || J.dets.n != n) throw std::logic_error("join rows without an index");
  cudaStream_t s = c->stream;
  JoinView v{J.K,      J.n_up, J.n_elecs, J.dets.p, J.pairs.p, J.span.p,
             J.jdet.p, n_prev, 0,         nullptr,  nullptr,   nullptr};
  if (mode == 0) {
    k_hjoin<0, false><<<grid, kJoinWarps * 32, 0, s>>>(c->dI, n, v, row_cnt, nullptr, nullptr,
                                                        nullptr, nullptr, nullptr, work, absacc);
    SHCI_LAUNCH_CHECK();
    c->launches += 1;
    return;
  }
  // A warp takes about 75 ns a candidate however few others there are, so rows go to one warp each
  // only while the longest is no longer than half a resident warp's share of all candidates, else
  // in parts of a quarter of that share.  30,000 dets of n = 40 (24 million candidates): 0.43 ms in
  // parts, 1.69 by rows; 120,000 (134 million): 1.96 and 4.95, most of it the longest row's warp
  // alone; 1.2 million (1.86 G): 26.1 in parts of 8,192, 25.5 by rows.  SHCI_JOIN_PART sets the
  // candidates of a part (0: whole rows).
  int dev_sms = 0;
  SHCI_CUDA(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, c->device));
  const uint64_t share = caps.total / (static_cast<uint64_t>(dev_sms) * kJoinWarps * kJoinCtas);
  if (2 * caps.longest > share)
    v.part = static_cast<uint32_t>(std::max<uint64_t>(kMinPart, std::min<uint64_t>(share / 4, 1u << 30)));
  if (const char* e = std::getenv("SHCI_JOIN_PART"))
    v.part = caps.longest ? static_cast<uint32_t>(std::max(0, std::atoi(e))) : 0u;
  // (a long row has more than two parts of the candidates, and at most one part that is not full)
  if (v.part && caps.longest > 2ull * v.part) {
    const size_t long_max = std::min<size_t>(n, caps.total / (2ull * v.part));
    try {
      J.long_rows.resize(long_max);
      J.units.resize(caps.total / v.part + long_max);
      J.unit_cnt.resize(J.units.n);
      v.lists = J.lists.p;
      v.units = J.units.p;
      v.unit_cnt = J.unit_cnt.p;
    } catch (const OomError&) {  // no room for the lists: whole rows
    }
  }
  if (!v.lists) {
    launch_hjoin<false>(c, mode, n, v, row_cnt, row_ptr, col, v64, v32, r32, work, grid, absacc);
    return;
  }
  SHCI_CUDA(cudaMemsetAsync(J.lists.p, 0, 2 * sizeof(uint32_t), s));
  k_long_rows<<<grid_for(n, 256), 256, 0, s>>>(row_ptr, n, v.part, J.lists.p, J.units.p,
                                               J.long_rows.p);
  SHCI_LAUNCH_CHECK();
  launch_hjoin<true>(c, mode, n, v, row_cnt, row_ptr, col, v64, v32, r32, work, grid, absacc);
  if (mode == 1)
    k_close_rows<1><<<grid, kCloseThreads, 0, s>>>(row_ptr, v.part, J.lists.p, J.long_rows.p,
                                                   J.unit_cnt.p, row_cnt, col, v64, nullptr,
                                                   nullptr);
  else
    k_close_rows<2><<<grid, kCloseThreads, 0, s>>>(row_ptr, v.part, J.lists.p, J.long_rows.p,
                                                   J.unit_cnt.p, row_cnt, col, nullptr, v32, r32);
  SHCI_LAUNCH_CHECK();
  c->launches += 2;
}

JoinCaps join_row_caps(shci_ctx* c, uint64_t* row_start, uint32_t n_prev) {
  auto& J = c->join;
  const uint32_t n = static_cast<uint32_t>(c->up.size());
  cudaStream_t s = c->stream;
  k_join_caps<<<grid_for((size_t)n * 32, 256), 256, 0, s>>>(J.span.p, J.jdet.p, n, J.K, n_prev,
                                                           row_start, J.lists.p + 2);
  SHCI_LAUNCH_CHECK();
  uint64_t* total = reinterpret_cast<uint64_t*>(J.lists.p + 4);
  exclusive_scan_u64_async(row_start, row_start, n, s, c->sort, total);
  SHCI_CUDA(cudaMemcpyAsync(row_start + n, total, 8, cudaMemcpyDeviceToDevice, s));
  uint32_t h[4];  // one wait: most candidates of a row, error, total
  SHCI_CUDA(cudaMemcpyAsync(h, J.lists.p + 2, sizeof(h), cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  c->launches += 1;
  if (h[1]) throw ArgError(kBadCounts);
  return {h[2] | static_cast<uint64_t>(h[3]) << 32, h[0]};
}

void join_check(shci_ctx* c) {
  uint32_t err = 0;
  SHCI_CUDA(cudaMemcpyAsync(&err, c->join.lists.p + 3, 4, cudaMemcpyDeviceToHost, c->stream));
  SHCI_CUDA(cudaStreamSynchronize(c->stream));
  if (err) throw ArgError(kBadCounts);
}

void join_release(shci_ctx* c) {
  auto& J = c->join;
  J.keys.release();
  J.keys32.release();
  J.jdet.release();
  J.span.release();
  J.dets.release();
  J.lists.release();
  J.units.release();
  J.long_rows.release();
  J.unit_cnt.release();
  J.m = 0;
}

}  // namespace shci
