// Walking the heat-bath windows of determinants (PT2 emission and selection).
//
// ChemSystem::find_connected_dets (src/chem/chem_system.cc:289-402) walks, for each electron and each
// electron pair of a determinant (a slot), the entries of one queue from eps_max down to eps_min.
// The windows of all determinants are cut into pieces of kPieceMin to kPieceLen entries; a warp takes
// a piece at a time.
#pragma once

#include "ctx.h"
#include "heatbath.cuh"

namespace shci {

// Entries a warp walks at most before the next piece: the heaviest determinant's window holds
// 100,000 entries, 3,000 rounds of one warp, and a piece costs the search of its source's slots again.
// Longer pieces where there are many entries: the PT2 emissions of an n = 40 run (297M entries and
// more a stage) 24.3 ms with at most 4,096, 21.7 with 8,192, 20.8 with 16,384, 22.1 with 32,768 (30.3
// with 2,048).  Shorter ones where warps would have none: the selections of an n = 16 variation took
// 0.43 ms in pieces of 4,096 and take 0.20, those of an n = 26 variation 0.84 and 0.41.
constexpr uint32_t kPieceLen = 16384, kPieceMin = 256;
constexpr uint32_t kWalkWarps = 32;  // resident warps of a walk per SM
constexpr uint32_t kWalkSlots = 256;  // slots listed at a time
// Ranges of at least this many entries are walked slot by slot, the others flattened over the lanes:
// a round of 32 costs about 40 instructions with one slot's strings in registers and about 100
// when every lane finds its slot (PT2 at n = 40: 6.4 -> 5.4 ms a pseudo-stochastic batch, 13.4 ->
// 11.9 ms for six stochastic iterations; a limit of 24 measures the same).
constexpr uint32_t kWalkLong = 12;

// A warp's shared memory.
struct WalkWarp {
  // slots of the current source with a non-empty range: first entry, entries, code; long ranges
  // from the front, short ones from the back
  uint32_t s_lo[kWalkSlots], s_cnt[kWalkSlots], s_code[kWalkSlots];
  uint8_t occ[128];  // electron -> spatial orbital, alpha electrons first
};

// Entries [skip, skip + left) of det (up, dn)'s windows [eps_min, eps_max), 32 at a time: all lanes
// call push(valid, free, x, e) with x = slot code and targets, e = queue entry, free = both
// targets are free (valid lanes only).
template <class Push>
__device__ __forceinline__ void walk_window(const SelParams& P, WalkWarp& W, uint64_t up,
                                            uint64_t dn, double eps_min, double eps_max,
                                            uint32_t skip, uint32_t left, Push&& push) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int n = P.n_orbs;
  const uint32_t n_off = static_cast<uint32_t>(n);  // an alpha-beta pair's s is stored as s + n
  const uint64_t bu = up | P.inactive, bd = dn | P.inactive;  // (inactive targets: active space)
  __syncwarp();
  for (int o = lane; o < n; o += 32) {
    if (up >> o & 1) W.occ[popc64(up & below(o))] = static_cast<uint8_t>(o);
    if (dn >> o & 1) W.occ[P.n_up + popc64(dn & below(o))] = static_cast<uint8_t>(o);
  }
  __syncwarp();
  const int n_slots = P.n_elecs + P.n_pairs;
  for (int f0 = 0; f0 < n_slots && left; f0 += kWalkSlots) {
    // the non-empty slots of this stretch (a piece's entries: the long ranges in slot order, then
    // the short ones)
    uint32_t n_long = 0, n_short = 0;
    const int f1 = min(n_slots, f0 + (int)kWalkSlots);
    for (int s0 = f0; s0 < f1; s0 += 32) {
      uint32_t lo = 0, c = 0, code = 0;
      if (s0 + (int)lane < f1)
        code = slot_window(P, [&](int e) { return W.occ[e]; }, s0 + lane, eps_min, eps_max, &lo, &c);
      const unsigned bl = __ballot_sync(kFull, c >= kWalkLong);
      const unsigned bs = __ballot_sync(kFull, c && c < kWalkLong);
      if (c) {
        const uint32_t k = c >= kWalkLong ? n_long + __popc(bl & lt)
                                        : kWalkSlots - 1u - n_short - __popc(bs & lt);
        W.s_lo[k] = lo;
        W.s_cnt[k] = c;
        W.s_code[k] = code;
      }
      n_long += __popc(bl);
      n_short += __popc(bs);
    }
    __syncwarp();
    // long ranges: a slot at a time, its strings in registers
    for (uint32_t k = 0; k < n_long && left; k++) {
      const uint32_t c = W.s_cnt[k];
      if (skip >= c) {
        skip -= c;
        continue;
      }
      const uint32_t end = min(c, skip + left);
      left -= end - skip;
      const uint32_t code = W.s_code[k];
      const uint64_t A = code & kADn ? bd : bu;
      const uint64_t B = code & kOne ? 0ull : code & kBDn ? bd : bu;
      const uint32_t lo = W.s_lo[k];
      const uint32_t* __restrict__ q = (code & kOne ? P.s_r : P.d_rs) + lo;
      for (uint32_t t = skip + lane; t < end + lane; t += 64) {
        const bool v0 = t < end, v1 = t + 32 < end;
        const uint32_t x0 = v0 ? q[t] : 0u, x1 = v1 ? q[t + 32] : 0u;
        uint32_t s0 = x0 >> 16, s1 = x1 >> 16;
        if (s0 >= n_off) s0 -= n_off;
        if (s1 >= n_off) s1 -= n_off;
        const uint32_t r0 = x0 & 0xffffu, r1 = x1 & 0xffffu;
        push(v0, v0 && !(bit_of(A, r0) | bit_of(B, s0)), code | r0 << kRBit | s0 << kSBit, lo + t);
        push(v1, v1 && !(bit_of(A, r1) | bit_of(B, s1)), code | r1 << kRBit | s1 << kSBit,
             lo + t + 32);
      }
      skip = 0;
    }
    // short ranges: 32 slots' entries flattened over the lanes
    for (uint32_t g = 0; g < n_short && left; g += 32) {
      const uint32_t k = kWalkSlots - 1u - (g + lane);
      const uint32_t c = g + lane < n_short ? W.s_cnt[k] : 0u;
      uint32_t inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, inc, o);
        if (lane >= (unsigned)o) inc += t;
      }
      const uint32_t total = __shfl_sync(kFull, inc, 31);
      if (skip >= total) {
        skip -= total;
        continue;
      }
      const uint32_t end = min(total, skip + left);
      left -= end - skip;
      const uint32_t first = inc - c;  // of this lane's slot
      for (uint32_t t0 = skip; t0 < end; t0 += 32) {
        const uint32_t t = t0 + lane;
        uint32_t ol = 0;  // owner: the number of slots that end at or before t
#pragma unroll
        for (uint32_t step = 16; step; step >>= 1) {
          const uint32_t v = __shfl_sync(kFull, inc, ol + step - 1);
          if (v <= t) ol += step;
        }
        const uint32_t o_first = __shfl_sync(kFull, first, ol);
        bool free = false;
        uint32_t x = 0, e = 0;
        if (t < end) {
          const uint32_t ok = kWalkSlots - 1u - (g + ol);
          e = W.s_lo[ok] + (t - o_first);
          free = entry_code(P, W.s_code[ok], e, bu, bd, &x);
        }
        push(t < end, free, x, e);
      }
      skip = 0;
    }
    __syncwarp();
  }
}

// ---- pieces -------------------------------------------------------------------------------------

// Pieces of a set of sources (on the device); piece p's region is [off[p], off[p + 1]).
struct PieceList {
  DevBuf<uint32_t> src, begin, len;
  DevBuf<uint64_t> off;
  size_t n = 0;
  uint64_t tot = 0;
  explicit PieceList(shci_ctx* c) {
    src.mt = begin.mt = len.mt = &c->mem;
    off.mt = &c->mem;
  }
};

// walk.cu: pieces of the sources with `entries` window entries each (device).  A piece's region: its
// length with one batch; with several, a piece's members are a binomial(len, 1 / n_batches) count
// per entry of the source (ent_off: a det walked once for several entries), and len / n_batches *
// slack + pad exceeds its mean by many standard deviations (pieces that overflow are emitted
// again).
// flag: a device word whose value is returned (read with the wait for the pieces' number).
unsigned make_pieces(shci_ctx* c, const DevBuf<uint64_t>& entries, uint32_t n_src,
                     uint64_t n_batches, double slack, double pad, const uint32_t* ent_off,
                     PieceList& L, const unsigned* flag = nullptr);

// walk.cu: the end of the run of pieces from k0 whose regions together hold at most `cap` (one piece
// at least); base = off[k0], *end = off[result].
size_t piece_run(shci_ctx* c, const PieceList& L, size_t k0, uint64_t base, uint64_t cap,
                 uint64_t* end);

}  // namespace shci
