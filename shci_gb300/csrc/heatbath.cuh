// Heat-bath candidate generation shared by selection (select.cu) and PT2 (pt2.cu).
//
// The reference's ChemSystem::find_connected_dets (src/chem/chem_system.cc:289-402) walks
// singles_queue[p] and hci_queue[pq] (sorted by descending |H|) until the first entry below
// eps_min, skipping doubles with |H| >= eps_max.  The same queues sit in HBM in CSR form and
// a binary search gives each (det, slot) its exact entry range.  A det has n_elecs "single"
// slots (one per electron) and n_elecs (n_elecs - 1) / 2 "double" slots (one per electron
// pair, in the reference's p_id < q_id order).
#pragma once

#include "common.cuh"

namespace shci {

constexpr int kSelWarps = 8;
constexpr uint64_t kInvalid = ~0ull;

struct SelParams {
  DevIntegrals I;
  const uint64_t* up;
  const uint64_t* dn;
  const double* coef;
  double* eps_tried;
  const uint64_t* d_off;
  const double* d_H;
  const uint32_t* d_rs;
  const uint32_t* s_off;
  const double* s_S;
  const uint32_t* s_r;
  const uint32_t* pair_tab;  // pair k -> p_id | q_id << 16
  const unsigned long long* set_hash;  // hash set of the variational dets (see set_index)
  uint64_t set_hash_mask;
  double eps_var;
  double max_hci, max_singles;
  int n_orbs, n_up, n_elecs, n_pairs;
  int var_sd;
  // second rejection (chem_system.cc:300-308, 318-324, 364-370): off unless rej_on
  int rej_on;
  double rej_factor;  // second_rejection_factor
  double e_hf_1b;     // sum of h_pp over the HF det's electrons (chem_system.cc:812-823)
  int time_sym;       // time-reversal symmetry: list holds up <= dn, open dets stand for pairs
  // find_connected_dets options: no double excitations (has_double_excitation false,
  // chem_system.cc:345) and orbitals that may not be targets (the active space,
  // chem_system.cc:327-329, 383-387); 0 and 0 are the reference's defaults
  int no_doubles;
  uint64_t inactive;
};

constexpr double kSqrt2 = 1.4142135623730951;  // Util::SQRT2 (src/util.h:58)

// Position of the k-th set bit of x (k from 0, below the number of bits): halves by population
// count, a third of the instructions of __fns.
__device__ __forceinline__ int nth_bit(uint64_t x, int k) {
  unsigned w = static_cast<unsigned>(x);
  int pos = 0, c = __popc(w);
  if (k >= c) {
    k -= c;
    w = static_cast<unsigned>(x >> 32);
    pos = 32;
  }
#pragma unroll
  for (int h = 16; h; h >>= 1) {
    c = __popc(w & ((1u << h) - 1u));
    if (k >= c) {
      k -= c;
      w >>= h;
      pos += h;
    }
  }
  return pos;
}

// First k in [lo, hi) with a[k] < x, for a descending array of non-negative values and
// any x.  Non-negative doubles order like the integers of their bit patterns (a negative or
// NaN x compares false against every entry, as in FP64), so the comparisons run on the
// integer pipe (the FP64 pipe is slow on GB300) with the same result.
__device__ __forceinline__ uint32_t first_below(const double* a, uint32_t lo, uint32_t hi,
                                                double x) {
  long long xb = __double_as_longlong(x);
  if ((xb & 0x7fffffffffffffffll) > 0x7ff0000000000000ll) xb = -1;  // NaN: never above an entry
  const long long* ab = reinterpret_cast<const long long*>(a);
  // the usual cases: the window starts at the slot's largest entry or is empty
  if (lo < hi && ab[lo] < xb) return lo;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (ab[mid] < xb) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

__device__ __forceinline__ size_t c2(size_t a, size_t b) {
  return a > b ? (a * (a + 1)) / 2 + b : (b * (b + 1)) / 2 + a;
}

// Slot code: the orbitals p and q that the electrons leave, and the strings that the targets r and s
// of an entry must be free in; an entry's code adds its targets.  A queue entry's r | s << 16 holds
// the targets of the stored pair; a beta-beta pair is stored as its alpha image and an alpha-beta
// pair p > q as (q, p) (chem_system.cc:347-361), so the strings follow from the slot alone.
constexpr int kPBit = 0, kQBit = 6, kRBit = 12, kSBit = 18;
enum : uint32_t { kADn = 1u << 24, kBDn = 1u << 25, kOne = 1u << 26 };

// Entry range [lo, lo + cnt) of slot `slot` of a det in the eps window [eps_min, eps_max), and the
// slot's code; orb(e) is the spatial orbital of electron e, alpha electrons first.
template <class Orb>
__device__ __forceinline__ uint32_t slot_window(const SelParams& P, Orb&& orb, int slot,
                                                double eps_min, double eps_max, uint32_t* lo,
                                                uint32_t* cnt) {
  *lo = 0;
  *cnt = 0;
  const int n = P.n_orbs;
  if (slot < P.n_elecs) {
    if (eps_min > P.max_singles) return 0;
    const uint32_t p = orb(slot);
    const uint32_t a = P.s_off[p], b = P.s_off[p + 1];
    *lo = a;
    *cnt = first_below(P.s_S, a, b, eps_min) - a;
    return p << kPBit | kOne | (slot < P.n_up ? 0u : kADn);
  }
  if (P.no_doubles || eps_min > P.max_hci) return 0;
  const uint32_t pr = P.pair_tab[slot - P.n_elecs];
  const int e1 = pr & 0xffff, e2 = pr >> 16;
  const uint32_t p = orb(e1), q = orb(e2);
  const bool dn1 = e1 >= P.n_up, dn2 = e2 >= P.n_up;
  uint32_t code;
  size_t pq;
  if (dn1 == dn2) {
    pq = c2(p, q);
    code = p << kPBit | q << kQBit | (dn1 ? kADn | kBDn : 0u);
  } else if (p > q) {  // stored as (q, p + n): r goes to beta, s to alpha
    pq = c2(q, p + n);
    code = p << kPBit | q << kQBit | kADn;
  } else {
    pq = c2(p, q + n);
    code = p << kPBit | q << kQBit | kBDn;
  }
  const uint32_t a = static_cast<uint32_t>(P.d_off[pq]), b = static_cast<uint32_t>(P.d_off[pq + 1]);
  const uint32_t s = first_below(P.d_H, a, b, eps_max);
  *lo = s;
  *cnt = first_below(P.d_H, s, b, eps_min) - s;
  return code;
}

// The same with the orbitals from the det's strings.
__device__ __forceinline__ uint32_t slot_range(const SelParams& P, uint64_t up, uint64_t dn,
                                               int slot, double eps_min, double eps_max,
                                               uint32_t* lo, uint32_t* cnt) {
  return slot_window(
      P, [&](int e) { return e < P.n_up ? nth_bit(up, e) : nth_bit(dn, e - P.n_up); }, slot, eps_min,
      eps_max, lo, cnt);
}

__device__ __forceinline__ uint32_t bit_of(uint64_t x, uint32_t k) {
  const uint32_t w = k & 32u ? static_cast<uint32_t>(x >> 32) : static_cast<uint32_t>(x);
  return w >> (k & 31u) & 1u;
}

// Code of queue entry e of the slot with code `code`; false where a target is occupied or inactive
// (active space): bu and bd hold those orbitals.
__device__ __forceinline__ bool entry_code(const SelParams& P, uint32_t code, uint32_t e,
                                           uint64_t bu, uint64_t bd, uint32_t* x) {
  const uint32_t n = static_cast<uint32_t>(P.n_orbs);  // an alpha-beta pair's s is stored as s + n
  const uint64_t A = code & kADn ? bd : bu;
  const uint64_t B = code & kOne ? 0ull : code & kBDn ? bd : bu;
  const uint32_t rs = code & kOne ? P.s_r[e] : P.d_rs[e];
  const uint32_t r = rs & 0xffffu;
  uint32_t s = rs >> 16;
  if (s >= n) s -= n;
  *x = code | r << kRBit | s << kSBit;
  return !(bit_of(A, r) | bit_of(B, s));
}

// The determinant that entry `code` (with its targets) makes of (*u, *d).
__device__ __forceinline__ void apply_entry(uint32_t code, uint64_t* u, uint64_t* d) {
  const uint64_t out1 = 1ull << (code >> kPBit & 63u), out2 = 1ull << (code >> kQBit & 63u);
  const uint64_t in1 = 1ull << (code >> kRBit & 63u), in2 = 1ull << (code >> kSBit & 63u);
  // (targets are in the strings A and B; the electrons that leave: of the first electron's string
  // and the second's, which for a swapped pair are B and A)
  const bool a_dn = code & kADn, b_dn = code & kBDn;
  if (code & kOne) {
    if (a_dn) *d ^= out1 | in1;
    else *u ^= out1 | in1;
  } else if (a_dn == b_dn) {
    const uint64_t x = out1 | out2 | in1 | in2;
    if (a_dn) *d ^= x;
    else *u ^= x;
  } else {
    *u ^= out1 | (a_dn ? in2 : in1);
    *d ^= out2 | (a_dn ? in1 : in2);
  }
}

// Slot hash of a det for the variational hash set (this set is internal: no other hash has
// to agree with it): the strings combined by one multiply, then a multiply-xorshift finaliser
// so that the low bits index the table and the high bits fingerprint.  About a dozen integer
// instructions, against about seventy for the reference's det hash plus a finaliser; every
// PT2 candidate and selection candidate pays it.
__host__ __device__ __forceinline__ uint64_t set_slot_hash(uint64_t u, uint64_t d) {
  uint64_t h = u * 0x9E3779B97F4A7C15ull + d;
  h ^= h >> 32;
  h *= 0xD6E8FEB86659FD93ull;
  h ^= h >> 29;
  return h;
}

// Id of det (u, d) in the hash set of the variational dets, or -1 (slots hold fingerprint << 32 |
// det id + 1, linear probing, at most half full): one or two probes, then a comparison against
// the det list.
__device__ __forceinline__ long long set_index(const SelParams& P, uint64_t u, uint64_t d) {
  const uint64_t h = set_slot_hash(u, d);
  const uint32_t fp = static_cast<uint32_t>(h >> 32);
  uint64_t p = h & P.set_hash_mask;
  for (uint64_t probe = 0; probe <= P.set_hash_mask; probe++) {
    const unsigned long long v = P.set_hash[p];
    if (v == 0ull) return -1;
    if (static_cast<uint32_t>(v >> 32) == fp) {
      const uint32_t id = static_cast<uint32_t>(v) - 1u;
      if (P.up[id] == u && P.dn[id] == d) return id;
    }
    p = (p + 1) & P.set_hash_mask;
  }
  return -1;
}

__device__ __forceinline__ bool in_set(const SelParams& P, uint64_t u, uint64_t d) {
  return set_index(P, u, d) >= 0;
}

__device__ __forceinline__ double src_eps_min(const SelParams& P, uint32_t i) {
  double e = P.eps_var / fabs(P.coef[i]);
  if (i == 0 && P.var_sd) e = 0.0;
  if (P.time_sym && P.up[i] != P.dn[i]) e *= kSqrt2;  // solver.h:447
  return e;
}

}  // namespace shci
