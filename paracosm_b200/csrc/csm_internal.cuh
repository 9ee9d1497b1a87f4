// Internal device-side layout shared by the engine's translation units.
//
// Data graph in HBM: a label-partitioned dynamic CSR.
//   - Row v lives at pool[row[v].x .. row[v].x + row[v].y); its first
//     deg(v) slots hold neighbour ids, grouped by "combo" = (neighbour vertex
//     label, edge label) and sorted by id inside each group, so the segment
//     S(v, a, l) (neighbours of v with vertex label a over edges labelled l)
//     is contiguous.  The remaining row[v].y - deg slots are slack for
//     insertions; a row that outgrows its slack is moved to fresh pool space.
//   - dir[v * (NC + 1) + c] is the offset of combo c's segment inside row v
//     (dir[..NC] = deg(v)), so a segment is found with two 4-byte loads.
//   - Two pools alternate: when the active pool cannot absorb a batch's
//     relocations, every row is copied to the other pool with fresh slack.
// Edge updates of one batch are applied to the CSR before the search (the
// "union graph"), and each edge inserted or deleted inside the batch gets a
// temporal entry (its presence intervals in update-sequence numbers), so
// every update of the batch sees exactly the graph the sequential order
// gives it (ParaCOSM/CSM/matching/main.cpp:628-674).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/csm_gpu.h"

namespace csm {

constexpr uint32_t kNone = 0xffffffffu;
constexpr int32_t kTimeInf = 0x7fffffff;
constexpr uint32_t kMaxQ = 32;        // max query vertices
constexpr uint32_t kMaxQE = 256;      // max query edges
constexpr uint32_t kMaxBack = 32;     // backward entries per position
constexpr uint32_t kMaxBatch = 65536;

__host__ __device__ inline uint64_t mix64(uint64_t x) {  // MurmurHash3 fmix64
  x ^= x >> 33; x *= 0xff51afd7ed558ccdULL;
  x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ULL;
  x ^= x >> 33; return x;
}
// Per (query vertex, data vertex) term of the order-independent match hash.
__host__ __device__ inline uint64_t pair_hash(uint32_t q, uint32_t v) {
  return mix64((((uint64_t)(q + 1)) << 32) ^ (uint64_t)v ^ 0x9E3779B97F4A7C15ULL);
}

// Packed sort key of a directed entry (x, combo, y): x in the top bits, then
// the combo, then y, so that sorting groups rows and orders each row by
// (combo, id).  Widths are fixed per context; ids are < 2^yb - 1 so that the
// all-ones key is a sentinel that sorts after every real entry.
struct KeyBits {
  uint32_t yb;  // bits of a vertex id
  uint32_t cb;  // bits of a combo
  __host__ __device__ uint64_t pack(uint32_t x, uint32_t c, uint32_t y) const {
    return ((uint64_t)x << (cb + yb)) | ((uint64_t)c << yb) | (uint64_t)y;
  }
  __host__ __device__ uint32_t x_of(uint64_t k) const { return (uint32_t)(k >> (cb + yb)); }
  __host__ __device__ uint32_t c_of(uint64_t k) const { return (uint32_t)((k >> yb) & ((1ULL << cb) - 1)); }
  __host__ __device__ uint32_t y_of(uint64_t k) const { return (uint32_t)(k & ((1ULL << yb) - 1)); }
  __host__ __device__ uint32_t total() const { return 2 * yb + cb; }
  __host__ __device__ uint64_t sentinel() const { return total() >= 64 ? ~0ULL : ((1ULL << total()) - 1); }
  // Real entries are below the sentinel; unused list slots hold the
  // sentinel or all ones (memset 0xff), both of which fail this test.
  __host__ __device__ bool real(uint64_t k) const { return k < sentinel(); }
};

// Bump allocators and flags of the two alternating row pools.
struct PoolState {
  unsigned long long top[2];  // next free slot of each pool
  unsigned long long need;    // relocation demand of the current batch
  uint32_t active;            // index of the active pool
  uint32_t compact;           // set when this batch must compact first
  uint32_t error;             // nonzero: internal error code (see kErr*)
  uint32_t arrived;           // blocks of a kernel that have arrived (last_block)
};
enum : uint32_t { kErrNone = 0, kErrPoolFull = 1, kErrListOverflow = 2, kErrTaskOverflow = 3, kErrWaitTimeout = 4,
                  kErrBadTask = 5, kErrRingState = 6, kErrTaskGuard = 7, kErrRowState = 8, kErrRowTable = 9 };

// Device view of the dynamic CSR (pointers into device memory).
struct DevGraph {
  uint32_t* vlabel;      // [n_cap]
  uint2* row;            // [n_cap]  x: offset into the active pool, y: capacity
  uint32_t* dir;         // [n_cap * (nc + 1)]
  uint32_t* pools[2];    // the two row pools
  PoolState* ps;
  // temporal entries of the current batch, sorted by packed key (x, combo, nbr)
  uint32_t* t_count;     // [n_cap]  0 = vertex untouched in this batch
  uint64_t* t_key;       // packed keys
  int2* t_span;          // presence interval [start, end] in batch sequence numbers
  ulonglong2* t_tab;     // hash table (key, value) over them: see touched_present
  uint32_t t_mask;       // its slots - 1 for the current batch
  uint64_t pool_cap;     // entries per pool
  // label folding: sorted distinct query labels; label i of the list maps
  // to i, every other label to the inert label (n_qv / n_qe)
  const uint32_t* qlab_v;
  const uint32_t* qlab_e;
  uint32_t n_qv, n_qe;
  uint32_t n, n_cap, n_vl, n_el, nc;  // n_vl = n_qv + 1, n_el = n_qe + 1
  KeyBits kb;
  // Row tables: the entries of row v -- the union graph's during a batch --
  // as a hash set of cap / 4 buckets of 8 slots at htab[2 * off ..), so that
  // "is x a neighbour of v over label l" is one 32-byte load instead of a
  // binary search in v's segment.  An entry whose bucket is full goes to the
  // next one (cyclically); a bucket with an empty slot was never full, which
  // ends a search.  The region moves with the row and is at most half full of
  // live entries; htomb[v] counts its deleted slots.
  // null: no tables (an id and a label do not fit in 31 bits, or no memory).
  uint32_t* htab;
  uint32_t* htomb;       // [n_cap]
  uint32_t hlb;          // bits of a folded edge label in a table entry
};

// Row-table entries: neighbour id, then the folded edge label in the low hlb
// bits, 31 bits together; the top bit marks an entry touched in this batch
// (it has temporal entries).  Two values no entry takes, with or without that
// bit, mark empty and deleted slots.
constexpr uint32_t kSlotEmpty = 0xffffffffu, kSlotTomb = 0xfffffffeu, kSlotTouched = 0x80000000u;
__host__ __device__ __forceinline__ uint32_t row_entry(uint32_t y, uint32_t l, uint32_t hlb) { return (y << hlb) | l; }
// With tables a row's slots come in multiples of four, so that its table starts on a bucket.
__host__ __device__ __forceinline__ uint32_t row_round(uint32_t cap) { return (cap + 3u) & ~3u; }
// Home bucket of an entry in a row table of `buckets` buckets.
__device__ __forceinline__ uint32_t row_bucket(uint32_t entry, uint32_t buckets) {
  // multiplicative hashing, folded once so that the low bits count too; the
  // multipliers are the first two primes of xxHash32
  uint32_t h = entry * 0x9E3779B1u;
  h ^= h >> 15;
  h *= 0x85EBCA77u;
  return __umulhi(h, buckets);
}
// A bucket in one 32-byte load, past L1: its lines are scattered over the
// lanes, and no other load of the SM is likely to want them.
struct RowBucket {
  uint32_t k[8];
};
__device__ __forceinline__ RowBucket ld_bucket(const uint32_t* a) {
  uint64_t w0, w1, w2, w3;
  asm volatile("ld.global.L1::no_allocate.v4.b64 {%0,%1,%2,%3}, [%4];"
               : "=l"(w0), "=l"(w1), "=l"(w2), "=l"(w3)
               : "l"(a));
  return RowBucket{{(uint32_t)w0, (uint32_t)(w0 >> 32), (uint32_t)w1, (uint32_t)(w1 >> 32), (uint32_t)w2,
                    (uint32_t)(w2 >> 32), (uint32_t)w3, (uint32_t)(w3 >> 32)}};
}
// Loads of driver segments, read once per use: they may fill L1 (the next step
// reads on in the line) but go first when L1 needs room.
__device__ __forceinline__ uint32_t ld_stream(const uint32_t* a) {
  uint32_t v;
  asm("ld.global.L1::evict_first.u32 %0, [%1];" : "=r"(v) : "l"(a));
  return v;
}

// Loads scattered over the lanes, whose lines no other load of the SM is likely
// to want: past L1 altogether.
__device__ __forceinline__ uint64_t ld_gather(const uint64_t* a) {
  uint64_t v;
  asm("ld.global.L1::no_allocate.u64 %0, [%1];" : "=l"(v) : "l"(a));
  return v;
}
// The word of `entry` in the row table of row r (with its touched bit), or
// kSlotEmpty when it is not there.  One load settles nearly every search: at
// the tables' load of 0.4 a bucket of 8 overflows for one row entry in 200,
// where linear probing over single slots made a warp wait for the longest of
// its 32 chains (about 8 dependent loads; the hash-enumerating search of 3,001
// updates 9.7 -> 5.9 ms).
__device__ __forceinline__ uint32_t row_find(const DevGraph& g, uint2 r, uint32_t entry) {
  const uint32_t buckets = r.y >> 2;
  const uint32_t* tab = g.htab + 2ull * r.x;
  uint32_t s = row_bucket(entry, buckets);
#pragma unroll 1
  for (uint32_t n = 0; n < buckets; n++) {
    const RowBucket b = ld_bucket(tab + 8ull * s);
    uint32_t hit = kSlotEmpty;
    bool open = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if ((b.k[i] & ~kSlotTouched) == entry) hit = b.k[i];
      open = open || b.k[i] == kSlotEmpty;
    }
    if (hit != kSlotEmpty || open) return hit;
    if (++s == buckets) s = 0;
  }
  return kSlotEmpty;
}

__device__ __forceinline__ uint32_t fold_label(const uint32_t* sorted, uint32_t n, uint32_t l) {
  uint32_t lo = 0, hi = n;
#pragma unroll 1
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (sorted[mid] < l) lo = mid + 1; else hi = mid;
  }
  return (lo < n && sorted[lo] == l) ? lo : n;
}
__device__ __forceinline__ uint32_t fold_vlabel(const DevGraph& g, uint32_t l) {
  return l == kNone ? kNone : fold_label(g.qlab_v, g.n_qv, l);
}
__device__ __forceinline__ uint32_t fold_elabel(const DevGraph& g, uint32_t l) { return fold_label(g.qlab_e, g.n_qe, l); }

// Segment [lo, hi) of combo c in row v, as absolute pool offsets.
__device__ __forceinline__ void segment(const DevGraph& g, uint32_t v, uint32_t c, uint64_t& lo, uint64_t& hi) {
  const uint32_t* d = g.dir + (size_t)v * (g.nc + 1) + c;
  const uint64_t base = g.row[v].x;
  lo = base + d[0];
  hi = base + d[1];
}

// lower_bound over a sorted uint32 range; returns the first index with a[i] >= x.
__device__ __forceinline__ uint64_t lower_bound_u32(const uint32_t* a, uint64_t lo, uint64_t hi, uint32_t x) {
#pragma unroll 1
  while (lo < hi) {
    uint64_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ bool contains_u32(const uint32_t* a, uint64_t lo, uint64_t hi, uint32_t x) {
  uint64_t p = lower_bound_u32(a, lo, hi, x);
  return p < hi && a[p] == x;
}

// Finds edge (x, y) in the union graph; returns its folded label or kNone.
__device__ __forceinline__ uint32_t find_label(const DevGraph& g, const uint32_t* pool, uint32_t x, uint32_t y) {
  const uint32_t ly = g.vlabel[y];
#pragma unroll 1
  for (uint32_t l = 0; l < g.n_el; l++) {
    uint64_t lo, hi;
    segment(g, x, ly * g.n_el + l, lo, hi);
    if (contains_u32(pool, lo, hi, y)) return l;
  }
  return kNone;
}

// Temporal table: a hash set (linear probing, empty key kTempEmpty) that holds,
// for every touched entry (v, c, w) of the batch, its presence, and for every
// segment (v, c) with touched entries -- key (v, c, all ones) -- the run of
// them in t_key: first index, and length in the upper half.  An entry's value
// is its one interval (start + 1, end), or, when it has several, kTempMany and
// the run of t_span indices (first, and length in the upper half).
constexpr uint64_t kTempEmpty = ~0ULL, kTempMany = 1ULL << 63;
__device__ __forceinline__ uint64_t temporal_head(const DevGraph& g, uint32_t v, uint32_t c) {
  return g.kb.pack(v, c, (uint32_t)((1ULL << g.kb.yb) - 1));
}
__device__ __forceinline__ uint32_t temporal_slot(uint64_t key, uint32_t mask) {
  uint64_t h = key * 0x9E3779B97F4A7C15ULL;
  h ^= h >> 32;
  return (uint32_t)h & mask;
}
// Value of a key, or kTempEmpty.
__device__ __forceinline__ uint64_t temporal_find(const DevGraph& g, uint64_t key) {
  uint32_t s = temporal_slot(key, g.t_mask);
#pragma unroll 1
  for (;; s = (s + 1) & g.t_mask) {  // at most a quarter full: an empty slot ends it
    const ulonglong2 e = g.t_tab[s];
    if (e.x == key) return e.y;
    if (e.x == kTempEmpty) return kTempEmpty;
  }
}
__device__ __forceinline__ bool temporal_present(const DevGraph& g, uint64_t val, int32_t t) {
  if (!(val & kTempMany)) return (int32_t)(uint32_t)val - 1 <= t && t <= (int32_t)(val >> 32);
  const uint32_t beg = (uint32_t)val, n = (uint32_t)((val & ~kTempMany) >> 32);
#pragma unroll 1
  for (uint32_t i = beg; i < beg + n; i++) {
    const int2 s = g.t_span[i];
    if (s.x <= t && t <= s.y) return true;
  }
  return false;
}

// Is edge (v, w) with combo c present at batch time t?  Only called for
// edges found in the union graph; edges not touched in this batch are present.
__device__ __forceinline__ bool touched_present(const DevGraph& g, uint32_t v, uint32_t c, uint32_t w, int32_t t) {
  const uint64_t val = temporal_find(g, g.kb.pack(v, c, w));
  return val == kTempEmpty || temporal_present(g, val, t);
}

// Entries of a segment's run [beg, end) of touched entries that are absent at
// batch time t, as far as every step-th index from `at` on tells: an entry's
// intervals do not overlap, so it is its first index less the one interval that
// holds t.  Negative shares are made up for by others.  (Unrolled four times it
// takes the registers of every search: counting ones 4 to 8 % slower.)
__device__ __forceinline__ int32_t seg_absent(const DevGraph& g, uint32_t at, uint32_t beg, uint32_t end,
                                              uint32_t step, int32_t t) {
  int32_t absent = 0;
#pragma unroll 1
  for (uint32_t i = at; i < end; i += step) {
    const bool first = i == beg || g.t_key[i - 1] != g.t_key[i];
    const int2 sp = g.t_span[i];
    absent += (int32_t)first - (int32_t)(sp.x <= t && t <= sp.y);
  }
  return absent;
}

// Number of entries of segment (v, c) present at batch time t, given its
// union-graph bounds: entries touched in this batch and absent at t are
// subtracted.
__device__ __forceinline__ uint32_t seg_size_at(const DevGraph& g, uint32_t v, uint32_t c, uint64_t lo, uint64_t hi,
                                                int32_t t) {
  const uint32_t size = (uint32_t)(hi - lo);
  if (size == 0 || g.t_count[v] == 0) return size;
  const uint64_t run = temporal_find(g, temporal_head(g, v, c));
  if (run == kTempEmpty) return size;
  const uint32_t beg = (uint32_t)run, end = beg + (uint32_t)(run >> 32);
  return size - (uint32_t)seg_absent(g, beg, beg, end, 1, t);
}

// ---- query plan ------------------------------------------------------
// One plan per anchor query edge: positions 0 and 1 are the anchor's end
// points, the others follow the GraphFlow order of that edge
// (ParaCOSM/CSM/matching/GraphFlow/graphflow.cpp:36-169).  Position d >= 2
// has back entries (earlier position, combo of the edge to it) and a mask of
// earlier positions with the same vertex label (injectivity).
struct PlanPos {
  uint8_t qv;          // query vertex at this position
  uint8_t nb;          // number of back entries
  uint16_t boff;       // first back entry in PlanAnchor::back_*
  uint32_t samelab;    // bitmask over earlier positions with the same label
};

// Independent tail of an order: positions tail_at + 1 .. n - 1 have no query
// edge among them and no vertex label more than kTailGroup times, so once
// positions 0 .. tail_at are matched the completions are a product over the
// tail's label groups of injective assignments, counted without enumerating
// them.  Groups are listed in order of their first position (gpos: the
// positions, group after group, ascending inside a group; gsize: sizes).
constexpr uint32_t kTailGroup = 3;

struct PlanAnchor {
  uint32_t la, lb, el;       // label triple of the anchor (pos 0 label, pos 1 label, edge label)
  uint32_t tree;             // the anchor is an edge of the TurboFlux spanning tree (compat deletions)
  uint32_t prefix_mask;      // positions 0 .. tail_at
  uint8_t tail_at;           // last position matched one by one before the tail; 0: no tail
  uint8_t n_groups;
  uint8_t pad_[2];
  uint8_t gsize[kMaxQ];
  uint8_t gpos[kMaxQ];
  PlanPos pos[kMaxQ];
  uint8_t back_pos[kMaxQE];
  uint16_t back_combo[kMaxQE];
  uint8_t back_el[kMaxQE];   // folded edge label of each back entry
};

struct Plan {
  uint32_t n;          // query vertices
  uint32_t n_anchor;   // query edges
  PlanAnchor anchors[kMaxQE];
};

// Root search task: one (update, anchor edge, orientation) seed.
struct Task {
  uint32_t upd;        // index of the update inside the batch (= its batch time)
  uint16_t anchor;
  uint8_t orient;      // 0: (v1, v2) -> positions (0, 1); 1: swapped
  uint8_t pad;
};

// Batch-level per-update working state.
struct UpdInfo {
  uint32_t v1, v2;     // endpoints as given
  uint32_t label;      // anchor label used for counting (existing label for deletions)
  uint32_t flags;      // bit0 valid edge update, bit1 insertion, bit2 mutation applied, bit3 invalid
};
// UF_DUP: an insertion of an edge that is present at that point of the batch
enum : uint32_t { UF_VALID = 1u, UF_ADD = 2u, UF_MUT = 4u, UF_INVALID = 8u, UF_DUP = 16u };

}  // namespace csm
