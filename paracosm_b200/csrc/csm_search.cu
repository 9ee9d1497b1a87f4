// Search kernels: seeding, the warp-cooperative expansion, finalisation.
//
// Reference semantics restated (paths inside ParaCOSM/CSM):
//   seeds of an edge update ......... matching/GraphFlow/graphflow.cpp:305-352 (each query
//                                     edge whose label triple matches, both orientations)
//   candidate generation / join ..... matching/GraphFlow/graphflow.cpp:181-265 (label filter,
//                                     adjacency to every matched query neighbour, injectivity)
//   index filter (TurboFlux/SymBi) .. matching/SymBi/symbi.cpp:516 (candidate must have d2 set)
//   per-update cap .................. matching/SymBi/symbi.cpp:583 (stop at exactly the cap)
//   Classify (safe update) .......... matching/Parallel_GraphFlow/parallel_graphflow.cpp:1990-2016
//
// Expansion scheme.  A warp owns one root task (update, anchor edge,
// orientation) at a time and walks its search tree depth first, but each
// level holds up to 32 partial matches at once: to extend level d the warp
// takes the next 32 (entry, driver element) pairs of level d's entries -- the
// driver being the smallest back-neighbour segment -- so lanes stay busy even
// when segments are a few elements long.  A step first applies the two tests
// that settle most candidates and need nothing but the entry -- the candidate
// filter's bit and one probe of a row table -- and only the candidates left
// rebuild their prefix for the other joins, the same-label matched vertices
// (injectivity) and the batch-time presence of every back edge; survivors are
// compacted with a ballot into level d + 1 together with the driver segment
// of their own next level (an empty next-level segment prunes them right
// away).  Leaves are only counted.
#include <algorithm>

#include "csm_kernels.cuh"

namespace csm {

// One level of a warp's walk: up to 32 partial matches, each with the driver
// segment of the next position.  The segments are laid end to end, so the
// level's work is the range [cur, total) of (entry, driver element) pairs and
// a pair's pool offset is base[entry] + its place in the range.
// Level 1 has one entry: v[0] is position 1's vertex, and its parent, v[1],
// position 0's.
struct LevelSM {
  uint32_t v[32];     // data vertex of this level's position
  uint32_t incl[32];  // end of each entry's driver segment in the range
  uint32_t base[32];  // pool offset of the segment minus its start in the range
  uint32_t jv[32];    // matched vertex of the entry's first join
  uint8_t par[32];    // entry index in the previous level
  uint8_t dsel[32];   // back entry that is the driver (kSelTouched: its row has touched entries)
  uint8_t jsel[32];   // back entry of the first join: the smallest segment but the driver's
  uint8_t jel[32];    // its edge label
  uint32_t cnt, cur, total;
  uint32_t burst;     // tail's level: entries the next stage takes
};

// Elements of a level's or a tail member's range: 32-bit positions, and a step
// looks up to 64 past the last one.  (Another limit than the default is for
// testing: it has every walk reach what otherwise takes rows of 2^27 entries.)
#ifndef CSM_RANGE_MAX
#define CSM_RANGE_MAX 0xffffff00u
#endif
constexpr uint32_t kRangeMax = CSM_RANGE_MAX;
// 32 segments below this size fit in a range.
constexpr uint32_t kRangeWide = kRangeMax / 32 + 1;

// Graphs without row tables, or with rows that long, take instantiations of
// their own (GEN below): the few instructions that look for either cost the
// counting search of 2,000 insertions on a graph in L2 10 % and of 4,097 updates
// on 2^19 vertices 7 %.
static bool search_general(const DevGraph& g) { return !g.htab || g.n_cap >= kRangeWide; }

// Levels a walk of this plan may use: 1 .. n - 2, or, where every order's
// independent tail is counted, up to the tail with the class counters of
// tail_stage above it.
static uint32_t search_levels(const Plan& plan, int mode) {
  const uint32_t n = plan.n;
  uint32_t levels = n > 2 ? n - 2 : 1;
  if (mode != 2) return levels;
  constexpr uint32_t kCounters = (((1u << kTailGroup) - 1u) * 32u * 4u + sizeof(LevelSM) - 1) / sizeof(LevelSM);
  uint32_t need = 1;
  for (uint32_t a = 0; a < plan.n_anchor; a++)
    need = std::max<uint32_t>(need, plan.anchors[a].tail_at ? plan.anchors[a].tail_at + kCounters : levels);
  return need;
}

// Shared memory of one warp: its levels, then its walk's plan (WalkPlan).
SearchShape search_shape_of(const Plan& plan, int mode, const DevGraph& g) {
  SearchShape s;
  s.general = search_general(g);
  s.levels = search_levels(plan, mode);
  const uint32_t words = 3 * plan.n + (plan.n_anchor ? plan.n_anchor - 1 : 0);  // every query edge but the anchor is a back entry once
  s.warp_bytes = s.levels * (uint32_t)sizeof(LevelSM) + ((4 * words + 15) & ~15u);
  return s;
}

__device__ __forceinline__ bool d2_bit(const uint64_t* d2, uint64_t words, uint32_t q, uint32_t v) {
  return (d2[(uint64_t)q * words + (v >> 6)] >> (v & 63)) & 1ULL;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Per launch: tickets keep counting up across launches (the ring's slot
// sequence numbers stay consistent); hunger and pending start afresh, and the
// tickets that warps still waiting at the end of the last launch held (never
// filled) are handed out again.
__device__ __forceinline__ void search_prep(SearchQueue* q, SearchStats* ss, uint32_t tasks, unsigned int* error) {
  if (q->head < q->tail) atomicExch(error, kErrRingState);
  q->head = q->tail;  // tickets that waiting warps held when the last launch ended were never filled
  q->hungry = 0;
  q->pending = tasks;
  ss->launch_t0 = global_ns();
}
__global__ void k_search_prep(SearchQueue* q, const unsigned int* n_tasks, uint32_t task_cap, SearchStats* ss,
                              unsigned int* error) {
  search_prep(q, ss, min(*n_tasks, task_cap), error);
}

// One warp per update, a lane per anchor (one thread trying the anchors in
// turn took 9.6 us for a single update of a 35-edge query, its loads one
// after another).  With `q` (one update only) the warp also prepares the
// search's queue, as k_search_prep does.
__global__ void k_seed(uint32_t B, const UpdInfo* info, DevGraph g, const Plan* plan, const uint64_t* d2,
                       uint64_t d2_words, Task* tasks, unsigned int* n_tasks, uint32_t task_cap,
                       uint32_t* safe, unsigned int* error, Counters ctr, uint32_t shard_rank, uint32_t shard_count,
                       uint32_t turboflux_compat, uint32_t dup_zero, SearchQueue* q, SearchStats* ss) {
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= B) return;
  const UpdInfo u = info[s];
  bool matches = false;
  uint32_t made = 0;
  // dup_zero: an insertion of a present edge counts nothing (CaLiG skips it,
  // ParaCOSM/CSM/matching/Parallel_CaLiG/parallel_calig.cpp:1249)
  if ((u.flags & UF_VALID) && !(u.flags & UF_INVALID) && !(dup_zero && (u.flags & UF_DUP))) {
    const uint32_t L1 = g.vlabel[u.v1], L2 = g.vlabel[u.v2], l = u.label;
    const uint32_t na = plan->n_anchor;
    // The reference's TurboFlux deletion seeds every query edge whose vertex
    // labels match, whatever its edge label, and filters the endpoints by d2
    // only on spanning-tree edges (ParaCOSM/CSM/matching/TurboFlux/turboflux.cpp:966-1022)
    const bool compat_del = turboflux_compat && !(u.flags & UF_ADD);
    for (uint32_t a = lane; a < na; a += 32) {
      const PlanAnchor* A = &plan->anchors[a];
      const uint32_t el = A->el, la = A->la, lb = A->lb;
      if (el != l && !compat_del) continue;
      const bool o0 = la == L1 && lb == L2;
      const bool o1 = la == L2 && lb == L1;
      matches = matches || o0 || o1;
      for (int o = 0; o < 2; o++) {
        if (!(o ? o1 : o0)) continue;
        const uint32_t x = o ? u.v2 : u.v1, y = o ? u.v1 : u.v2;
        if (d2 && (!compat_del || A->tree) &&
            !(d2_bit(d2, d2_words, A->pos[0].qv, x) && d2_bit(d2, d2_words, A->pos[1].qv, y)))
          continue;
        if (shard_count > 1 && (s + 2 * a + (uint32_t)o) % shard_count != shard_rank) continue;  // another GPU's
        unsigned int i = atomicAdd(n_tasks, 1u);
        if (i >= task_cap) { atomicExch(error, kErrTaskOverflow); continue; }
        tasks[i] = Task{s, (uint16_t)a, (uint8_t)o, 0};
        made++;
      }
    }
  }
  matches = __any_sync(0xffffffffu, matches);
  if (lane == 0) {
    safe[s] = matches ? 0u : 1u;
    ctr.count[s] = 0; ctr.hash[s] = 0; ctr.bytes[s] = 0; ctr.stop[s] = 0;
  }
  if (q) {
    made = __reduce_add_sync(0xffffffffu, made);
    if (lane == 0) search_prep(q, ss, made, error);
  }
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, uint32_t lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= (uint32_t)o) v += t;
  }
  return v;
}

// A walk's order in the warp's shared memory, copied from the plan when a task
// starts: three words a position (query vertex, back entries and the first
// one; same-label positions; positions with a back entry), then one word a
// back entry (position, edge label, combo).  Every step reads it, and L1 is
// swept by the search's random loads.
struct WalkPlan {
  const uint32_t* w;
  uint32_t n;
  __device__ __forceinline__ uint32_t qv(uint32_t pos) const { return w[3 * pos] & 0xffu; }
  __device__ __forceinline__ uint32_t nb(uint32_t pos) const { return (w[3 * pos] >> 8) & 0xffu; }
  __device__ __forceinline__ uint32_t samelab(uint32_t pos) const { return w[3 * pos + 1]; }
  __device__ __forceinline__ uint32_t backmask(uint32_t pos) const { return w[3 * pos + 2]; }
  __device__ __forceinline__ uint32_t back(uint32_t pos, uint32_t b) const {
    return w[3 * n + (w[3 * pos] >> 16) + b];
  }
};
__device__ __forceinline__ uint32_t back_el(uint32_t w) { return (w >> 8) & 0xffu; }
__device__ __forceinline__ uint32_t back_combo(uint32_t w) { return w >> 16; }

// `same`: the same-label positions an injectivity test looks at (none under
// homomorphism; only those before the tail when it is counted).
__device__ __forceinline__ void load_walk_plan(uint32_t* w, const PlanAnchor* A, uint32_t n, uint32_t same,
                                               uint32_t lane) {
  uint32_t backs = 0;
  if (lane < n) {
    const PlanPos P = A->pos[lane];
    uint32_t bm = 0;
#pragma unroll 1
    for (uint32_t b = 0; b < P.nb; b++) bm |= 1u << A->back_pos[P.boff + b];
    w[3 * lane] = (uint32_t)P.qv | ((uint32_t)P.nb << 8) | ((uint32_t)P.boff << 16);
    w[3 * lane + 1] = P.samelab & same;
    w[3 * lane + 2] = bm;
    backs = (uint32_t)P.boff + P.nb;
  }
  backs = __reduce_max_sync(0xffffffffu, backs);
  for (uint32_t i = lane; i < backs; i += 32)
    w[3 * n + i] = (uint32_t)A->back_pos[i] | ((uint32_t)A->back_el[i] << 8) | ((uint32_t)A->back_combo[i] << 16);
  __syncwarp();
}

// Visits (position, data vertex) of the prefix of entry e of level d at the
// positions of `mask`, the last one first.  Every position is read from the
// levels when it is needed: a copy of the prefix per lane would be local
// memory, and the random loads leave it no room in L1.
template <class F>
__device__ __forceinline__ void walk_prefix(const LevelSM* lv, int d, uint32_t e, uint32_t mask, F visit) {
#pragma unroll 1
  for (int j = d; mask; --j) {
    const LevelSM& S = lv[j ? j : 1];
    if ((mask >> j) & 1u) {
      visit((uint32_t)j, S.v[e]);
      mask &= ~(1u << j);
    }
    e = S.par[e];
  }
}

// Candidate filter bit of x for query vertex qv.
__device__ __forceinline__ bool filter_bit(const SearchParams& p, uint32_t qv, uint32_t x) {
  return !p.d2 || ((ld_gather(p.d2 + (uint64_t)qv * p.d2_words + (x >> 6)) >> (x & 63)) & 1ULL);
}

// The paths few candidates take are functions of their own: inlined and
// unrolled into every use they made the search 290 KB of code, several times
// the instruction cache, and warps waited for instructions as long as for
// data (7.8 of 33 cycles per instruction on a graph that stays in L2).
__device__ __noinline__ bool present_slow(const SearchParams& p, uint32_t v, uint32_t c, uint32_t w, int32_t t) {
  return touched_present(p.g, v, c, w, t);
}
__device__ __noinline__ uint32_t seg_size_slow(const SearchParams& p, uint32_t v, uint32_t c, uint32_t lo, uint32_t hi,
                                               int32_t t) {
  return seg_size_at(p.g, v, c, lo, hi, t);
}
// Join without row tables: a binary search in v's segment.  The first join of a
// candidate runs before the gather here as well (run_levels): left to
// check_rest, behind the filter and one after another from the last position
// on, the joins took the search of 65,536 updates on 2^22 vertices 310 ms
// (168 ms now, with tables 117), of 4,097 on 2^19 29 (27, 18), of a
// hash-enumerating 3,001 on 2^17 8.4 (5.5, 4.0).
__device__ __noinline__ uint32_t join_search(const SearchParams& p, const uint32_t* pool, uint32_t v, uint32_t c,
                                             uint32_t x) {
  uint64_t lo, hi;
  segment(p.g, v, c, lo, hi);
  if (!contains_u32(pool, lo, hi, x)) return kSlotEmpty;
  return p.g.t_count[v] ? kSlotTouched : 0u;
}

// Is x a neighbour of v over back entry bw?  kSlotEmpty when it is not, else
// a word whose touched bit says that the edge's presence intervals must be
// asked.  One probe of v's row table, or a binary search in v's segment where
// the graph has no tables.
template <bool GEN>
__device__ __forceinline__ uint32_t join_find(const SearchParams& p, const uint32_t* pool, uint32_t v, uint32_t bw,
                                              uint32_t x) {
  if (!GEN || p.g.htab) return row_find(p.g, p.g.row[v], row_entry(x, back_el(bw), p.g.hlb));
  return join_search(p, pool, v, back_combo(bw), x);
}

// LevelSM::dsel: the driver, and whether its row has entries touched in this
// batch (else every entry of the segment is present at every batch time).
constexpr uint32_t kSelMask = 0x1fu, kSelTouched = 0x80u, kSelNone = 0xffu;

// The tests of candidate x for position `pos` beyond the filter bit, for the
// prefix of entry e of level d: injectivity, every join, the batch-time
// presence of every back edge.  `dsel` (LevelSM::dsel) is the back entry whose
// segment produced x (kSelNone: none) and `joined` one that was found before,
// with word jhit (0xff: none).  The joins run one at a time and stop at the
// first that fails; where no test needs the prefix, it is not walked.
template <bool GEN>
__device__ __forceinline__ bool check_rest(const SearchParams& p, const uint32_t* pool, const LevelSM* lv,
                                           const WalkPlan& wp, int d, uint32_t e, uint32_t pos, uint32_t x,
                                           uint32_t dsel, uint32_t joined, uint32_t jhit, int32_t t) {
  const uint32_t same = wp.samelab(pos), bm = wp.backmask(pos);
  uint32_t joins = bm;
  if (dsel != kSelNone && !(dsel & kSelTouched)) joins &= ~(1u << (wp.back(pos, dsel & kSelMask) & 0xffu));
  if (joined != 0xffu && !(jhit & kSlotTouched)) joins &= ~(1u << (wp.back(pos, joined) & 0xffu));
  bool ok = true;
  walk_prefix(lv, d, e, same | joins, [&](uint32_t j, uint32_t v) {
    if ((same >> j) & 1u) ok = ok && v != x;
    if (((joins >> j) & 1u) && ok) {
      const uint32_t b = __popc(bm & ((1u << j) - 1u));
      const uint32_t bw = wp.back(pos, b);
      const uint32_t hit = b == joined ? jhit : join_find<GEN>(p, pool, v, bw, x);
      ok = hit != kSlotEmpty && (!(hit & kSlotTouched) || present_slow(p, v, back_combo(bw), x, t));
    }
  });
  return ok;
}

// Driver of position np (the smallest union-graph back segment, the first of
// equals; with kSelTouched) for the prefix of entry e of level d, continued by x at position
// d + 1 when `with_x`; false if some back segment is empty at batch time t.
// `jsel` and `jv` are the first join -- the back entry of the smallest segment
// but the driver's, and its vertex: the row most likely to lack a candidate,
// and the row table whose lines a warp's lanes share most -- and `bytes`
// receives 4 B x the sizes at time t of all back segments: the
// algorithmic bytes of expanding this node.  Segment bounds and touch counts
// are loaded four back entries at a time, all loads independent.
__device__ __forceinline__ bool pick_driver(const SearchParams& p, const LevelSM* lv, const WalkPlan& wp, int d,
                                            uint32_t e, bool with_x, uint32_t x, uint32_t np, int32_t t,
                                            uint32_t& dlo, uint32_t& dn, uint32_t& dsel, uint32_t& jsel,
                                            uint32_t& jv, unsigned long long& bytes) {
  const DevGraph& g = p.g;
  const uint32_t nb = wp.nb(np), bm = wp.backmask(np);
  uint32_t best = 0xffffffffu, second = 0xffffffffu, dv = 0;
  jsel = 0; jv = 0;
  bool empty = false;
  unsigned long long b4 = 0;
#pragma unroll 1
  for (uint32_t end = nb; end > 0;) {
    const uint32_t beg = end > 4u ? end - 4u : 0u;
    uint32_t v[4] = {0, 0, 0, 0};
    auto visit = [&](uint32_t j, uint32_t u) {
      const uint32_t b = __popc(bm & ((1u << j) - 1u));
#pragma unroll
      for (uint32_t i = 0; i < 4; i++)
        if (b == beg + i && b < end) v[i] = u;
    };
    if (with_x && (bm >> (d + 1)) & 1u) visit((uint32_t)d + 1u, x);
    walk_prefix(lv, d, e, bm & ((2u << d) - 1u), visit);
    uint32_t lo[4], hi[4], tc[4], c[4];
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
      lo[i] = 0; hi[i] = 0; tc[i] = 0; c[i] = 0;
      if (beg + i < end) {
        c[i] = back_combo(wp.back(np, beg + i));
        const uint32_t* dir = g.dir + (size_t)v[i] * (g.nc + 1) + c[i];
        const uint32_t base = g.row[v[i]].x;
        lo[i] = base + dir[0];
        hi[i] = base + dir[1];
        tc[i] = g.t_count[v[i]];
      }
    }
#pragma unroll
    for (int i = 3; i >= 0; i--) {
      if (beg + (uint32_t)i < end) {
        const uint32_t sz = hi[i] - lo[i];
        const uint32_t szt = (tc[i] == 0 || sz == 0) ? sz : seg_size_slow(p, v[i], c[i], lo[i], hi[i], t);
        b4 += 4ull * szt;
        if (szt == 0) empty = true;
        if (sz <= best) {
          second = best; jsel = dsel & kSelMask; jv = dv;
          best = sz; dsel = (beg + (uint32_t)i) | (tc[i] ? kSelTouched : 0u); dv = v[i]; dlo = lo[i];
        } else if (sz <= second) {
          second = sz; jsel = beg + (uint32_t)i; jv = v[i];
        }
      }
    }
    end = beg;
  }
  dn = best;
  bytes = b4;
  return !empty;
}

// The survivors of level d (one a lane: candidate x of entry `own`, driver
// segment of `size` elements for the next position, 0: none) do not fit in one
// range together: the first ones that do stay, one at least.  Returns the first
// lane left out (32: none), and, in the upper half, the cursor of level d there.
// Cold: it takes rows of 2^27 entries.
__device__ __noinline__ unsigned long long range_refit(const uint32_t* pool, const LevelSM& S, uint32_t lane,
                                                       uint32_t size, uint32_t own, uint32_t x, uint32_t cur) {
  unsigned long long sum = size;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= (uint32_t)o) sum += v;
  }
  const uint32_t out = __ballot_sync(0xffffffffu, size && sum > kRangeMax && sum != size);
  if (!out) return 32ull | ((unsigned long long)cur << 32);
  const uint32_t first = (uint32_t)__ffs((int)out) - 1u;
  const uint32_t fx = __shfl_sync(0xffffffffu, x, first), fo = __shfl_sync(0xffffffffu, own, first);
  const uint32_t beg = S.base[fo] + (fo ? S.incl[fo - 1] : 0u), end = S.base[fo] + S.incl[fo];
  // a segment is sorted
  return first | ((unsigned long long)((uint32_t)lower_bound_u32(pool, beg, end, fx) - S.base[fo]) << 32);
}

// Per-task accumulators, flushed to the update's counters when the task ends;
// bytes are each lane's own until then.
struct TaskAcc {
  unsigned long long cnt, hash, bytes;
  uint32_t iters;
};

// Hands unexpanded work at the shallowest level with work left to idle warps:
// whole entries from the end of that level's buffer, or, when only the entry
// in progress is left, parts of its remaining driver range.  Each
// donated task is a partial match (positions 0..L) plus a driver range for
// position L + 1.
__device__ __noinline__ void donate(const SearchParams& p, LevelSM* lv, int d, uint32_t lane, uint32_t idle_now,
                                    uint32_t t, uint32_t anchor, uint32_t orient, int tail_level) {
  // Ranges are split down to two elements near the root (where every element
  // heads a large subtree) and only from 64 elements further down.  Lane L
  // looks at level L; the shallowest level that has something to give wins.
  const int n = (int)p.plan->n;
  const int me = (int)lane;
  uint32_t give = 0;  // 1: whole entries, 2: split the entry in progress
  if (me >= 1 && me <= d && me <= n - 2) {
    const LevelSM& S = lv[me];
    const uint32_t cnt = S.cnt, cur = S.cur, total = S.total;
    if (cur < total) {
      const uint32_t min_split = (me + 5 <= n) ? 2u : (p.split_deep ? p.split_deep : 64u);
      if (cnt >= 2 && cur < S.incl[cnt - 2]) give = 1;
      else if (me != tail_level && total - cur >= min_split) give = 2;  // the tail stage takes whole entries only
    }
  }
  const uint32_t who = __ballot_sync(0xffffffffu, give != 0);
  if (!who) {
    if (lane == 0) atomicAdd(&p.sstat->starved, 1ULL);
    return;
  }
  const int Ls = __ffs((int)who) - 1;
  const uint32_t mode = __shfl_sync(0xffffffffu, give, Ls);
  LevelSM& S = lv[Ls];
  const uint32_t cnt = S.cnt, cur = S.cur, total = S.total;
  // the entry in progress
  const uint32_t ce = __popc(__ballot_sync(0xffffffffu, lane < cnt && S.incl[lane] <= cur));
  // a range in progress is cut into up to 16 parts of at least half the
  // smallest range worth splitting; the first stays here
  const uint32_t floor_part = (Ls + 5 <= n) ? 1u : max(1u, (p.split_deep ? p.split_deep : 64u) / 2);
  const uint32_t avail = mode == 1 ? min(cnt - ce - 1, 32u) : min((total - cur) / floor_part - 1u, 15u);
  // take up to `avail` units of hunger (idle warps not yet promised a
  // record; a signed count): one subtraction, the excess given back, no
  // retries however many warps donate at once
  unsigned long long base = 0;
  uint32_t k = 0;
  if (lane == 0) {
    const uint32_t want = min(avail, idle_now);
    const int old = (int)atomicSub(&p.q->hungry, want);
    k = old <= 0 ? 0u : min((uint32_t)old, want);
    if (k < want) atomicAdd(&p.q->hungry, want - k);
    if (k) {
      atomicAdd(&p.q->pending, k);
      base = atomicAdd(&p.q->tail, (unsigned long long)k);
      atomicAdd(&p.sstat->donations, 1ULL);
    }
  }
  k = __shfl_sync(0xffffffffu, k, 0);
  if (k == 0) return;
  base = __shfl_sync(0xffffffffu, base, 0);
  // entry handed to lane j and its driver range
  uint32_t e = 0, dlo = 0, dn = 0;
  const uint32_t rem = total - cur;
  const uint32_t beg = (uint32_t)((unsigned long long)rem * (lane + 1u) / (k + 1u));  // part lane + 1 of k + 1
  const uint32_t end = (uint32_t)((unsigned long long)rem * (lane + 2u) / (k + 1u));
  const uint32_t keep = rem / (k + 1u);
  if (mode == 1) {
    e = cnt - k + lane;
    if (lane < k) {
      const uint32_t start = S.incl[e - 1];  // e > ce
      dlo = S.base[e] + start;
      dn = S.incl[e] - start;
    }
  } else {
    e = ce;
    dlo = S.base[ce] + cur + beg;
    dn = end - beg;
  }
  if (lane < k) {
    const unsigned long long ticket = base + lane;
    const uint32_t slot = (uint32_t)(ticket & (p.qcap - 1));
    // the slot is free for this ticket once its previous reader released it
    volatile unsigned long long* sq = p.qseq + slot;
    const unsigned long long t0 = global_ns();
    bool ok = true;
    while (*sq != ticket) {
      __nanosleep(64);
      if (global_ns() - t0 > p.slot_limit_ns) { atomicExch(p.error, kErrWaitTimeout); ok = false; break; }
    }
    DTask* D = p.dq + slot;
    uint32_t idx = e;
#pragma unroll 1
    for (int L = Ls; L >= 0; --L) {
      const LevelSM& X = lv[L ? L : 1];
      D->m[L] = X.v[idx];
      idx = X.par[idx];
    }
    D->upd = ok ? t : 0xffffffffu;  // a record that could not be placed is published as void
    D->anchor = (uint16_t)anchor; D->orient = (uint8_t)orient; D->depth = (uint8_t)Ls;
    D->dlo = dlo; D->dn = dn; D->sel = (uint32_t)S.dsel[e] | ((uint32_t)S.jsel[e] << 8);
    __threadfence();
    *sq = ticket + 1;  // publish
  }
  __syncwarp();
  if (lane == 0) {
    if (mode == 1) { S.cnt = cnt - k; S.total = S.incl[cnt - k - 1]; }
    else S.total = cur + keep;
  }
  __syncwarp();
}

// ---------------------------------------------------------------- tail stage

constexpr unsigned long long kTailSat = 1ULL << 58;  // a warp's sum of 32 saturated counts stays below 2^63

__device__ __forceinline__ unsigned long long sat_mul(unsigned long long a, unsigned long long b) {
  if (a == 0 || b == 0) return 0;
  return a > kTailSat / b ? kTailSat : min(kTailSat, a * b);
}

// Injective assignments of a label group of g <= kTailGroup tail positions,
// from N[M]: the number of candidates whose set of group members they are a
// candidate of is exactly M.  Members served by candidates of one class M
// form a subset R of M, in N[M] (N[M] - 1) ... (N[M] - |R| + 1) ways; a
// dynamic program over the set of served members.  Without injectivity
// (homo) it is the product of the members' candidate counts.  Saturates.
__device__ __noinline__ unsigned long long group_assignments(uint32_t g, const unsigned long long* N, int homo) {
  const uint32_t full = (1u << g) - 1u;
  if (homo) {
    unsigned long long prod = 1;
#pragma unroll 1
    for (uint32_t i = 0; i < g; i++) {
      unsigned long long c = 0;
#pragma unroll 1
      for (uint32_t M = 1; M <= full; M++)
        if ((M >> i) & 1u) c = min(kTailSat, c + N[M]);
      prod = sat_mul(prod, c);
    }
    return prod;
  }
  unsigned long long f[1u << kTailGroup], h[1u << kTailGroup];
  for (uint32_t S = 0; S <= full; S++) f[S] = S == 0 ? 1ull : 0ull;
#pragma unroll 1
  for (uint32_t M = 1; M <= full; M++) {
    if (!N[M]) continue;
    for (uint32_t S = 0; S <= full; S++) h[S] = 0;
#pragma unroll 1
    for (uint32_t S = 0; S <= full; S++) {
      if (!f[S]) continue;
      const uint32_t fr = M & ~S;
#pragma unroll 1
      for (uint32_t R = fr;; R = (R - 1u) & fr) {  // every subset of fr, the empty one last
        unsigned long long ways = 1;
#pragma unroll 1
        for (uint32_t r = 0, k = (uint32_t)__popc(R); r < k; r++) ways = sat_mul(ways, N[M] > r ? N[M] - r : 0ull);
        if (ways) h[S | R] = min(kTailSat, h[S | R] + sat_mul(f[S], ways));
        if (R == 0) break;
      }
    }
    for (uint32_t S = 0; S <= full; S++) f[S] = h[S];
  }
  return f[full];
}

// Counts the completions of the next LevelSM::burst entries of level L (= the
// anchor's tail_at: complete matches of the positions before the independent
// tail) and moves the level's cursor past them.  For each
// label group of the tail, every member's candidates are listed from its
// driver segment (32 (entry, element) pairs at a time, as in run_levels) and
// classified by the other members they are candidates of; a candidate is
// counted under the first member it belongs to, in per-entry class counters
// kept in the unused levels above L.  Each entry's completions are the
// product over groups of group_assignments.  A group is not looked at for
// entries whose product is already 0.  Not inlined: it runs once per 32 prefixes
// and would take registers from the walk.
struct TailOut {
  unsigned long long sum, bytes;  // completions (all lanes), bytes (this lane's)
  uint32_t iters;
  bool stopped;                   // the update was stopped (deadline or stop flag)
};
template <bool GEN>
__device__ __noinline__ TailOut tail_stage(const SearchParams& p, const uint32_t* pool, LevelSM* lv,
                                           const uint32_t* plan_words, uint32_t n, int L, uint32_t lane, uint32_t t,
                                           uint32_t anchor) {
  const PlanAnchor* A = &p.plan->anchors[anchor];
  const WalkPlan wp{plan_words, n};
  volatile unsigned int* stop = p.stop;
  LevelSM& S = lv[L];
  const uint32_t cnt = S.cnt, cur = S.cur;
  const uint32_t first = __popc(__ballot_sync(0xffffffffu, lane < cnt && S.incl[lane] <= cur));
  const uint32_t end = min(cnt, first + S.burst);
  const bool has = lane >= first && lane < end;
  const uint32_t e_mine = has ? lane : 0u;
  uint32_t* cntr = reinterpret_cast<uint32_t*>(&lv[L + 1]);  // [class][entry], levels L+1.. are unused here
  TailOut out{0, 0, 0, false};
  unsigned long long prod = has ? 1ull : 0ull;
  uint32_t gp = 0;
#pragma unroll 1
  for (uint32_t gi = 0; gi < A->n_groups; gi++) {
    const uint32_t g = A->gsize[gi];
    const uint32_t ncls = (1u << g) - 1u;
    for (uint32_t c = 0; c < ncls; c++) cntr[c * 32 + lane] = 0;
    __syncwarp();
    uint32_t done = 0;  // entries of member j taken so far, where they are taken one by one
#pragma unroll 1
    for (uint32_t j = 0; j < g && !out.stopped; j++) {
      const uint32_t ps = A->gpos[gp + j];
      uint32_t dlo = 0, dn = 0, dsel = 0, jsel = 0, jv = 0;
      if (prod) {
        if (ps == (uint32_t)L + 1) {  // the entry's own driver, found when it was pushed
          const uint32_t start = e_mine ? S.incl[e_mine - 1] : 0u;
          dlo = S.base[e_mine] + start; dn = S.incl[e_mine] - start; dsel = S.dsel[e_mine];
          jsel = S.jsel[e_mine]; jv = S.jv[e_mine];
        } else {
          unsigned long long b4 = 0;
          if (!pick_driver(p, lv, wp, L, e_mine, false, 0u, ps, (int32_t)t, dlo, dn, dsel, jsel, jv, b4)) dn = 0;
          if (!GEN || !done) out.bytes += b4;
        }
      }
      if (GEN && __any_sync(0xffffffffu, dn >= kRangeWide)) {  // not all in one range: member j again for every entry
        const uint32_t todo = __ballot_sync(0xffffffffu, dn != 0) & ~done, who = todo & (0u - todo);
        if (!((who >> lane) & 1u)) dn = 0;
        done = todo == who ? 0u : done | who;
      }
      const uint32_t incl = warp_incl_scan(dn, lane);
      const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
      for (uint32_t base = 0; base < total; base += 32) {
        if ((++out.iters & 63) == 0) {
          unsigned int st = 0;
          if (lane == 0) {
            if (p.deadline_ns && global_ns() - p.sstat->launch_t0 > p.deadline_ns)
              atomicCAS(const_cast<unsigned int*>(stop) + t, 0u, kStopDeadline);
            st = stop[t];
          }
          if (__shfl_sync(0xffffffffu, st, 0)) { out.stopped = true; break; }
        }
        const uint32_t gidx = base + lane;
        uint32_t owner = 0;
#pragma unroll
        for (uint32_t step = 16; step; step >>= 1) {
          const uint32_t v = __shfl_sync(0xffffffffu, incl, owner + step - 1);
          if (v <= gidx) owner += step;
        }
        const uint32_t own = owner & 31u;
        const uint32_t prev = __shfl_sync(0xffffffffu, incl, (owner - 1u) & 31u);
        const uint32_t o_dlo = __shfl_sync(0xffffffffu, dlo, own);
        const uint32_t o_sel = __shfl_sync(0xffffffffu, dsel | (jsel << 8), own);
        const uint32_t o_dsel = o_sel & 0xffu;
        const uint32_t o_jv = __shfl_sync(0xffffffffu, jv, own);
        if (gidx < total) {
          const uint32_t x = ld_stream(pool + (uint64_t)o_dlo + (gidx - (owner ? prev : 0u)));
          uint32_t joined = 0xffu, jhit = 0;
          bool ok = filter_bit(p, wp.qv(ps), x);
          if (ok && wp.nb(ps) > 1) {
            joined = o_sel >> 8;
            jhit = join_find<GEN>(p, pool, o_jv, wp.back(ps, joined), x);
            ok = jhit != kSlotEmpty;
          }
          if (ok && check_rest<GEN>(p, pool, lv, wp, L, owner, ps, x, o_dsel, joined, jhit, (int32_t)t)) {
            uint32_t M = 1u << j;
            bool seen = false;
#pragma unroll 1
            for (uint32_t i = 0; i < g && !seen; i++) {
              const uint32_t pi = A->gpos[gp + i];
              if (i == j || !filter_bit(p, wp.qv(pi), x) ||
                  !check_rest<GEN>(p, pool, lv, wp, L, owner, pi, x, kSelNone, 0xffu, 0u, (int32_t)t))
                continue;
              if (i < j) seen = true;
              else M |= 1u << i;
            }
            if (!seen) atomicAdd(&cntr[(M - 1u) * 32u + owner], 1u);
          }
        }
      }
      __syncwarp();
      if (GEN && done) j--;
    }
    gp += g;
    if (out.stopped) break;
    if (prod) {
      unsigned long long N[1u << kTailGroup];
      N[0] = 0;
      for (uint32_t c = 1; c <= ncls; c++) N[c] = cntr[(c - 1u) * 32u + lane];
      prod = sat_mul(prod, group_assignments(g, N, p.homo));
    }
    __syncwarp();
    if (!__any_sync(0xffffffffu, prod != 0)) break;
  }
  unsigned long long sum = prod;
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  out.sum = out.stopped ? 0ull : sum;
  __syncwarp();
  if (lane == 0) {
    S.cur = S.incl[end - 1];
    S.burst = min(32u, 2u * S.burst);
  }
  __syncwarp();
  return out;
}

// Result of update s once its search is done.
__device__ __forceinline__ void write_result(const ResultArgs& a, uint32_t s) {
  const UpdInfo u = a.info[s];
  csm_result r;
  r.pos = 0; r.neg = 0; r.hash = 0; r.work_bytes = 0; r.latency_ns = 0;
  r.status = CSM_ST_OK; r.safe = a.safe ? a.safe[s] : 1u;
  if ((u.flags & UF_INVALID) || !(u.flags & UF_VALID)) {
    r.status = (u.flags & UF_INVALID) ? CSM_ST_INVALID : CSM_ST_OK;  // vertex updates count nothing
    r.safe = 1;
  } else {
    unsigned long long c = __ldcg(a.count + s);
    if (a.cap && c >= a.cap) { c = a.cap; r.status = CSM_ST_CAPPED; }
    else if (a.stop && __ldcg(a.stop + s) == kStopDeadline) r.status = CSM_ST_TIMED_OUT;  // c is a lower bound
    if (u.flags & UF_ADD) r.pos = c; else r.neg = c;
    if (a.want_hash && r.status == CSM_ST_OK) r.hash = __ldcg(a.hash + s);
    r.work_bytes = (a.bytes ? __ldcg(a.bytes + s) : 0ull) + ((u.flags & UF_MUT) ? (unsigned long long)a.mut_bytes : 0ull);
  }
  if (a.stamp) r.latency_ns = global_ns() - a.stamp[0];
  a.out[s] = r;
}

// A warp's counters of one launch.
struct WarpStat {
  unsigned long long busy, idle, root, last_root, longest, iters, checks, hungry;
  unsigned long long began;  // start of the current task
};

// Depth-first walk over chunked levels starting at level `d` (see the file
// comment).  MODE 1 compiles the match-set append in, MODE 2 the tail stage;
// each is a separate instantiation so that the others keep their registers.
//
// What bounds a step is how many cache lines the SM can have in flight: its
// loads are scattered over the lanes, and with 24 warps of 80 registers the
// spilled ones swept through L1 with them and came back from L2.  Sixteen
// warps of 128 registers spill nothing but six words where tails are counted
// (12,000 -> 4,200 cycles a step, and the
// search of a 65,536-update batch on the 2^22-vertex stream 131 -> 68 ms).  So
// the common step -- no candidate survives -- reads little: the level's cursor
// and segment ends live in registers, the range layout of LevelSM needs no
// scan, the order of the joins is in shared memory (WalkPlan), and nothing of
// the prefix is touched before a candidate has passed its first join and the
// filter.  Those that have are few (1.4 of 30 a step there, in 70 % of the
// steps), and what they need next is a long chain of loads: they are gathered
// over the level's steps in `wait` (x; entry, touched bit of the first join)
// and go through it 32 at a time.
template <int MODE, bool GEN>
__device__ __forceinline__ void run_levels(const SearchParams& p, const uint32_t* pool, LevelSM* lv,
                                           const WalkPlan& wp, uint2* wait, int d, uint32_t lane, const Task& T,
                                           WarpStat& ws, TaskAcc& acc) {
  const uint32_t n = wp.n;
  const uint32_t t = T.upd;
  const DevGraph& g = p.g;
  volatile unsigned int* stop = p.stop;
  uint32_t iter = 0;
  constexpr bool EN = MODE == 1;
  const int tail_level = (MODE == 2 && p.tail && p.plan->anchors[T.anchor].tail_at) ? (int)p.plan->anchors[T.anchor].tail_at : -1;
  uint32_t seen_stop = 0, seen_hungry = 0;  // lane 0: flags loaded at the last check
  uint32_t hungry = 0;                      // idle warps seen
  const uint32_t every = p.donate_every ? p.donate_every : 1u;  // steps between hand-over checks (a power of two)
  bool enter = true;
  uint32_t cur = 0, total = 0, my_incl = 0, qv = 0, held = 0;
  bool joins = false;  // the next position has a join beside its driver
  const uint64_t* filter = nullptr;  // candidate filter of the level's next position
  // the pair of this lane at cur, loaded a step ahead: entry, candidate, and
  // the row of the entry's first join; `fresh` when they are cur's
  bool fresh = false;
  uint32_t own = 0, x = 0;
  uint2 jrow = make_uint2(0, 0);
  auto fetch = [&](uint32_t c) {
    const uint32_t at = c + lane;
    // bit i of `ends`: an entry ends before the pair of lane i
    const uint32_t end = my_incl - c;
    const uint32_t ends = __reduce_or_sync(0xffffffffu, end - 1u < 31u ? 1u << end : 0u);
    own = __popc(__ballot_sync(0xffffffffu, my_incl <= c)) + __popc(ends & (0xffffffffu >> (31u - lane)));
    if (at < total) {
      const LevelSM& L = lv[d];
      x = ld_stream(pool + (L.base[own] + at));
      if (joins && (!GEN || g.htab)) jrow = g.row[L.jv[own]];
    }
  };
  // a single update's own range is handed over at once, while every other warp
  // waits (its calls take 4 to 8 % less; in batches it only breaks up work)
  if (lane == 0 && p.dq && p.batch == 1 && lv[d].total > 32u)
    seen_hungry = (uint32_t)max((int)*(volatile unsigned int*)&p.q->hungry, 0);
  for (;;) {
    if (enter) {
      // the level's cursor and segment ends (lane e: entry e's)
      const LevelSM& L = lv[d];
      cur = L.cur;
      total = L.total;
      my_incl = lane < L.cnt ? L.incl[lane] : 0xffffffffu;
      qv = wp.qv((uint32_t)d + 1u);
      filter = p.d2 ? p.d2 + (uint64_t)qv * p.d2_words : nullptr;
      joins = wp.nb((uint32_t)d + 1u) > 1;
      enter = false;
      fresh = false;
    }
    ++iter;
    if ((iter & 63) == 0) {
      unsigned int quit = 0;
      if (lane == 0) {
        const unsigned long long now = global_ns();
        if (p.deadline_ns && now - p.sstat->launch_t0 > p.deadline_ns) {
          atomicCAS(const_cast<unsigned int*>(stop) + t, 0u, kStopDeadline);
          quit = 1;
        }
        if (now - ws.began > p.task_limit_ns) {
          quit = 1;
          atomicExch(p.error, kErrTaskGuard);
          if (atomicCAS(&p.sstat->guard_set, 0u, 1u) == 0u) {
            p.sstat->guard_d = (unsigned)d; p.sstat->guard_upd = t; p.sstat->guard_iters = iter;
#pragma unroll 1
            for (int L = 1; L <= d && L <= 16; L++) {
              p.sstat->guard_lv[4 * (L - 1) + 0] = lv[L].cnt;
              p.sstat->guard_lv[4 * (L - 1) + 1] = lv[L].cur;
              p.sstat->guard_lv[4 * (L - 1) + 2] = lv[L].total;
              p.sstat->guard_lv[4 * (L - 1) + 3] = lv[L].incl[0];
            }
          }
        }
      }
      if (__shfl_sync(0xffffffffu, quit, 0)) break;
    }
    // the stop flag and the idle-warp count are loaded every fourth step, each
    // a round trip to a line other warps update, and looked at a step later, so
    // that the trip overlaps a step; lane 0's view decides for the warp
    if ((iter & 3) == 1) {
      if (__shfl_sync(0xffffffffu, seen_stop, 0)) break;
      hungry = __shfl_sync(0xffffffffu, seen_hungry, 0);
    } else if ((iter & 3) == 0 && lane == 0) {
      seen_stop = stop[t];
      seen_hungry = p.dq ? (uint32_t)max((int)*(volatile unsigned int*)&p.q->hungry, 0) : 0u;
    }
    if (hungry && (iter & (every - 1)) == 0) {
      if (lane == 0) { lv[d].cur = cur; ws.hungry++; }
      __syncwarp();
      donate(p, lv, d, lane, hungry, t, T.anchor, T.orient, tail_level);
      total = lv[d].total;
      if (lane >= lv[d].cnt) my_incl = 0xffffffffu;
    }
    if constexpr (MODE == 2) {
      if (d == tail_level) {
        const TailOut r = tail_stage<GEN>(p, pool, lv, wp.w, n, d, lane, t, T.anchor);
        acc.bytes += r.bytes;
        acc.iters += r.iters;
        acc.cnt += r.sum;
        if (r.stopped) break;
        if (r.sum && p.cap) {
          unsigned int hit = 0;
          if (lane == 0) {
            const unsigned long long old = atomicAdd(&p.count[t], acc.cnt);
            if (old + r.sum >= p.cap) { stop[t] = kStopCap; hit = 1; }
          }
          acc.cnt = 0;
          if (__shfl_sync(0xffffffffu, hit, 0)) break;
        }
        cur = lv[d].cur;
        if (cur < total) continue;
      }
    }
    if (cur >= total) {  // level done (and none of its candidates waits)
      if (--d < 1) break;
      enter = true;
      continue;
    }
    acc.iters++;
    // the next 32 (entry, driver element) pairs of this level: the first join,
    // then the filter bit of those it leaves.  This order reads fewest lines:
    // on the 2^22-vertex stream the join leaves 7 % and the filter 66 %
    // (filter first 234 ms of search, join first 211 ms, both at once 268 ms).
    // The following pairs are fetched between the two.
    const uint32_t pos = (uint32_t)d + 1;
    if (!fresh) fetch(cur);
    const uint32_t cx = x;
    uint32_t meta = own;
    bool valid = cur + lane < total;
    if (valid && joins) {
      const uint32_t hit = !GEN || g.htab
                               ? row_find(g, jrow, row_entry(cx, lv[d].jel[own], g.hlb))
                               : join_search(p, pool, lv[d].jv[own], back_combo(wp.back(pos, lv[d].jsel[own])), cx);
      valid = hit != kSlotEmpty;
      meta |= (hit & kSlotTouched) >> 15;
    }
    fresh = cur + 32u < total;
    if (fresh) fetch(cur + 32u);
    if (valid && filter) valid = (ld_gather(filter + (cx >> 6)) >> (cx & 63u)) & 1ULL;
    // the candidates left wait until 32 of them, or all of the level's, are
    // together; a step that finds more than there is room for ends before the
    // first of those
    const uint32_t found = __ballot_sync(0xffffffffu, valid);
    if (found == 0 && (held == 0 || cur + 32u < total)) {
      cur += 32u;
      continue;
    }
    const uint32_t rank = held + __popc(found & ((1u << lane) - 1u));
    if (valid && rank < 32u) wait[rank] = make_uint2(cx, meta);
    held += __popc(found);
    cur += 32u;
    if (held > 32u) {
      cur += (uint32_t)__ffs((int)__ballot_sync(0xffffffffu, valid && rank >= 32u)) - 33u;
      held = 32u;
      fresh = false;
    }
    if (held == 0 || (held < 32u && cur < total)) continue;
    __syncwarp();
    // injectivity, remaining joins, presence, next driver
    uint32_t ndlo = 0, ndn = 0, ndsel = 0, njsel = 0, njv = 0;
    uint32_t wx = 0, wown = 0;
    unsigned long long nb4 = 0;
    valid = lane < held;
    if (valid) {
      const uint2 w = wait[lane];
      wx = w.x;
      wown = w.y & 31u;
      const uint32_t wsel = lv[d].dsel[wown];
      valid = check_rest<GEN>(p, pool, lv, wp, d, wown, pos, wx, wsel, joins ? lv[d].jsel[wown] : 0xffu,
                              (w.y << 15) & kSlotTouched, (int32_t)t);
      if (valid && pos + 1 < n) {
        valid = pick_driver(p, lv, wp, d, wown, true, wx, pos + 1, (int32_t)t, ndlo, ndn, ndsel, njsel, njv, nb4);
        if (!GEN) acc.bytes += nb4;
      }
    }
    held = 0;
    if constexpr (GEN) {
      if (__any_sync(0xffffffffu, ndn >= kRangeWide)) {  // a leaf has no segment
        const unsigned long long r = range_refit(pool, lv[d], lane, valid ? ndn : 0u, wown, wx, cur);
        if ((uint32_t)r < 32u) {  // the level goes on from the first one left out
          cur = (uint32_t)(r >> 32);
          fresh = false;
          valid = valid && lane < (uint32_t)r;
          if (lane >= (uint32_t)r) nb4 = 0;
        }
      }
      acc.bytes += nb4;
    }
    const uint32_t mask = __ballot_sync(0xffffffffu, valid);
    if (!mask) continue;
    if (pos == n - 1) {
      const uint32_t c = __popc(mask);
      if (EN) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(p.enum_n, (unsigned long long)c);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (valid) {
          const unsigned long long r = base + __popc(mask & ((1u << lane) - 1u));
          if (r < p.enum_cap) {
            uint32_t* rec = p.enum_buf + r * p.enum_stride;
            rec[0] = p.enum_base + t;
            rec[1 + qv] = wx;
            walk_prefix(lv, d, wown, (2u << d) - 1u, [&](uint32_t j, uint32_t v) { rec[1 + wp.qv(j)] = v; });
          }
        }
      }
      if (MODE != 2 && p.want_hash && valid) {
        uint64_t s = pair_hash(qv, wx);
        walk_prefix(lv, d, wown, (2u << d) - 1u, [&](uint32_t j, uint32_t v) { s += pair_hash(wp.qv(j), v); });
        acc.hash += mix64(s);
      }
      acc.cnt += c;
      if (p.cap) {
        unsigned int hit = 0;
        if (lane == 0) {
          const unsigned long long old = atomicAdd(&p.count[t], acc.cnt);
          if (old + c >= p.cap) { stop[t] = kStopCap; hit = 1; }
        }
        acc.cnt = 0;
        if (__shfl_sync(0xffffffffu, hit, 0)) break;
      }
    } else {
      // survivors become level pos, their driver segments laid end to end
      LevelSM& N = lv[pos];
      const uint32_t mine = valid ? ndn : 0u;
      const uint32_t incl = warp_incl_scan(mine, lane);
      if (valid) {
        const uint32_t slot = __popc(mask & ((1u << lane) - 1u));
        N.v[slot] = wx; N.par[slot] = (uint8_t)wown; N.dsel[slot] = (uint8_t)ndsel;
        N.jsel[slot] = (uint8_t)njsel; N.jel[slot] = (uint8_t)back_el(wp.back(pos + 1, njsel)); N.jv[slot] = njv;
        N.incl[slot] = incl; N.base[slot] = ndlo - (incl - mine);
      }
      if (lane == 31) { N.cnt = __popc(mask); N.cur = 0; N.total = incl; lv[d].cur = cur; }
      __syncwarp();
      d = (int)pos;
      enter = true;
    }
  }
  if (lane == 0 && p.dq) ws.checks += iter / every;
}

__device__ __forceinline__ void flush_acc(const SearchParams& p, uint32_t t, uint32_t lane, TaskAcc& acc) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    acc.bytes += __shfl_xor_sync(0xffffffffu, acc.bytes, o);
    if (p.want_hash) acc.hash += __shfl_xor_sync(0xffffffffu, acc.hash, o);
  }
  if (lane == 0) {
    if (acc.cnt) {
      const unsigned long long old = atomicAdd(&p.count[t], acc.cnt);
      if (p.cap && old + acc.cnt >= p.cap) p.stop[t] = kStopCap;
    }
    if (p.want_hash && acc.hash) atomicAdd(&p.hash[t], acc.hash);
    if (acc.bytes) atomicAdd(&p.bytes[t], acc.bytes);
  }
  acc.cnt = 0; acc.hash = 0; acc.bytes = 0;
  __syncwarp();
}

// Same-label positions the injectivity tests of this anchor's walk look at: all,
// or those before a counted tail (whose own vertices are told apart by their
// classes); none under homomorphism.
__device__ __forceinline__ uint32_t same_mask(const SearchParams& p, const PlanAnchor* A) {
  if (p.homo) return 0u;
  return p.tail ? A->prefix_mask : 0xffffffffu;
}

// Root task: positions 0 and 1 are the updated edge; level 1 holds the driver
// segment of position 2.  Returns false when there is nothing to walk.
struct RootOut {
  unsigned long long cnt, hash, bytes;  // of the whole (two-vertex) query; bytes of the first node
  bool walk;
};
template <int MODE>
__device__ __noinline__ RootOut setup_root(const SearchParams& p, LevelSM* lv, uint32_t* plan_words, uint32_t n,
                                           uint32_t lane, uint32_t t, uint32_t anchor, uint32_t orient) {
  RootOut out{0, 0, 0, false};
  const PlanAnchor* A = &p.plan->anchors[anchor];
  const UpdInfo U = p.info[t];
  const uint32_t m0 = orient ? U.v2 : U.v1, m1 = orient ? U.v1 : U.v2;
  if (n == 2) {
    out.cnt = 1;
    if (lane == 0) {
      if (p.want_hash) out.hash = mix64(pair_hash(A->pos[0].qv, m0) + pair_hash(A->pos[1].qv, m1));
      if (MODE == 1) {
        const unsigned long long r = atomicAdd(p.enum_n, 1ull);
        if (r < p.enum_cap) {
          uint32_t* rec = p.enum_buf + r * p.enum_stride;
          rec[0] = p.enum_base + t;
          rec[1 + A->pos[0].qv] = m0;
          rec[1 + A->pos[1].qv] = m1;
        }
      }
    }
    return out;
  }
  const PlanPos P2 = A->pos[2];
  uint32_t sz = 0xffffffffu, szt = 1, touched = 0;
  uint64_t lo = 0, hi = 0, run = kTempEmpty;
  if (lane < P2.nb) {
    const uint32_t j = A->back_pos[P2.boff + lane], c = A->back_combo[P2.boff + lane];
    const uint32_t v = j == 0 ? m0 : m1;
    segment(p.g, v, c, lo, hi);
    sz = (uint32_t)(hi - lo);
    touched = p.g.t_count[v];
    szt = sz;
    if (touched && sz) run = temporal_find(p.g, temporal_head(p.g, v, c));
  }
  // sizes at the update's time, a segment's touched entries by the whole warp: a
  // batch whose updates meet at one vertex has them all there, for every root
  // task (20,000 insertions at one vertex, then their deletions: 540 ms by one
  // lane a segment, 17 ms so)
  for (uint32_t todo = __ballot_sync(0xffffffffu, run != kTempEmpty); todo; todo &= todo - 1) {
    const uint32_t b = (uint32_t)__ffs((int)todo) - 1;
    const uint64_t r = __shfl_sync(0xffffffffu, run, b);
    const uint32_t beg = (uint32_t)r, end = beg + (uint32_t)(r >> 32);
    const int32_t absent = __reduce_add_sync(0xffffffffu, seg_absent(p.g, beg + lane, beg, end, 32, (int32_t)t));
    if (lane == b) szt = sz - (uint32_t)absent;
  }
  if (lane < P2.nb) out.bytes = 4ull * szt;
  if (__any_sync(0xffffffffu, szt == 0)) return out;
  uint64_t key = ((uint64_t)sz << 32) | lane;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    uint64_t other = __shfl_xor_sync(0xffffffffu, key, o);
    key = other < key ? other : key;
  }
  const uint32_t minsz = (uint32_t)(key >> 32), sel = (uint32_t)key;
  touched = __shfl_sync(0xffffffffu, touched, sel);
  const uint32_t other = sel == 0 ? 1u : 0u;  // position 2 has one back entry or two
  const uint32_t dlo0 = (uint32_t)__shfl_sync(0xffffffffu, lo, sel);
  if (lane == 0) {
    lv[1].cnt = 1; lv[1].cur = 0; lv[1].total = minsz;
    lv[1].incl[0] = minsz; lv[1].base[0] = dlo0;
    lv[1].dsel[0] = (uint8_t)(sel | (touched ? kSelTouched : 0u));
    lv[1].v[0] = m1; lv[1].par[0] = 1; lv[1].v[1] = m0;
    if (MODE == 2 && A->tail_at) lv[A->tail_at].burst = p.tail;
    lv[1].jsel[0] = (uint8_t)other;
    lv[1].jel[0] = P2.nb > 1 ? A->back_el[P2.boff + other] : 0;
    lv[1].jv[0] = P2.nb > 1 ? (A->back_pos[P2.boff + other] == 0 ? m0 : m1) : 0u;
  }
  load_walk_plan(plan_words, A, n, same_mask(p, A), lane);
  out.walk = true;
  return out;
}

// Donated task: rebuild the chain of the partial match (exhausted levels
// 1 .. depth-1) and continue from level `depth`.  `hw` holds record words
// 0..4 in lanes 0..4 and `mv` holds m[lane] (see DTask).  Returns the level
// to start from, 0 when there is nothing to walk.
struct DonatedOut {
  Task task;
  int depth;  // level to start from; 0: nothing to walk
};
__device__ __noinline__ DonatedOut setup_donated(const SearchParams& p, LevelSM* lv, uint32_t* plan_words, uint32_t n,
                                             uint32_t lane, uint32_t hw, uint32_t mv,
                                             unsigned long long ticket, unsigned long long seen_seq) {
  const uint32_t upd = __shfl_sync(0xffffffffu, hw, 0);
  const uint32_t w1 = __shfl_sync(0xffffffffu, hw, 1);
  const uint32_t dlo = __shfl_sync(0xffffffffu, hw, 2);
  const uint32_t dn = __shfl_sync(0xffffffffu, hw, 3);
  const uint32_t w4 = __shfl_sync(0xffffffffu, hw, 4), dsel = w4 & 0xffu;
  const uint32_t anchor = w1 & 0xffffu, orient = (w1 >> 16) & 0xffu, depth = w1 >> 24;
  DonatedOut out{Task{upd, (uint16_t)anchor, (uint8_t)orient, 0}, 0};
  if (upd == 0xffffffffu) return out;  // void record (its donor flagged an error)
  if (upd >= p.batch || anchor >= p.plan->n_anchor || depth < 1 || depth + 2 > n || depth > p.levels || dn == 0 ||
      (unsigned long long)dlo + dn > p.g.pool_cap) {
    if (lane == 0) {
      atomicExch(p.error, kErrBadTask);
      if (atomicCAS(&p.sstat->bad_set, 0u, 1u) == 0u) {
        p.sstat->bad_ticket = ticket; p.sstat->bad_seq = seen_seq; p.sstat->bad_batch = p.batch;
        p.sstat->bad_words[0] = upd; p.sstat->bad_words[1] = w1; p.sstat->bad_words[2] = dlo;
        p.sstat->bad_words[3] = dn; p.sstat->bad_words[4] = w4;
      }
    }
    out.task.upd = 0xffffffffu;
    return out;
  }
  const unsigned int stopped =
      __shfl_sync(0xffffffffu, lane == 0 ? *(volatile unsigned int*)(p.stop + upd) : 0u, 0);
  if (stopped) return out;
  const PlanAnchor* A = &p.plan->anchors[anchor];
  const uint32_t jsel = w4 >> 8;
  const PlanPos N = A->pos[depth + 1];
  const uint32_t jv = __shfl_sync(0xffffffffu, mv, N.nb > 1 ? A->back_pos[N.boff + min(jsel, N.nb - 1u)] : 0);
  if (lane >= 1 && lane <= depth) {
    LevelSM& S = lv[lane];
    S.cnt = 1; S.cur = 0; S.v[0] = mv; S.par[0] = lane == 1 ? 1 : 0;
    S.total = lane < depth ? 0u : dn;
    S.incl[0] = dn; S.base[0] = dlo; S.dsel[0] = (uint8_t)dsel;
    S.jsel[0] = (uint8_t)jsel; S.jel[0] = A->back_el[N.boff + min(jsel, N.nb - 1u)]; S.jv[0] = jv;
  }
  if (lane == 0) {
    lv[1].v[1] = mv;
    if (p.tail && A->tail_at) lv[A->tail_at].burst = p.tail;
  }
  load_walk_plan(plan_words, A, n, same_mask(p, A), lane);
  out.depth = (int)depth;
  return out;
}

// Kernel body; MODE 0 counts (and hashes), 1 also appends match sets, 2
// counts independent tails (tail_stage).
template <int W, int MODE, bool GEN>
__device__ __forceinline__ void search_body(const SearchParams& p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint4 task_scratch[W * 10];  // one 160-byte record per warp
  __shared__ uint2 waiting[W][32];         // candidates past their first join (run_levels)
  __shared__ WarpStat stats[W];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n = p.plan->n;
  unsigned char* mine = smem_raw + (size_t)warp * p.warp_bytes;
  LevelSM* lv = reinterpret_cast<LevelSM*>(mine) - 1;  // levels 1 .. p.levels
  uint32_t* plan_words = reinterpret_cast<uint32_t*>(mine + (size_t)p.levels * sizeof(LevelSM));
  const WalkPlan wp{plan_words, n};
  const uint32_t* pool = p.g.pools[p.g.ps->active];
  const uint32_t ntask = min(*p.n_tasks, p.task_cap);
  volatile unsigned int* stop = p.stop;
  volatile SearchQueue* q = p.q;
  WarpStat& ws = stats[warp];
  if (lane == 0) ws = WarpStat{};
  bool roots = ntask > 0;
  while (ntask) {
    TaskAcc acc{0, 0, 0, 0};
    Task T;
    int d = 0;
    unsigned long long tb = 0;
    const bool root = roots;
    if (roots) {
      // 1. root tasks, in claim order
      uint32_t ti = 0;
      if (lane == 0) ti = atomicAdd(p.task_next, 1u);
      ti = __shfl_sync(0xffffffffu, ti, 0);
      if (ti >= ntask) {
        roots = false;
        if (!p.dq) break;
        continue;
      }
      T = p.tasks[ti];
      tb = global_ns();
      if (lane == 0 && p.deadline_ns && tb - p.sstat->launch_t0 > p.deadline_ns)
        atomicCAS(const_cast<unsigned int*>(stop) + T.upd, 0u, kStopDeadline);
      // stop flags change under our feet: one lane reads, the warp follows it
      const unsigned int stopped = __shfl_sync(0xffffffffu, lane == 0 ? stop[T.upd] : 0u, 0);
      if (!stopped) {
        const RootOut r = setup_root<MODE>(p, lv, plan_words, n, lane, T.upd, T.anchor, T.orient);
        acc.cnt = r.cnt; acc.hash = r.hash; acc.bytes = r.bytes;
        d = r.walk ? 1 : 0;
      }
    } else {
      // 2. donated tasks until every task is done.  The queue is a bounded ring
      // of DTask slots with per-slot sequence numbers: slot (ticket % qcap) holds
      // ticket T's record once seq == T + 1, and is free for ticket T + qcap once
      // its reader stores seq = T + qcap.  Claims take a ticket by fetch-and-add:
      // a compare-and-swap on the head, retried by thousands of idle warps at
      // once, took most of the warps' time late in a batch.  A warp that finds
      // no task pending takes no ticket.
      unsigned long long claimed = ~0ULL, seen = 0;
      if (lane == 0 && q->pending != 0) {
        const unsigned long long t0 = global_ns();
        // this warp's ticket, and one unit of hunger for it: donors fill the
        // tickets in order, one per unit they take
        const unsigned long long tk = atomicAdd((unsigned long long*)&p.q->head, 1ull);
        atomicAdd(&p.q->hungry, 1u);
        unsigned int nap = 32;
        for (uint32_t poll = 0;; poll++) {
          const unsigned long long sv = *(volatile unsigned long long*)(p.qseq + (tk & (p.qcap - 1)));
          if (sv == tk + 1) { claimed = tk; seen = sv; break; }
          if ((poll & 3u) == 0 && q->pending == 0) break;  // the one word every waiting warp reads
          __nanosleep(nap);
          nap = min(nap * 2, 1024u);
          if (global_ns() - t0 > p.wait_limit_ns) { atomicExch(p.error, kErrWaitTimeout); break; }
        }
        ws.idle += global_ns() - t0;
      }
      claimed = __shfl_sync(0xffffffffu, claimed, 0);
      if (claimed == ~0ULL) break;
      // lane 0 copies the record through L2 (records share cache lines with other
      // slots) into the warp's scratch, and only then frees the slot for reuse
      uint4* scratch = task_scratch + warp * 10;
      if (lane == 0) {
        __threadfence();
        const uint32_t slot = (uint32_t)(claimed & (p.qcap - 1));
        const uint4* src = reinterpret_cast<const uint4*>(p.dq + slot);
#pragma unroll
        for (int i = 0; i < 10; i++) scratch[i] = __ldcg(src + i);
        __threadfence();
        *(volatile unsigned long long*)(p.qseq + slot) = claimed + p.qcap;
      }
      __syncwarp();
      const uint32_t* Dw = reinterpret_cast<const uint32_t*>(scratch);
      const uint32_t hw = lane < 5 ? Dw[lane] : 0u;
      const uint32_t mv = Dw[5 + lane];
      __syncwarp();
      tb = global_ns();
      const DonatedOut r = setup_donated(p, lv, plan_words, n, lane, hw, mv, claimed, seen);
      T = r.task;
      d = r.depth;
    }
    if (lane == 0) ws.began = tb;
    if (d > 0) run_levels<MODE, GEN>(p, pool, lv, wp, waiting[warp], d, lane, T, ws, acc);
    if (T.upd < p.batch) flush_acc(p, T.upd, lane, acc);
    if (lane == 0) {
      if (p.dq) atomicSub(&p.q->pending, 1u);
      const unsigned long long te = global_ns(), took = te - ws.began;
      ws.busy += took;
      ws.longest = max(ws.longest, took);
      if (root) { ws.root += took; ws.last_root = te; }
      ws.iters += acc.iters;
    }
    __syncwarp();
  }
  // one set of counter updates per block
  __syncthreads();
  if (threadIdx.x == 0) {
    WarpStat s{};
    for (int i = 0; i < W; i++) {
      s.busy += stats[i].busy; s.idle += stats[i].idle; s.root += stats[i].root;
      s.last_root = max(s.last_root, stats[i].last_root); s.longest = max(s.longest, stats[i].longest);
      s.iters += stats[i].iters; s.checks += stats[i].checks; s.hungry += stats[i].hungry;
    }
    if (s.busy) atomicAdd(&p.sstat->busy_ns, s.busy);
    if (s.idle) atomicAdd(&p.sstat->idle_ns, s.idle);
    if (s.root) atomicAdd(&p.sstat->root_busy_ns, s.root);
    if (s.last_root) atomicMax(&p.sstat->last_root_ns, s.last_root - p.sstat->launch_t0);
    if (s.longest) atomicMax(&p.sstat->max_task_ns, s.longest);
    if (s.iters) atomicAdd(&p.sstat->iters, s.iters);
    if (s.checks) atomicAdd(&p.sstat->checks, s.checks);
    if (s.hungry) atomicAdd(&p.sstat->checks_hungry, s.hungry);
  }
  // the results, by the block that ends last (small batches: SearchParams)
  if (p.result.out) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
      __threadfence();
      last = atomicAdd(p.ended, 1u) + 1u == gridDim.x;
      if (last) *p.ended = 0;
      __threadfence();
    }
    __syncthreads();
    if (last)
      for (uint32_t i = threadIdx.x; i < p.batch; i += W * 32) write_result(p.result, i);
  }
}

// Sixteen warps per SM, 128 registers a thread (run_levels says why).
constexpr int min_blocks(int w) { return w == 16 ? 1 : 16 / w; }

template <int W, bool EN>
__global__ void __launch_bounds__(W * 32, min_blocks(W)) k_search(const __grid_constant__ SearchParams p) {
  search_body<W, EN ? 1 : 0, false>(p);
}

template <int W>
__global__ void __launch_bounds__(W * 32, min_blocks(W)) k_search_tail(const __grid_constant__ SearchParams p) {
  search_body<W, 2, false>(p);
}

// Graphs without row tables or with very long rows (search_general): eight warps
// a block whatever is configured.
template <int MODE>
__global__ void __launch_bounds__(256, 2) k_search_general(const __grid_constant__ SearchParams p) {
  search_body<8, MODE, true>(p);
}

namespace {

using SearchKernel = void (*)(SearchParams);

template <int W>
SearchKernel search_kernel(int mode) {
  return mode == 2 ? k_search_tail<W> : mode == 1 ? k_search<W, true> : k_search<W, false>;
}

// mode: 0 plain, 1 match sets, 2 tail counting; `warps` is set to what the kernel takes
SearchKernel search_kernel(uint32_t& warps, int mode, bool general) {
  if (warps != 4 && warps != 16) warps = 8;
  if (general) {
    warps = 8;
    return mode == 2 ? k_search_general<2> : mode == 1 ? k_search_general<1> : k_search_general<0>;
  }
  return warps == 4 ? search_kernel<4>(mode) : warps == 16 ? search_kernel<16>(mode) : search_kernel<8>(mode);
}

// Lets a kernel take all of a block's shared memory that its own arrays leave.
// The limit is the kernel's, for every context of the device: set to a launch's
// own size, another thread's smaller query would lower it between setting and
// launch.
cudaError_t allow_shared(SearchKernel k, uint32_t warps) {
  constexpr uint32_t kBlock = 227 * 1024;
  const uint32_t own = warps * (uint32_t)(10 * sizeof(uint4) + 32 * sizeof(uint2) + sizeof(WarpStat)) + 64u;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kBlock - own));
}

}  // namespace

// Blocks of the search kernel that can be resident on one SM for walks of
// this shape (registers, shared memory and warp slots), from the
// occupancy API.  `mode` selects the instantiation: 0 plain counting (and hashes), 1 match
// sets, 2 tail counting.
uint32_t search_max_blocks(const SearchShape& shape, uint32_t warps, int mode) {
  const SearchKernel k = search_kernel(warps, mode, shape.general);
  const size_t smem = (size_t)shape.warp_bytes * warps;
  int nb = 0;
  cudaError_t e = allow_shared(k, warps);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, (int)warps * 32, smem);
  if (e != cudaSuccess) { cudaGetLastError(); return 0; }
  return (uint32_t)nb;
}

int search_mode(const SearchParams& p) { return p.enum_buf ? 1 : (p.tail ? 2 : 0); }

// A shape that does not fit fails to launch, which the caller's cudaGetLastError reports.
void launch_search(const SearchParams& p, uint32_t blocks, uint32_t warps, cudaStream_t s, bool prepared) {
  if (p.q && !prepared) k_search_prep<<<1, 1, 0, s>>>(p.q, p.n_tasks, p.task_cap, p.sstat, p.error);
  const SearchKernel k = search_kernel(warps, search_mode(p), search_general(p.g));
  const size_t smem = (size_t)p.warp_bytes * warps;
  if (allow_shared(k, warps) == cudaSuccess) k<<<blocks, warps * 32, smem, s>>>(p);
}

__global__ void k_finalize(uint32_t B, ResultArgs a) {
  uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < B) write_result(a, s);
}

__global__ void k_classify(uint64_t n, const csm_update* ups, DevGraph g, const Plan* plan, uint8_t* safe) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const csm_update u = ups[i];
  uint8_t sf = 1;
  if (u.id1 < g.n && u.id2 < g.n) {
    const uint32_t L1 = g.vlabel[u.id1], L2 = g.vlabel[u.id2];
    for (uint32_t a = 0; a < plan->n_anchor && sf; a++) {
      const PlanAnchor* A = &plan->anchors[a];
      const uint32_t el = fold_elabel(g, u.label);
      if (A->el == el && ((A->la == L1 && A->lb == L2) || (A->la == L2 && A->lb == L1))) sf = 0;
    }
  }
  safe[i] = sf;
}

}  // namespace csm
