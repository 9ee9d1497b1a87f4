// Candidate index of the TurboFlux / SymBi plugins (meaning and layout in
// csm_index.cuh).
//
// Kernels (all integer work, bound by L2/HBM latency of the segment reads):
//   k_ix_freq   query-edge frequencies and label counts that choose the root
//               (ParaCOSM/CSM/matching/SymBi/symbi.cpp:116-195)
//   k_ix_eval   evaluates every flag of one query vertex (index build)
//   k_ix_round  one round after edges or a vertex changed: marks the vertices
//               concerned (the reference's per-edge Insertion/Deletion
//               TopDown/BottomUp entry, symbi.cpp:679-735), re-evaluates marked
//               flags query vertex by query vertex in DAG order, and marks the
//               DAG-neighbour-side neighbours of vertices whose flag changed
//               (the Q1 / Q2 propagation loops, symbi.cpp:714-735)
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>

#include "csm_index.cuh"

namespace cg = cooperative_groups;

namespace csm {

namespace {

constexpr uint32_t kLaneScanMax = 48;  // entries a single lane scans before handing a vertex to the warp

__device__ __forceinline__ bool bit_of(const uint64_t* a, uint32_t v) { return (a[v >> 6] >> (v & 63)) & 1ULL; }

__device__ __forceinline__ uint64_t warp_or64(uint64_t x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x |= __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Does some neighbour w in segment [lo, hi) of the pool have flag[w]?  One lane.
__device__ __forceinline__ bool lane_support(const uint32_t* pool, uint64_t lo, uint64_t hi, const uint64_t* flag) {
  for (uint64_t k = lo; k < hi; k++)
    if (bit_of(flag, pool[k])) return true;
  return false;
}

// Entries of v in combo c (the union graph's segment during a batch).
__device__ __forceinline__ uint64_t seg_count(const DevGraph& g, uint32_t v, uint32_t c) {
  uint64_t lo, hi;
  segment(g, v, c, lo, hi);
  return hi - lo;
}

// The same over the whole warp (every lane must call it with equal arguments).
__device__ __forceinline__ bool warp_support(const uint32_t* pool, uint64_t lo, uint64_t hi, const uint64_t* flag,
                                             uint32_t lane) {
  for (uint64_t b = lo; b < hi; b += 32) {
    const uint64_t k = b + lane;
    const bool hit = k < hi && bit_of(flag, pool[k]);
    if (__any_sync(0xffffffffu, hit)) return true;
  }
  return false;
}

}  // namespace

// Per query edge (u < u' in adjacency order): directed entries v -> v' with
// L(v) = L(u), L(v') = L(u') and the edge's label = sum over v of L(u) of the
// segment size S(v, L(u'), l).  Also the number of vertices per folded label.
__global__ void k_ix_freq(DevGraph g, uint32_t ne, const uint32_t* __restrict__ ecombo,
                          const uint32_t* __restrict__ elab_u, unsigned long long* freq, unsigned long long* lcount) {
  __shared__ unsigned long long s_freq[kMaxQE];
  __shared__ unsigned long long s_lc[kMaxQ + 1];
  for (uint32_t i = threadIdx.x; i < ne; i += blockDim.x) s_freq[i] = 0;
  for (uint32_t i = threadIdx.x; i <= kMaxQ; i += blockDim.x) s_lc[i] = 0;
  __syncthreads();
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    const uint32_t lv = g.vlabel[v];
    if (lv == kNone) continue;
    if (lv <= kMaxQ) atomicAdd(&s_lc[lv], 1ull);
    const uint32_t* d = g.dir + (size_t)v * (g.nc + 1);
    for (uint32_t e = 0; e < ne; e++) {
      if (elab_u[e] != lv) continue;
      const uint32_t c = ecombo[e];
      const uint32_t sz = d[c + 1] - d[c];
      if (sz) atomicAdd(&s_freq[e], (unsigned long long)sz);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < ne; i += blockDim.x)
    if (s_freq[i]) atomicAdd(&freq[i], s_freq[i]);
  for (uint32_t i = threadIdx.x; i <= kMaxQ; i += blockDim.x)
    if (s_lc[i]) atomicAdd(&lcount[i], s_lc[i]);
}

// Does v keep its flag for query vertex u (phase 1: d1, phase 2: d2)?  One lane;
// `far` instead when a segment is too long for one.
__device__ __forceinline__ bool ix_lane_eval(const DevGraph& g, const uint32_t* pool, const IxDag* dag,
                                             const IxBits& b, uint32_t u, uint32_t phase, uint32_t v, bool& far) {
  const uint32_t nchk = phase == 1 ? dag->npar[u] : dag->nchd[u];
  const uint64_t* sup = (phase == 1 || dag->lighting) ? b.d1 : b.d2;
  const uint32_t nreq = (phase == 1 && dag->lighting) ? dag->nreq[u] : 0u;
  bool ok = phase == 1 ? g.vlabel[v] == dag->qlab[u] : bit_of(b.d1 + (uint64_t)u * b.words, v);
  for (uint32_t r = 0; r < nreq && ok; r++) ok = seg_count(g, v, dag->req_combo[u][r]) >= dag->req_mult[u][r];
  for (uint32_t s = 0; s < nchk && ok; s++) {
    const uint32_t q = phase == 1 ? dag->par[u][s] : dag->chd[u][s];
    uint64_t lo, hi;
    segment(g, v, phase == 1 ? dag->par_vcombo[u][s] : dag->chd_vcombo[u][s], lo, hi);
    if (hi - lo > kLaneScanMax) { far = true; break; }
    ok = lane_support(pool, lo, hi, sup + (uint64_t)q * b.words);
  }
  return ok;
}

// The same by a whole warp.  Lane s looks up segment s, all at once, and the
// first few entries of every segment are tried together; what that leaves open
// is scanned segment by segment.
__device__ __forceinline__ bool ix_warp_eval(const DevGraph& g, const uint32_t* pool, const IxDag* dag,
                                             const IxBits& b, uint32_t u, uint32_t phase, uint32_t v, uint32_t lane) {
  const uint32_t nchk = phase == 1 ? dag->npar[u] : dag->nchd[u];
  const uint64_t* sup = (phase == 1 || dag->lighting) ? b.d1 : b.d2;
  const uint32_t nreq = (phase == 1 && dag->lighting) ? dag->nreq[u] : 0u;
  bool ok = phase == 1 ? g.vlabel[v] == dag->qlab[u] : bit_of(b.d1 + (uint64_t)u * b.words, v);
  if (lane < nreq) ok = ok && seg_count(g, v, dag->req_combo[u][lane]) >= dag->req_mult[u][lane];
  uint64_t lo = 0, hi = 0;
  uint32_t q = 0;
  if (lane < nchk) {
    q = phase == 1 ? dag->par[u][lane] : dag->chd[u][lane];
    segment(g, v, phase == 1 ? dag->par_vcombo[u][lane] : dag->chd_vcombo[u][lane], lo, hi);
    ok = ok && lo < hi;
  }
  if (!__all_sync(0xffffffffu, ok)) return false;
  if (nchk == 0) return true;
  const uint32_t few = 32u / nchk;  // entries of each segment tried together; nchk <= 31
  const uint32_t s = lane / few, k = lane % few;
  const uint64_t slo = __shfl_sync(0xffffffffu, lo, s & 31u), shi = __shfl_sync(0xffffffffu, hi, s & 31u);
  const uint32_t sq = __shfl_sync(0xffffffffu, q, s & 31u);
  const bool hit = s < nchk && slo + k < shi && bit_of(sup + (uint64_t)sq * b.words, pool[slo + k]);
  const uint32_t found = __reduce_or_sync(0xffffffffu, hit ? 1u << s : 0u);
  const uint32_t over = __ballot_sync(0xffffffffu, lane < nchk && hi - lo <= few);  // wholly tried
  const uint32_t all = 0xffffffffu >> (32u - nchk);
  if (over & ~found) return false;
  for (uint32_t open = all & ~found; open; open &= open - 1) {
    const uint32_t i = (uint32_t)__ffs((int)open) - 1;
    const uint64_t* flag = sup + (uint64_t)__shfl_sync(0xffffffffu, q, i) * b.words;
    if (!warp_support(pool, __shfl_sync(0xffffffffu, lo, i) + few, __shfl_sync(0xffffffffu, hi, i), flag, lane))
      return false;
  }
  return true;
}

// Every flag of query vertex u from its definition (index build).  Each warp
// owns whole words of the target bitset, so its updates need no atomics.
__global__ void k_ix_eval(DevGraph g, const IxDag* __restrict__ dag, IxBits b, uint32_t u, uint32_t phase) {
  const uint32_t lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t* pool = g.pools[g.ps->active];
  const uint32_t lu = dag->qlab[u];
  const uint64_t off = (uint64_t)u * b.words;
  uint64_t* target = (phase == 1 ? b.d1 : b.d2) + off;
  for (uint64_t wi = warp; wi < b.words; wi += nwarps) {
    uint64_t cand;
    if (phase == 1) {
      const uint64_t v0 = wi * 64 + lane, v1 = v0 + 32;
      const bool a = v0 < g.n && g.vlabel[v0] == lu;
      const bool c = v1 < g.n && g.vlabel[v1] == lu;
      cand = (uint64_t)__ballot_sync(0xffffffffu, a) | ((uint64_t)__ballot_sync(0xffffffffu, c) << 32);
    } else {
      cand = b.d1[off + wi];
    }
    if (!cand) continue;
    // one candidate per lane (the j-th set bit goes to lane j % 32), then the
    // vertices with a long segment by the whole warp
    uint64_t mine = 0, defer = 0, rest = cand;
    for (uint32_t j = 0; rest; j++) {
      const uint32_t bitpos = (uint32_t)(__ffsll((long long)rest) - 1);
      rest &= rest - 1;
      if ((j & 31) != lane) continue;
      bool far = false;
      const bool ok = ix_lane_eval(g, pool, dag, b, u, phase, (uint32_t)(wi * 64 + bitpos), far);
      if (far) defer |= 1ull << bitpos;
      else if (ok) mine |= 1ull << bitpos;
    }
    uint64_t bits = warp_or64(mine);
    defer = warp_or64(defer);
    for (; defer; defer &= defer - 1) {
      const uint32_t bitpos = (uint32_t)(__ffsll((long long)defer) - 1);
      if (ix_warp_eval(g, pool, dag, b, u, phase, (uint32_t)(wi * 64 + bitpos), lane)) bits |= 1ull << bitpos;
    }
    if (lane == 0) target[wi] = bits;
    __syncwarp();
  }
}

// Marks v for re-evaluation of its d1 (phase 1) or d2 (phase 2) flag of u.
__device__ __forceinline__ void ix_mark(const IxBits& b, uint32_t nq, uint32_t phase, uint32_t u, uint32_t v) {
  const uint64_t bit = 1ull << (v & 63);
  uint64_t* word = (phase == 1 ? b.m1 : b.m2) + (uint64_t)u * b.words + (v >> 6);
  if (atomicOr((unsigned long long*)word, bit) & bit) return;
  const uint32_t row = (phase == 1 ? 0u : nq) + u;
  const uint32_t i = atomicAdd(&b.count[row], 1u);
  if (i < b.list_cap) b.list[(size_t)row * b.list_cap + i] = v;
}

// Marks for DAG edge e and the changed directed entry k = x -> y (combo = (L(y),
// l)), when its labels are the edge's: y for d1 of the child, x for d2 of the
// parent.  The reverse entry y -> x covers the other orientation.
__device__ __forceinline__ void ix_seed(const DevGraph& g, const IxDag* dag, const IxBits& b, uint64_t k,
                                        uint32_t lx, uint32_t e) {
  const uint32_t c = g.kb.c_of(k);
  if (dag->eel[e] != c % g.n_el) return;
  const uint32_t p = dag->ep[e], ch = dag->ec[e];
  if (dag->qlab[p] != lx || dag->qlab[ch] != c / g.n_el) return;
  ix_mark(b, dag->nq, 1, ch, g.kb.y_of(k));
  ix_mark(b, dag->nq, 2, p, g.kb.x_of(k));
}

// Re-evaluates u's flag of vertex v in each lane with `has` (their marks are
// taken off here), and marks what depends on the flags that changed.
__device__ __forceinline__ void ix_items(const DevGraph& g, const uint32_t* pool, const IxDag* dag,
                                         const IxBits& b, uint32_t u, uint32_t phase, bool has, uint32_t v,
                                         bool by_lane, uint32_t lane) {
  const uint64_t off = (uint64_t)u * b.words;
  const uint64_t bit = 1ull << (v & 63);
  unsigned long long* target = (unsigned long long*)((phase == 1 ? b.d1 : b.d2) + off + (v >> 6));
  bool ok = false, far = !by_lane;
  if (has && by_lane) ok = ix_lane_eval(g, pool, dag, b, u, phase, v, far);
  for (uint32_t todo = __ballot_sync(0xffffffffu, has && far); todo; todo &= todo - 1) {
    const uint32_t l = (uint32_t)__ffs((int)todo) - 1;
    const bool r = ix_warp_eval(g, pool, dag, b, u, phase, __shfl_sync(0xffffffffu, v, l), lane);
    if (l == lane) ok = r;
  }
  bool changed = false;
  if (has) {
    atomicAnd((unsigned long long*)((phase == 1 ? b.m1 : b.m2) + off + (v >> 6)), ~bit);
    changed = ((*target & bit) != 0) != ok;  // no other lane has this vertex
    if (changed) atomicXor(target, bit);
    if (changed && phase == 1) ix_mark(b, dag->nq, 2, u, v);
  }
  // phase 1: the d1 of u's children (their d2 in lighting mode) over v's
  // neighbours; phase 2: the d2 of u's parents
  if (phase == 2 && dag->lighting) return;
  const uint32_t n_to = phase == 1 ? dag->nchd[u] : dag->npar[u];
  const uint32_t to_phase = (phase == 2 || dag->lighting) ? 2u : 1u;
  for (uint32_t todo = __ballot_sync(0xffffffffu, changed); todo; todo &= todo - 1) {
    const uint32_t w = __shfl_sync(0xffffffffu, v, (uint32_t)__ffs((int)todo) - 1);
    for (uint32_t s = 0; s < n_to; s++) {
      const uint32_t q = phase == 1 ? dag->chd[u][s] : dag->par[u][s];
      uint64_t lo, hi;
      segment(g, w, phase == 1 ? dag->chd_vcombo[u][s] : dag->par_vcombo[u][s], lo, hi);
      for (uint64_t k = lo + lane; k < hi; k += 32) ix_mark(b, dag->nq, to_phase, q, pool[k]);
    }
  }
}

// One incremental round in a single cooperative launch (every block resident),
// for the changed directed entries keys[0, L) and, when it is not kNone, the
// new or removed vertex `vert`.  The marks come first; then, step by step of
// the order, the flags on the work lists of the step's query vertices, d1
// before d2.  Query vertices that do not draw on one another's flags share a
// step, and steps of empty lists are passed over.  What bounds a round is the
// number of grid barriers and the chain of loads between two, so the marks of a
// few entries and every run of steps of at most kAlone vertices are worked off by
// block 0 alone, with barriers of the block, while the others wait at one grid
// barrier; after it they go on with the step that block 0 left (b.count[2 nq]).
// For one edge update of a 13-vertex query on 2^19 vertices 52 barriers over
// whole bitsets took 153 us, a barrier per step with work 28 us, block 0 alone
// 18.7 us (a batch of 100: 289, 78 and 71 us).
//
// All blocks take the same way: a list's length is final when the last step
// that can mark it is done, and it is taken back only by block 0 after a barrier
// from which on nobody asks for it.
// Two vertices a warp.  Two batches of 100: 8 0.73 ms, 32 0.69, 128 0.72; single
// updates do not tell them apart.
constexpr uint32_t kAlone = 32;

// Do the marks of L entries and ne DAG edges keep no more than these threads busy?
__host__ __device__ constexpr bool ix_few(uint32_t L, uint32_t ne, uint32_t threads) { return (uint64_t)L * ne <= threads; }
static_assert(ix_few(2, 256, 512) && !ix_few(3, 256, 512), "the limit itself");
static_assert(!ix_few(1u << 24, 256, 512), "a vertex of 2^23 edges under a query of 256: the product passes 32 bits");

__global__ void __launch_bounds__(512) k_ix_round(DevGraph g, const IxDag* __restrict__ gdag, IxBits b, IxOrder ord,
                                                  const uint64_t* __restrict__ keys, uint32_t L, uint32_t vert) {
  cg::grid_group grid = cg::this_grid();
  __shared__ __align__(16) IxDag sdag;  // every step's chain of loads starts in it
  __shared__ uint32_t scount[2 * kMaxQ];
  for (uint32_t i = threadIdx.x; i < sizeof(IxDag) / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(&sdag)[i] = reinterpret_cast<const uint32_t*>(gdag)[i];
  __syncthreads();
  const IxDag* dag = &sdag;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t ne = dag->n_edges, nq = dag->nq;
  const uint32_t* pool = g.pools[g.ps->active];
  const uint32_t steps1 = ord.steps[0], steps = steps1 + ord.steps[1];
  const bool first = blockIdx.x == 0;
  bool alone = ix_few(L, ne, blockDim.x);  // block 0 works, the others wait
  uint32_t from = 0;                  // block 0: first step whose lists' lengths are to be taken back
  if (!alone || first) {
    const uint32_t tid = (alone ? 0u : blockIdx.x * blockDim.x) + threadIdx.x;
    const uint32_t nthreads = alone ? blockDim.x : gridDim.x * blockDim.x;
    if (L <= 64) {  // a thread per (entry, DAG edge)
      for (uint32_t i = tid; i < L * ne; i += nthreads) {
        const uint64_t k = keys[i / ne];
        if (g.kb.real(k)) ix_seed(g, dag, b, k, g.vlabel[g.kb.x_of(k)], i % ne);
      }
    } else {
      for (uint32_t i = tid; i < L; i += nthreads) {
        const uint64_t k = keys[i];
        if (!g.kb.real(k)) continue;
        const uint32_t lx = g.vlabel[g.kb.x_of(k)];
        for (uint32_t e = 0; e < ne; e++) ix_seed(g, dag, b, k, lx, e);
      }
    }
    if (vert != kNone && tid < nq) {
      ix_mark(b, nq, 1, tid, vert);
      ix_mark(b, nq, 2, tid, vert);
    }
    if (alone) { __threadfence(); __syncthreads(); }
  }
  if (!alone) grid.sync();
  for (uint32_t s = 0;;) {
    if (alone && !first) {
      grid.sync();
      alone = false;
      s = *(volatile unsigned int*)&b.count[2 * nq];
      if (s == steps) break;
    }
    if (threadIdx.x < 2 * nq) scount[threadIdx.x] = *(volatile unsigned int*)&b.count[threadIdx.x];
    __syncthreads();
    uint32_t n_step = 0, phase = 1, beg = 0, end = 0;
    for (; s < steps; s++) {
      phase = s < steps1 ? 1u : 2u;
      const uint32_t t = phase == 1 ? s : s - steps1;
      beg = t ? ord.end[phase - 1][t - 1] : 0u;
      end = ord.end[phase - 1][t];
      for (uint32_t i = beg; i < end; i++) n_step += scount[(phase == 1 ? 0u : nq) + ord.order[phase - 1][i]];
      if (n_step) break;
    }
    if (alone) {  // block 0
      if (n_step == 0 || n_step > kAlone) {
        if (threadIdx.x == 0) *(volatile unsigned int*)&b.count[2 * nq] = s;
        grid.sync();
        alone = false;
        for (uint32_t r = from; r < s; r++) {
          const uint32_t ph = r < steps1 ? 0u : 1u, t = ph ? r - steps1 : r;
          const uint32_t i = (t ? ord.end[ph][t - 1] : 0u) + threadIdx.x;
          if (i < ord.end[ph][t]) b.count[ph * nq + ord.order[ph][i]] = 0;
        }
        if (n_step == 0) break;
      }
    } else if (n_step == 0) {
      break;
    } else if (n_step <= kAlone) {
      alone = true;
      from = s;
      if (!first) continue;
    }
    const uint32_t warp = (alone ? 0u : blockIdx.x * (blockDim.x >> 5)) + (threadIdx.x >> 5);
    const uint32_t nwarps = (alone ? 1u : gridDim.x) * (blockDim.x >> 5);
    uint32_t used = 0;  // warps' shares given out in this step so far: the next list starts with the next warp
    for (uint32_t i = beg; i < end; i++) {
      const uint32_t u = ord.order[phase - 1][i];
      const uint32_t row = (phase == 1 ? 0u : nq) + u;
      const uint32_t n = scount[row];
      if (n == 0) continue;
      const uint32_t w0 = (warp + nwarps - used % nwarps) % nwarps;
      if (n <= b.list_cap) {
        // as many items per warp as it takes to share them out; with several,
        // each lane first tries its own
        const uint32_t* list = b.list + (size_t)row * b.list_cap;
        const uint32_t per = min(32u, (n + nwarps - 1) / nwarps);
        for (uint32_t base = w0 * per; base < n; base += nwarps * per) {
          const bool has = lane < per && base + lane < n;
          ix_items(g, pool, dag, b, u, phase, has, has ? __ldcg(list + base + lane) : 0u, per > 4, lane);
        }
        used += (n + per - 1) / per;
      } else {
        const uint64_t* mark = (phase == 1 ? b.m1 : b.m2) + (uint64_t)u * b.words;
        for (uint64_t wi = w0; wi < b.words; wi += nwarps) {
          const uint64_t word = __ldcg(mark + wi);
          if (!word) continue;
#pragma unroll 1
          for (uint32_t half = 0; half < 2; half++)
            ix_items(g, pool, dag, b, u, phase, (word >> (32u * half + lane)) & 1ULL,
                     (uint32_t)(wi * 64 + 32u * half + lane), true, lane);
        }
        used += nwarps;
      }
    }
    if (alone) {
      __threadfence();
      __syncthreads();
    } else {
      grid.sync();
      const uint32_t i = beg + threadIdx.x;
      if (first && i < end) b.count[(phase == 1 ? 0u : nq) + ord.order[phase - 1][i]] = 0;
    }
    s++;
  }
}

__global__ void k_ix_popcount(const uint64_t* a, uint64_t n, unsigned long long* out) {
  unsigned long long s = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    s += (unsigned long long)__popcll(a[i]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, s);
}

// ------------------------------------------------------------------ host

namespace {

#define IXCK(x)                                                                              \
  do {                                                                                       \
    cudaError_t e_ = (x);                                                                    \
    if (e_ != cudaSuccess) return set_err(CSM_ECUDA, "%s: %s", #x, cudaGetErrorString(e_)); \
  } while (0)

// Work-list entries per query vertex and phase: 2 |V_Q| lists of 128 KB are a
// small part of the bitsets of a large graph, and a batch of 65,536 updates
// marks fewer vertices (a list that overflows is worked off from its marks).
constexpr uint32_t kListCap = 32768;

constexpr uint32_t kListCapSmall = 64;

// Words of a flag bitset: 32-byte aligned rows.
uint64_t index_words(uint32_t n_cap) { return (((uint64_t)n_cap + 63) / 64 + 3) & ~3ull; }

// An index's arrays.
void index_block(IndexState& ix, DevBlock& blk, uint32_t nq, uint32_t n_cap, uint32_t list_cap) {
  ix.bits.list_cap = std::min<uint32_t>(n_cap, list_cap);
  blk.add(ix.bits.d1, 32ull * nq * index_words(n_cap));
  blk.add(ix.d_dag, sizeof(IxDag));
  blk.add(ix.d_pop, 16);
  blk.add(ix.bits.list, 4ull * 2 * nq * ix.bits.list_cap);
  blk.add(ix.bits.count, 8ull * nq + 4);
}

// Root choice (ParaCOSM/CSM/matching/SymBi/symbi.cpp:116-195, identical in
// TurboFlux/turboflux.cpp:82-149): the first query edge (u < u', adjacency
// order) of least frequency; of its endpoints the one whose label is rarer in
// the data graph, ties to the larger query degree, then to the second one.
uint32_t choose_root(const IndexQuery& q, const std::vector<std::pair<uint32_t, uint32_t>>& edges,
                     const std::vector<unsigned long long>& freq, const std::vector<unsigned long long>& lcount) {
  size_t best = 0;
  for (size_t i = 1; i < edges.size(); i++)
    if (freq[i] < freq[best]) best = i;
  const uint32_t a = edges[best].first, b = edges[best].second;
  const auto& ql = *q.vlabels;
  const unsigned long long ca = ql[a] <= kMaxQ ? lcount[ql[a]] : 0, cb = ql[b] <= kMaxQ ? lcount[ql[b]] : 0;
  if (ca > cb) return b;
  if (ca < cb) return a;
  return (*q.nbr)[a].size() > (*q.nbr)[b].size() ? a : b;
}

}  // namespace

// The full first evaluation: per query vertex in DAG order d1, in reverse d2.
static int index_launch_build(IndexState& ix, const DevGraph& g, cudaStream_t st, uint64_t* launches) {
  const uint32_t nq = ix.h_dag.nq;
  const uint64_t warps_needed = std::max<uint64_t>(ix.words, 1);
  const uint32_t blocks = (uint32_t)std::min<uint64_t>((warps_needed + 7) / 8, (uint64_t)ix.sm_count * 8);
  for (uint32_t i = 0; i < 2 * nq; i++) {
    const uint32_t phase = i < nq ? 1u : 2u;
    k_ix_eval<<<blocks, 256, 0, st>>>(g, ix.d_dag, ix.bits, ix.order[phase == 1 ? i : 2 * nq - 1 - i], phase);
    (*launches)++;
  }
  IXCK(cudaGetLastError());
  return CSM_OK;
}

// DAG of the TurboFlux / SymBi plugin: root from the device edge frequencies,
// then the SymBi BFS orientation or the TurboFlux spanning tree.
static int dag_for(const IndexQuery& q, const DevGraph& g, int algo,
                   const std::vector<std::pair<uint32_t, uint32_t>>& edges, const std::vector<uint32_t>& e_lab,
                   int sm_count, DevMem& mem, cudaStream_t st, uint64_t* launches, uint32_t& root,
                   std::vector<std::vector<uint32_t>>& par, std::vector<std::vector<uint32_t>>& chd,
                   std::vector<std::vector<uint32_t>>& par_l, std::vector<std::vector<uint32_t>>& chd_l,
                   std::vector<uint32_t>& order) {
  const uint32_t nq = q.n;
  const auto& ql = *q.vlabels;
  const auto& nbr = *q.nbr;
  const auto& el = *q.elabel;
  const uint32_t ne = (uint32_t)edges.size();
  // frequencies on the device
  std::vector<uint32_t> h_ec(ne), h_el(ne);
  for (uint32_t i = 0; i < ne; i++) {
    h_ec[i] = ql[edges[i].second] * g.n_el + e_lab[i];
    h_el[i] = ql[edges[i].first];
  }
  uint32_t* d_e = nullptr;
  unsigned long long* d_f = nullptr;
  DevBlock blk;
  blk.add(d_e, 8ull * ne);
  blk.add(d_f, 8ull * (ne + kMaxQ + 1));
  void* tmp = nullptr;
  const int rc = blk.alloc(mem, &tmp);
  if (rc) return rc;
  IXCK(cudaMemcpyAsync(d_e, h_ec.data(), 4ull * ne, cudaMemcpyHostToDevice, st));
  IXCK(cudaMemcpyAsync(d_e + ne, h_el.data(), 4ull * ne, cudaMemcpyHostToDevice, st));
  IXCK(cudaMemsetAsync(d_f, 0, 8ull * (ne + kMaxQ + 1), st));
  k_ix_freq<<<sm_count * 4, 256, 0, st>>>(g, ne, d_e, d_e + ne, d_f, d_f + ne);
  (*launches)++;
  IXCK(cudaGetLastError());
  std::vector<unsigned long long> freq(ne + kMaxQ + 1);
  IXCK(cudaMemcpyAsync(freq.data(), d_f, 8ull * (ne + kMaxQ + 1), cudaMemcpyDeviceToHost, st));
  IXCK(cudaStreamSynchronize(st));
  mem.release(tmp, blk.total);
  std::vector<unsigned long long> lcount(freq.begin() + ne, freq.end());
  freq.resize(ne);
  root = choose_root(q, edges, freq, lcount);

  // the DAG: parents / children with edge labels
  auto ffreq = [&](uint32_t a, uint32_t b) {
    const uint32_t x = std::min(a, b), y = std::max(a, b);
    for (uint32_t i = 0; i < ne; i++)
      if (edges[i].first == x && edges[i].second == y) return freq[i];
    return 0ull;
  };
  auto qlabel_of = [&](uint32_t a, uint32_t b) {
    auto it = std::lower_bound(nbr[a].begin(), nbr[a].end(), b);
    return el[a][(size_t)(it - nbr[a].begin())];
  };
  if (algo == CSM_ALGO_SYMBI) {
    // BFS from the root over every query edge; an edge points from the
    // endpoint dequeued first (symbi.cpp:197-238)
    std::vector<char> seen(nq, 0), popped(nq, 0);
    order.push_back(root);
    seen[root] = 1;
    for (size_t h = 0; h < order.size(); h++) {
      const uint32_t u = order[h];
      popped[u] = 1;
      for (size_t i = 0; i < nbr[u].size(); i++) {
        const uint32_t w = nbr[u][i];
        if (!seen[w]) { seen[w] = 1; order.push_back(w); }
        if (!popped[w]) {
          chd[u].push_back(w); chd_l[u].push_back(el[u][i]);
          par[w].push_back(u); par_l[w].push_back(el[u][i]);
        }
      }
    }
  } else {
    // spanning tree grown level by level, cheapest pending edge first, other
    // pending edges into the chosen vertex dropped (turboflux.cpp:151-219)
    struct EF { uint32_t a, b; unsigned long long f; };
    std::vector<char> vis(nq, 0);
    vis[root] = 1;
    std::vector<EF> cur;
    for (uint32_t w : nbr[root]) cur.push_back({root, w, ffreq(root, w)});
    while (!cur.empty()) {
      std::vector<EF> next;
      while (!cur.empty()) {
        size_t best = 0;
        for (size_t i = 1; i < cur.size(); i++) if (cur[i].f < cur[best].f) best = i;
        const EF m = cur[best];
        std::vector<EF> keep;
        for (const EF& e : cur) if (e.b != m.b) keep.push_back(e);
        cur.swap(keep);
        if (vis[m.b]) continue;
        vis[m.b] = 1;
        const uint32_t l = qlabel_of(m.a, m.b);
        chd[m.a].push_back(m.b); chd_l[m.a].push_back(l);
        par[m.b].push_back(m.a); par_l[m.b].push_back(l);
        for (uint32_t w : nbr[m.b]) if (!vis[w]) next.push_back({m.b, w, ffreq(m.b, w)});
      }
      cur.swap(next);
    }
    order.push_back(root);
    for (size_t h = 0; h < order.size(); h++)
      for (uint32_t w : chd[order[h]]) order.push_back(w);
  }
  return CSM_OK;
}


// Device DAG, flag bitsets and the full first evaluation.
static int index_finish(IndexState& ix, DevMem& mem, const DevGraph& g, const IndexQuery& q, int algo, uint32_t root,
                        const std::vector<uint32_t>& order, const std::vector<std::vector<uint32_t>>& par,
                        const std::vector<std::vector<uint32_t>>& chd, const std::vector<std::vector<uint32_t>>& par_l,
                        const std::vector<std::vector<uint32_t>>& chd_l, cudaStream_t st, uint64_t* launches) {
  const uint32_t nq = q.n;
  const auto& ql = *q.vlabels;
  int rc = CSM_OK;
  IxDag& D = ix.h_dag;
  memset(&D, 0, sizeof(D));
  D.nq = nq;
  for (uint32_t u = 0; u < nq; u++) D.qlab[u] = ql[u];
  for (uint32_t u = 0; u < nq; u++) {
    D.npar[u] = (uint32_t)par[u].size();
    D.nchd[u] = (uint32_t)chd[u].size();
    for (size_t i = 0; i < par[u].size(); i++) {
      const uint32_t p = par[u][i], l = par_l[u][i];
      D.par[u][i] = (uint8_t)p;
      D.par_vcombo[u][i] = (uint16_t)(ql[p] * g.n_el + l);
    }
    for (size_t i = 0; i < chd[u].size(); i++) {
      const uint32_t c = chd[u][i], l = chd_l[u][i];
      D.chd[u][i] = (uint8_t)c;
      D.chd_vcombo[u][i] = (uint16_t)(ql[c] * g.n_el + l);
      D.ep[D.n_edges] = (uint8_t)u; D.ec[D.n_edges] = (uint8_t)c; D.eel[D.n_edges] = (uint16_t)l;
      D.n_edges++;
    }
  }
  if (algo == CSM_ALGO_CALIG || algo == CSM_ALGO_NEWSP) {
    // d1 requirements: per (vertex label, edge label) pair of u's query
    // edges, as many neighbours as u has of that pair (one under homo)
    D.lighting = 1;
    for (uint32_t u = 0; u < nq; u++)
      for (size_t i = 0; i < chd[u].size(); i++) {
        const uint16_t combo = D.chd_vcombo[u][i];
        uint32_t r = 0;
        while (r < D.nreq[u] && D.req_combo[u][r] != combo) r++;
        if (r == D.nreq[u]) { D.req_combo[u][r] = combo; D.req_mult[u][r] = 0; D.nreq[u]++; }
        if (!q.homo || D.req_mult[u][r] == 0) D.req_mult[u][r]++;
      }
  }
  ix.root = root;
  ix.order = order;
  // steps of a round: by longest path from a vertex without parents (d1) and
  // from one without children (d2); the lighting levels draw on no other
  // vertex's flag of the same level
  for (uint32_t f = 0; f < 2; f++) {
    uint32_t level[kMaxQ] = {}, deepest = 0, k = 0;
    for (uint32_t i = 0; i < nq && !D.lighting; i++) {
      const uint32_t u = order[f == 0 ? i : nq - 1 - i];
      for (uint32_t w : f == 0 ? par[u] : chd[u]) level[u] = std::max(level[u], level[w] + 1);
      deepest = std::max(deepest, level[u]);
    }
    ix.rounds.steps[f] = deepest + 1;
    for (uint32_t l = 0; l <= deepest; l++) {
      for (uint32_t u = 0; u < nq; u++)
        if (level[u] == l) ix.rounds.order[f][k++] = (uint8_t)u;
      ix.rounds.end[f][l] = (uint8_t)k;
    }
  }

  ix.words = index_words(g.n_cap);
  const uint64_t fam = 8ull * nq * ix.words;
  ix.bits.words = ix.words;
  DevBlock blk;
  for (uint32_t cap = kListCap;; cap = kListCapSmall) {  // short lists where there is no room for long ones
    blk = DevBlock{};
    index_block(ix, blk, nq, g.n_cap, cap);
    rc = blk.alloc(mem, &ix.block);
    if (rc == CSM_OK) break;
    if (cap == kListCapSmall) return rc;
  }
  ix.block_bytes = blk.total;
  ix.bits.d2 = ix.bits.d1 + nq * ix.words;
  ix.bits.m1 = ix.bits.d2 + nq * ix.words;
  ix.bits.m2 = ix.bits.m1 + nq * ix.words;
  IXCK(cudaMemsetAsync(ix.bits.count, 0, 8ull * nq + 4, st));
  IXCK(cudaMemsetAsync(ix.bits.d1, 0, 4 * fam, st));
  IXCK(cudaMemcpyAsync(ix.d_dag, &D, sizeof(IxDag), cudaMemcpyHostToDevice, st));
  ix.d2 = ix.bits.d2;
  ix.active = true;
  rc = index_launch_build(ix, g, st, launches);
  if (rc) return rc;
  IXCK(cudaStreamSynchronize(st));
  return CSM_OK;
}

uint64_t index_bytes(int algo, uint32_t nq, uint32_t n_cap) {
  if (algo != CSM_ALGO_TURBOFLUX && algo != CSM_ALGO_SYMBI && algo != CSM_ALGO_CALIG && algo != CSM_ALGO_NEWSP)
    return 0;
  IndexState ix;
  DevBlock blk;
  index_block(ix, blk, nq, n_cap, kListCap);
  return blk.total;
}

int index_build(IndexState& ix, DevMem& mem, const DevGraph& g, const IndexQuery& q, int algo, int sm_count,
                cudaStream_t st, uint64_t* launches) {
  index_free(ix, mem);
  ix.algo = algo;
  ix.sm_count = sm_count > 0 ? sm_count : 148;
  if (algo != CSM_ALGO_TURBOFLUX && algo != CSM_ALGO_SYMBI && algo != CSM_ALGO_CALIG && algo != CSM_ALGO_NEWSP)
    return CSM_OK;
  const bool lighting = algo == CSM_ALGO_CALIG || algo == CSM_ALGO_NEWSP;
  const uint32_t nq = q.n;
  const auto& nbr = *q.nbr;
  const auto& el = *q.elabel;
  // query edges u < u' in adjacency order, as the frequency scan visits them
  std::vector<std::pair<uint32_t, uint32_t>> edges;
  std::vector<uint32_t> e_lab;
  for (uint32_t u = 0; u < nq; u++)
    for (size_t i = 0; i < nbr[u].size(); i++)
      if (u < nbr[u][i]) { edges.emplace_back(u, nbr[u][i]); e_lab.push_back(el[u][i]); }
  const uint32_t ne = (uint32_t)edges.size();
  if (ne == 0 || ne > kMaxQE || nq > kMaxQ) return set_err(CSM_EUNSUPPORTED, "query size outside the index limits");
  if (lighting && 2 * ne > kMaxQE)
    return set_err(CSM_EUNSUPPORTED, "query has more than %u edges (lighting filter limit)", kMaxQE / 2);
  std::vector<std::vector<uint32_t>> par(nq), chd(nq), par_l(nq), chd_l(nq);
  std::vector<uint32_t> order;
  uint32_t root = 0;
  if (lighting) {
    // lighting: every query neighbour is a child, nobody has a parent
    for (uint32_t u = 0; u < nq; u++) {
      order.push_back(u);
      for (size_t i = 0; i < nbr[u].size(); i++) { chd[u].push_back(nbr[u][i]); chd_l[u].push_back(el[u][i]); }
    }
  } else {
    const int rc = dag_for(q, g, algo, edges, e_lab, ix.sm_count, mem, st, launches, root, par, chd, par_l, chd_l,
                           order);
    if (rc) return rc;
  }
  if (order.size() != nq) return set_err(CSM_EINVAL, "query graph is not connected");
  const int rc = index_finish(ix, mem, g, q, algo, root, order, par, chd, par_l, chd_l, st, launches);
  // the NewSP-style plugin filters candidates by the neighbour-label
  // frequencies alone (d1); d2 is still kept
  if (rc == CSM_OK && algo == CSM_ALGO_NEWSP) ix.d2 = ix.bits.d1;
  return rc;
}

// The incremental round (k_ix_round): one block per SM.
static int index_round(IndexState& ix, const DevGraph& g, const uint64_t* keys, uint32_t L, uint32_t vert,
                       cudaStream_t st, uint64_t* launches) {
  IxOrder ord = ix.rounds;
  DevGraph gv = g;
  const IxDag* dag = ix.d_dag;
  IxBits bits = ix.bits;
  void* args[] = {&gv, &dag, &bits, &ord, &keys, &L, &vert};
  IXCK(cudaLaunchCooperativeKernel((const void*)k_ix_round, dim3((unsigned)ix.sm_count), dim3(512), args, 0, st));
  (*launches)++;
  return CSM_OK;
}

int index_apply_edges(IndexState& ix, const DevGraph& g, const uint64_t* keys, uint32_t L, cudaStream_t st,
                      uint64_t* launches) {
  if (!ix.active || L == 0) return CSM_OK;
  return index_round(ix, g, keys, L, kNone, st, launches);
}

int index_vertex_update(IndexState& ix, const DevGraph& g, const csm_update& h, cudaStream_t st, uint64_t* launches) {
  if (!ix.active) return CSM_OK;
  if (h.type != 'v' || h.id1 >= g.n_cap) return CSM_OK;  // a new or a removed vertex: re-evaluate its flags
  return index_round(ix, g, nullptr, 0, h.id1, st, launches);
}

int index_counts(IndexState& ix, cudaStream_t st, uint64_t* d1_count, uint64_t* d2_count) {
  *d1_count = 0; *d2_count = 0;
  if (!ix.active) return CSM_OK;
  const uint64_t n = (uint64_t)ix.h_dag.nq * ix.words;
  IXCK(cudaMemsetAsync(ix.d_pop, 0, 16, st));
  k_ix_popcount<<<ix.sm_count * 2, 256, 0, st>>>(ix.bits.d1, n, (unsigned long long*)ix.d_pop);
  k_ix_popcount<<<ix.sm_count * 2, 256, 0, st>>>(ix.bits.d2, n, (unsigned long long*)ix.d_pop + 1);
  IXCK(cudaGetLastError());
  unsigned long long h[2];
  IXCK(cudaMemcpyAsync(h, ix.d_pop, 16, cudaMemcpyDeviceToHost, st));
  IXCK(cudaStreamSynchronize(st));
  *d1_count = h[0]; *d2_count = h[1];
  ix.entries = h[0]; ix.vertices = h[1];
  return CSM_OK;
}

void index_stats(const IndexState& ix, uint64_t* entries, uint64_t* vertices) {
  *entries = ix.entries;
  *vertices = ix.vertices;
}

void index_free(IndexState& ix, DevMem& mem) {
  if (ix.block) mem.release(ix.block, ix.block_bytes);
  ix.block = nullptr;
  ix.bits = IxBits{};
  ix.d_dag = nullptr;
  ix.d_pop = nullptr;
  ix.d2 = nullptr;
  ix.words = 0;
  ix.active = false;
  ix.order.clear();
}

}  // namespace csm
