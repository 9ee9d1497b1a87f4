// Data-graph kernels: load-time CSR build, per-batch resolution of edge
// lifetimes, in-place slack-block insertion / deletion, pool compaction.
//
// Reference semantics restated here:
//   Graph::AddEdge  (ParaCOSM/CSM/graph/graph.cpp:58-93)  sorted insert, duplicate = no-op
//   Graph::RemoveEdge (ParaCOSM/CSM/graph/graph.cpp:95-116) sorted erase, missing edge = error
//   Graph::GetEdgeLabel (ParaCOSM/CSM/graph/graph.cpp:133-174) label of an existing edge
#include <cub/block/block_radix_sort.cuh>

#include "csm_kernels.cuh"

namespace csm {

// ---------------------------------------------------------------------
// row tables (DevGraph::htab)
// ---------------------------------------------------------------------

// Places an entry that is not in the table (the rows are sets); entries of one
// row may be placed side by side.
__device__ __forceinline__ void row_table_insert(const DevGraph& g, uint2 r, uint32_t entry) {
  const uint32_t buckets = r.y >> 2;
  uint32_t* tab = g.htab + 2ull * r.x;
  uint32_t s = row_bucket(entry, buckets);
  for (uint32_t n = 0; n < buckets; n++) {
    const RowBucket b = ld_bucket(tab + 8ull * s);
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (b.k[i] == kSlotEmpty && atomicCAS(tab + 8ull * s + i, kSlotEmpty, entry) == kSlotEmpty) return;
    if (++s == buckets) s = 0;
  }
  atomicExch(&g.ps->error, kErrRowTable);  // no empty slot left
}

// Slot of `entry` in a row table (offset from its start), or kSlotEmpty;
// `open`: its bucket has an empty slot.
__device__ __forceinline__ uint32_t row_locate(const uint32_t* tab, uint32_t buckets, uint32_t entry, bool& open) {
  uint32_t s = row_bucket(entry, buckets);
  for (uint32_t n = 0; n < buckets; n++) {
    const RowBucket b = ld_bucket(tab + 8ull * s);
    uint32_t at = kSlotEmpty;
    open = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if ((b.k[i] & ~kSlotTouched) == entry) at = 8u * s + (uint32_t)i;
      open = open || b.k[i] == kSlotEmpty;
    }
    if (at != kSlotEmpty || open) return at;
    if (++s == buckets) s = 0;
  }
  return kSlotEmpty;
}

// A slot of a bucket that was never full is free again; in a full one a
// deleted slot keeps the searches going that run over it, and is counted.
__device__ __forceinline__ void row_table_delete(const DevGraph& g, uint32_t x, uint2 r, uint32_t entry) {
  uint32_t* tab = g.htab + 2ull * r.x;
  bool open = false;
  const uint32_t s = row_locate(tab, r.y >> 2, entry, open);
  if (s == kSlotEmpty) return;
  tab[s] = open ? kSlotEmpty : kSlotTomb;
  if (!open) atomicAdd(&g.htomb[x], 1u);
}

// ---------------------------------------------------------------------
// load-time CSR build
// ---------------------------------------------------------------------

__global__ void k_load_edge_keys(const uint32_t* e, uint64_t m, const uint32_t* vlabel, uint32_t n,
                                 uint64_t* key, uint64_t* idx, unsigned long long* bad) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const uint32_t a = e[3 * i], b = e[3 * i + 1];
  idx[i] = i;
  if (a == b) { key[i] = ~0ULL; return; }  // self loops are dropped
  if (a >= n || b >= n || vlabel[a] == kNone || vlabel[b] == kNone) {
    key[i] = ~0ULL;
    atomicAdd(bad, 1ULL);
    return;
  }
  key[i] = ((uint64_t)min(a, b) << 32) | (uint64_t)max(a, b);
}

// Folds raw vertex labels to the engine's compact labels (see DevGraph).
__global__ void k_fold_vlabels(uint32_t* vlabel, uint32_t n, DevGraph g) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  vlabel[v] = fold_vlabel(g, vlabel[v]);
}

// One directed entry pair per distinct undirected edge; repeats (same
// endpoints, later in the input) are dropped, so the first label wins.
__global__ void k_load_directed(const uint64_t* ukey, const uint64_t* uidx, uint64_t m, const uint32_t* e,
                                DevGraph g, uint64_t* dkey) {
  const KeyBits kb = g.kb;
  const uint32_t* vlabel = g.vlabel;
  const uint32_t n_el = g.n_el;
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint64_t k = ukey[j];
  if (k == ~0ULL || (j > 0 && ukey[j - 1] == k)) {
    dkey[2 * j] = kb.sentinel();
    dkey[2 * j + 1] = kb.sentinel();
    return;
  }
  const uint64_t i = uidx[j];
  const uint32_t x = (uint32_t)(k >> 32), y = (uint32_t)k, l = fold_elabel(g, e[3 * i + 2]);
  dkey[2 * j] = kb.pack(x, vlabel[y] * n_el + l, y);
  dkey[2 * j + 1] = kb.pack(y, vlabel[x] * n_el + l, x);
}

// Per (vertex, combo) run lengths (into dir, cleared before and scanned later)
// and the first position of each vertex in the sorted keys.  A run's first
// entry subtracts its place and its last adds the place after it (modulo
// 2^32): no thread walks a run (a hub's runs are long: 518 us on 2^19
// vertices and 4.2M edges).
__global__ void k_load_count(const uint64_t* dkey, uint64_t M, KeyBits kb, uint32_t nc, uint32_t* dir,
                             uint64_t* first, unsigned long long* n_valid) {
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  const uint64_t k = dkey[j];
  if (!kb.real(k)) return;
  const uint64_t before = j ? dkey[j - 1] : ~0ULL, after = j + 1 < M ? dkey[j + 1] : ~0ULL;
  if (!kb.real(after)) *n_valid = j + 1;
  const uint32_t x = kb.x_of(k);
  uint32_t* run = dir + (size_t)x * (nc + 1) + kb.c_of(k);
  if (j == 0 || kb.x_of(before) != x) first[x] = j;
  if (j == 0 || (before >> kb.yb) != (k >> kb.yb)) atomicSub(run, (uint32_t)j);
  if (!kb.real(after) || (after >> kb.yb) != (k >> kb.yb)) atomicAdd(run, (uint32_t)(j + 1));
}

// Capacities of a row of d entries when it is laid out and when it has to grow.
__device__ __forceinline__ uint32_t slack_cap(uint32_t d, bool tables) {
  const uint32_t c = d == 0 ? 0u : d + max(2u, d >> 2);
  return tables ? row_round(c) : c;
}
__device__ __forceinline__ uint32_t grow_cap(uint32_t d, bool tables) {
  const uint32_t c = d + max(8u, d >> 1);
  return tables ? row_round(c) : c;
}

__global__ void k_load_caps(const uint32_t* dir, uint32_t n_cap, uint32_t nc, uint32_t tables, uint64_t* cap64,
                            unsigned long long* sums) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t d = v < n_cap ? dir[(size_t)v * (nc + 1) + nc] : 0u;
  const uint32_t with = slack_cap(d, true), without = slack_cap(d, false);
  if (v < n_cap) cap64[v] = tables ? with : without;
  __shared__ unsigned long long s_sum[2];
  if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long a = with, b = without;
  for (int o = 16; o; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&s_sum[0], a);
    atomicAdd(&s_sum[1], b);
  }
  __syncthreads();
  if (threadIdx.x < 2) atomicAdd(sums + threadIdx.x, s_sum[threadIdx.x]);
}

// In place: row[v] holds the row's offset as one word before.
__global__ void k_load_rows(const uint32_t* dir, uint32_t n_cap, uint32_t nc, uint32_t tables, uint2* row) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_cap) return;
  row[v] = make_uint2(row[v].x, slack_cap(dir[(size_t)v * (nc + 1) + nc], tables));
}

// One thread per directed entry: its place in the row and its slot in the row
// table (emptied before).  Taking the entries side by side, each with its
// combo in the key, needs no search for the combo and no loop over long rows.
__global__ void k_load_scatter(const uint64_t* dkey, uint64_t M, const uint64_t* first, DevGraph g, uint32_t* pool) {
  const KeyBits kb = g.kb;
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  const uint64_t k = dkey[j];
  if (!kb.real(k)) return;
  const uint32_t x = kb.x_of(k), y = kb.y_of(k);
  const uint2 r = g.row[x];
  pool[r.x + (j - first[x])] = y;
  if (g.htab) row_table_insert(g, r, row_entry(y, kb.c_of(k) % g.n_el, g.hlb));
}

// Turns per-combo counts into row-relative segment offsets; dir[nc] = degree.
__global__ void k_dir_scan(uint32_t* dir, uint32_t n_cap, uint32_t nc) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_cap) return;
  uint32_t* d = dir + (size_t)v * (nc + 1);
  uint32_t run = 0;
  for (uint32_t c = 0; c < nc; c++) { uint32_t t = d[c]; d[c] = run; run += t; }
  d[nc] = run;
}

// ---------------------------------------------------------------------
// batch preparation
// ---------------------------------------------------------------------

// Sort key of a record that is no valid edge update (ids are below 2^yb - 1).
__device__ __forceinline__ uint64_t edge_sort_none(const KeyBits& kb) { return (1ULL << (2 * kb.yb)) - 1; }

__global__ void k_batch_init(const csm_update* ups, uint32_t B, DevGraph g, uint64_t* ukey, uint32_t* useq,
                             UpdInfo* info, unsigned int* cnt) {
  uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < 16) cnt[s] = 0;
  if (s >= B) return;
  const csm_update u = ups[s];
  UpdInfo inf;
  inf.v1 = u.id1; inf.v2 = u.id2; inf.label = fold_elabel(g, u.label); inf.flags = 0;
  useq[s] = s;
  uint64_t key = edge_sort_none(g.kb);
  if (u.type == 'e') {
    const bool ok = u.id1 < g.n && u.id2 < g.n && u.id1 != u.id2 && g.vlabel[u.id1] != kNone &&
                    g.vlabel[u.id2] != kNone;
    if (ok) {
      key = ((uint64_t)min(u.id1, u.id2) << g.kb.yb) | (uint64_t)max(u.id1, u.id2);
      inf.flags = UF_VALID | (u.is_add ? UF_ADD : 0u);
    } else {
      inf.flags = UF_INVALID;
    }
  }
  ukey[s] = key;
  info[s] = inf;
}

// Stable sort of short key lists, a block each.  The position in the list rides
// in the bits below the key, so pairs move as one word and their values are
// fetched at the end.  What bounds it is the latency of its passes (5 bits each,
// through shared memory).  A device-wide sort takes a launch for every 8 bits
// and three to six more, and the lists one after another: the four sorts of a
// batch of 1,500 updates took 118 us and their clears 20, the two launches here
// 35 us (batches of 100: 38 and 13 us; of 4,097: 166 and 67 us).  Longer lists are better off with
// the whole device.
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS) k_sort_block(SortJobs jobs) {
  using Sort = cub::BlockRadixSort<uint64_t, THREADS, ITEMS, cub::NullType, 5>;
  extern __shared__ __align__(16) unsigned char sort_smem[];
  const SortJob& job = jobs.job[blockIdx.x];
  uint64_t item[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; i++) {
    const uint32_t at = threadIdx.x * ITEMS + (uint32_t)i;
    item[i] = (at < job.n ? job.key[at] : ~0ULL) << kSortPosBits | at;
  }
  Sort(*reinterpret_cast<typename Sort::TempStorage*>(sort_smem))
      .SortBlockedToStriped(item, (int)kSortPosBits, (int)(kSortPosBits + job.bits));
#pragma unroll
  for (int i = 0; i < ITEMS; i++) {
    const uint32_t to = (uint32_t)i * THREADS + threadIdx.x;
    if (to >= job.n) continue;
    const uint32_t pos = (uint32_t)item[i] & ((1u << kSortPosBits) - 1u);
    job.out[to] = (item[i] >> kSortPosBits) & ((1ULL << job.bits) - 1);
    if (job.pos) job.pos[to] = pos;
    if (job.val) job.val_out[to] = job.val[pos];
  }
}

template <int THREADS, int ITEMS>
static cudaError_t sort_block(const SortJobs& jobs, uint32_t n_jobs, cudaStream_t st) {
  using Sort = cub::BlockRadixSort<uint64_t, THREADS, ITEMS, cub::NullType, 5>;
  constexpr int bytes = (int)sizeof(typename Sort::TempStorage);
  cudaError_t e = cudaFuncSetAttribute(k_sort_block<THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  k_sort_block<THREADS, ITEMS><<<n_jobs, THREADS, bytes, st>>>(jobs);
  return cudaGetLastError();
}

cudaError_t launch_sort_block(const SortJobs& jobs, uint32_t n_jobs, cudaStream_t st) {
  uint32_t n = 0;
  for (uint32_t i = 0; i < n_jobs; i++) n = n > jobs.job[i].n ? n : jobs.job[i].n;
  // few threads where they do: 320 keys take 18.5 us with 1,024 threads, 6.7 us with 256
  if (n <= 512) return sort_block<256, 2>(jobs, n_jobs, st);
  if (n <= 2048) return sort_block<512, 4>(jobs, n_jobs, st);
  if (n <= 4096) return sort_block<1024, 4>(jobs, n_jobs, st);
  return sort_block<1024, kSortMax / 1024>(jobs, n_jobs, st);
}

__device__ __forceinline__ void emit2(uint64_t* key, unsigned int* n, uint32_t cap, uint64_t k1, uint64_t k2,
                                      uint64_t* val, uint64_t v, unsigned int* err) {
  unsigned int i = atomicAdd(n, 2u);
  if (i + 2 > cap) { atomicExch(err, kErrListOverflow); return; }
  key[i] = k1; key[i + 1] = k2;
  if (val) { val[i] = v; val[i + 1] = v; }
}

// One thread per distinct edge key of the batch walks that edge's updates in
// sequence order, starting from its state before the batch.  It decides each
// update's effect (insert, duplicate insert, delete, delete of a missing
// edge), the label a deletion counts with, the presence intervals of the
// edge inside the batch, and the row insertions (before the search) and row
// deletions (after it) that turn the CSR into the union graph and back.
__global__ void k_resolve(const uint64_t* skey, const uint32_t* sseq, uint32_t B, DevGraph g,
                          const csm_update* ups, UpdInfo* info, ResolveOut out) {
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= B) return;
  const uint64_t k = skey[j];
  if (k == edge_sort_none(g.kb) || (j > 0 && skey[j - 1] == k)) return;
  const uint32_t x = (uint32_t)(k >> g.kb.yb), y = (uint32_t)(k & ((1ULL << g.kb.yb) - 1));
  const uint32_t lx = g.vlabel[x], ly = g.vlabel[y];
  const uint32_t* pool = g.pools[g.ps->active];
  const uint32_t l0 = find_label(g, pool, x, y);
  const bool present0 = (l0 != kNone);
  bool cur_p = present0;
  uint32_t cur_l = present0 ? l0 : 0u;
  int32_t cur_s = -1;
  uint64_t ins_mask = 0;
  unsigned int* err = &g.ps->error;
  for (uint32_t e = j; e < B && skey[e] == k; e++) {
    const uint32_t s = sseq[e];
    UpdInfo inf = info[s];
    const uint32_t label = inf.label;  // folded in k_batch_init
    if (inf.flags & UF_ADD) {
      if (cur_p) {
        inf.label = label;  // duplicate insert: graph unchanged, counted with the given label
        inf.flags |= UF_DUP;
      } else {
        cur_p = true; cur_l = label; cur_s = (int32_t)s;
        inf.label = label; inf.flags |= UF_MUT;
        if (!(present0 && label == l0)) ins_mask |= 1ULL << label;
      }
    } else {
      if (!cur_p) {
        inf.flags |= UF_INVALID;  // deleting a missing edge
      } else {
        inf.label = cur_l; inf.flags |= UF_MUT;
        const uint64_t span = (uint64_t)(uint32_t)cur_s | ((uint64_t)(uint32_t)s << 32);
        emit2(out.t_key, out.n_t, out.cap, g.kb.pack(x, ly * g.n_el + cur_l, y), g.kb.pack(y, lx * g.n_el + cur_l, x),
              out.t_span, span, err);
        cur_p = false;
      }
    }
    info[s] = inf;
  }
  if (cur_p && cur_s >= 0) {
    const uint64_t span = (uint64_t)(uint32_t)cur_s | ((uint64_t)(uint32_t)kTimeInf << 32);
    emit2(out.t_key, out.n_t, out.cap, g.kb.pack(x, ly * g.n_el + cur_l, y), g.kb.pack(y, lx * g.n_el + cur_l, x),
          out.t_span, span, err);
  }
  for (uint64_t m = ins_mask; m; m &= m - 1) {
    const uint32_t l = (uint32_t)__ffsll((long long)m) - 1;
    emit2(out.ins_key, out.n_ins, out.cap, g.kb.pack(x, ly * g.n_el + l, y), g.kb.pack(y, lx * g.n_el + l, x),
          nullptr, 0, err);
  }
  const uint64_t uni = ins_mask | (present0 ? (1ULL << l0) : 0ULL);
  const uint64_t endm = cur_p ? (1ULL << cur_l) : 0ULL;
  for (uint64_t m = uni & ~endm; m; m &= m - 1) {
    const uint32_t l = (uint32_t)__ffsll((long long)m) - 1;
    emit2(out.del_key, out.n_del, out.cap, g.kb.pack(x, ly * g.n_el + l, y), g.kb.pack(y, lx * g.n_el + l, x),
          nullptr, 0, err);
  }
}

// First index after j, up to `end`, whose key is not below `limit` (key[j] is):
// the end of a run in a sorted list.  Steps that double keep a run of one entry
// at one load and a hub's at a few.
__device__ __forceinline__ uint32_t run_end(const uint64_t* key, uint32_t j, uint32_t end, uint64_t limit) {
  uint32_t lo = j, step = 1;
  while (step < end - lo && key[lo + step] < limit) { lo += step; step <<= 1; }
  uint32_t hi = step < end - lo ? lo + step : end;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (key[mid] < limit) lo = mid; else hi = mid;
  }
  return hi;
}

// Appends one VRange per vertex run of a sorted packed-key list.  pad = 1
// marks a row longer than kBigRow entries before the batch: the mutation
// kernels give such rows a whole block instead of a warp.
__global__ void k_ranges(const uint64_t* key, uint32_t cap, KeyBits kb, VRange* ranges, unsigned int* n_ranges,
                         const uint32_t* dir, uint32_t nc) {
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= cap) return;
  const uint64_t k = key[j];
  if (!kb.real(k)) return;
  const uint32_t x = kb.x_of(k);
  if (j > 0 && kb.x_of(key[j - 1]) == x) return;
  const uint32_t t = run_end(key, j, cap, kb.pack(x + 1, 0, 0));
  unsigned int i = atomicAdd(n_ranges, 1u);
  const uint32_t big = dir[(size_t)x * (nc + 1) + nc] > kBigRow ? 1u : 0u;
  ranges[i] = VRange{x, j, t - j, big};
}

__device__ __forceinline__ void temporal_put(const DevGraph& g, uint64_t key, uint64_t val) {
  uint32_t s = temporal_slot(key, g.t_mask);
  for (uint32_t n = 0; n <= g.t_mask; n++, s = (s + 1) & g.t_mask) {
    if (atomicCAS((unsigned long long*)&g.t_tab[s].x, (unsigned long long)kTempEmpty, (unsigned long long)key) ==
        kTempEmpty) {
      g.t_tab[s].y = val;
      return;
    }
  }
  atomicExch(&g.ps->error, kErrListOverflow);  // no empty slot: more entries than the batch can have
}

// Temporal entries of the batch (g.t_key, sorted): their number for each row,
// the temporal table (emptied before), and the touched bit of every entry in
// its row table, so that the search asks for an edge's presence only where it
// can be in question.  Runs on the union graph, which holds every touched
// entry.
__global__ void k_temporal_set(uint32_t L, DevGraph g) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= L) return;
  const uint64_t k = g.t_key[j];
  if (!g.kb.real(k)) return;
  const uint32_t x = g.kb.x_of(k);
  if (g.htab && (j == 0 || g.t_key[j - 1] != k)) {
    const uint2 r = g.row[x];
    uint32_t* tab = g.htab + 2ull * r.x;
    bool open;
    const uint32_t s = row_locate(tab, r.y >> 2, row_entry(g.kb.y_of(k), g.kb.c_of(k) % g.n_el, g.hlb), open);
    if (s != kSlotEmpty) tab[s] |= kSlotTouched;
  }
  const uint64_t before = j > 0 ? g.t_key[j - 1] : ~0ULL;
  if (before != k) {  // the entry's intervals
    const uint32_t n = run_end(g.t_key, j, L, k + 1) - j;
    const int2 s = g.t_span[j];
    temporal_put(g, k, n == 1 ? (uint64_t)(uint32_t)(s.x + 1) | ((uint64_t)(uint32_t)s.y << 32)
                              : kTempMany | (uint64_t)j | ((uint64_t)n << 32));
  }
  if (j > 0 && (before >> g.kb.yb) == (k >> g.kb.yb)) return;
  const uint32_t n = run_end(g.t_key, j, L, ((k >> g.kb.yb) + 1) << g.kb.yb) - j;  // the segment's entries
  temporal_put(g, temporal_head(g, x, g.kb.c_of(k)), (uint64_t)j | ((uint64_t)n << 32));
  atomicAdd(&g.t_count[x], n);
}

// After the batch: the entries still in the graph lose the touched bit.
__global__ void k_temporal_clear(uint32_t L, DevGraph g) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= L) return;
  const uint64_t k = g.t_key[j];
  if (!g.kb.real(k)) return;
  const uint32_t x = g.kb.x_of(k);
  if (g.htab && (j == 0 || g.t_key[j - 1] != k)) {
    const uint2 r = g.row[x];
    uint32_t* tab = g.htab + 2ull * r.x;
    bool open;
    const uint32_t s = row_locate(tab, r.y >> 2, row_entry(g.kb.y_of(k), g.kb.c_of(k) % g.n_el, g.hlb), open);
    if (s != kSlotEmpty) tab[s] &= ~kSlotTouched;
  }
  if (j == 0 || g.kb.x_of(g.t_key[j - 1]) != x) g.t_count[x] = 0;
}

// True in every thread of the block that arrives last; *ctr is 0 before and after.
__device__ __forceinline__ bool last_block(unsigned int* ctr) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ctr, 1u) + 1u == gridDim.x;
    if (last) *ctr = 0;
    __threadfence();
  }
  __syncthreads();
  return last;
}

// Pool space that the batch's growing rows will take; the last block decides
// whether the pools are compacted first.
__global__ void k_reloc_need(const VRange* ranges, const unsigned int* n_ranges, DevGraph g) {
  PoolState* ps = g.ps;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long need = 0;
  if (i < *n_ranges) {
    const VRange r = ranges[i];
    const uint32_t deg = g.dir[(size_t)r.x * (g.nc + 1) + g.nc];
    if (deg + r.count > g.row[r.x].y) need = grow_cap(deg + r.count, g.htab);
  }
  // warp-aggregated add
  for (int o = 16; o; o >>= 1) need += __shfl_down_sync(0xffffffffu, need, o);
  if ((threadIdx.x & 31) == 0 && need) atomicAdd(&ps->need, need);
  if (last_block(&ps->arrived) && threadIdx.x == 0) {
    const unsigned long long all = atomicExch(&ps->need, 0ULL);
    ps->compact = all > g.pool_cap - ps->top[ps->active] ? 1u : 0u;
  }
}

// Combo of the row-relative entry index i: upper_bound(dir, i) - 1.
__device__ __forceinline__ uint32_t combo_at(const uint32_t* dirx, uint32_t nc, uint32_t i) {
  uint32_t lo = 0, hi = nc;  // find last c with dirx[c] <= i
  while (lo < hi) {
    uint32_t mid = (lo + hi + 1) >> 1;
    if (dirx[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Barrier of a group of G threads (a warp or a block).
template <int G>
__device__ __forceinline__ void group_sync() {
  if (G == 32) __syncwarp(); else __syncthreads();
}

// Builds row x's table from the row's entries (dirx: its directory, deg of
// them), by G threads; no thread of another group touches the region.  A thread
// takes four entries at a time, so that their chains of loads overlap: a call
// that moves a row of a million entries takes 5 ms, 11 ms one entry after another.
template <int G>
__device__ __forceinline__ void row_table_build(const DevGraph& g, const uint32_t* pool, uint32_t x, uint2 row,
                                                const uint32_t* dirx, uint32_t deg, uint32_t lane) {
  uint32_t* tab = g.htab + 2ull * row.x;
  for (uint32_t i = lane; i < 2u * row.y; i += G) tab[i] = kSlotEmpty;
  if (lane == 0) g.htomb[x] = 0;
  group_sync<G>();
  const uint32_t buckets = row.y >> 2;
  for (uint32_t i = lane; i < deg; i += 4 * G) {
    uint32_t entry[4], slot[4], was[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      const uint32_t at = min(i + u * G, deg - 1u);
      entry[u] = row_entry(pool[(uint64_t)row.x + at], combo_at(dirx, g.nc, at) % g.n_el, g.hlb);
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {  // the first empty slot of the home bucket
      const uint32_t s = 8u * row_bucket(entry[u], buckets);
      const RowBucket b = ld_bucket(tab + s);
      slot[u] = kSlotEmpty;
#pragma unroll
      for (int k = 7; k >= 0; k--)
        if (b.k[k] == kSlotEmpty) slot[u] = s + (uint32_t)k;
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      was[u] = 0;
      if (i + u * G < deg && slot[u] != kSlotEmpty) was[u] = atomicCAS(tab + slot[u], kSlotEmpty, entry[u]);
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; u++)  // the bucket was full, or another entry was faster
      if (i + u * G < deg && was[u] != kSlotEmpty) row_table_insert(g, row, entry[u]);
  }
}

// Deleted slots a row's table may hold before a deletion builds it afresh: a
// quarter of the row's capacity keeps the table (twice the capacity) at most
// five eighths full, so that most buckets keep an empty slot; rows of up to 16
// slots may have four (with eight live entries of a table of 16, three quarters).
// A batch's own deletions come on top until its check.
__device__ __forceinline__ uint32_t tomb_limit(uint32_t cap) { return max(4u, cap >> 2); }

// Copies every row into the other pool with fresh slack (runs only when the
// active pool cannot absorb this batch's relocations) and builds its table at
// its new place.  The rows that a block's threads size lie side by side there: the
// block empties their tables and takes their entries as one run, a thread an
// entry, whatever the rows' lengths.  What bounds it is the chain of loads of an
// entry's table insertion, so that no row may be one warp's: 3.5M rows and 11M
// entries, the longest row of 52,000, took 18 ms row by row, a warp each, and
// 2.5 ms so (4.1 ms for the copies alone, by a thread a row).
__global__ void __launch_bounds__(1024) k_compact_copy(DevGraph g) {
  PoolState* ps = g.ps;
  if (!ps->compact) return;
  const uint32_t src = ps->active, dst = 1u - src;
  const uint32_t* sp = g.pools[src];
  uint32_t* dp = g.pools[dst];
  __shared__ unsigned long long base;
  __shared__ uint32_t scan[1024], incl[1024];   // capacities and entries up to each row
  __shared__ uint32_t s_from[1024];             // where each row comes from
  const uint32_t me = threadIdx.x;
  for (uint64_t v0 = (uint64_t)blockIdx.x * blockDim.x; v0 < g.n_cap; v0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t v = v0 + me;
    uint32_t deg = 0, cap = 0;
    if (v < g.n_cap) { deg = g.dir[v * (g.nc + 1) + g.nc]; cap = slack_cap(deg, g.htab); }
    scan[me] = cap;
    incl[me] = deg;
    s_from[me] = v < g.n_cap ? g.row[v].x : 0u;
    __syncthreads();
    for (uint32_t o = 1; o < blockDim.x; o <<= 1) {  // inclusive scans
      const uint32_t t = me >= o ? scan[me - o] : 0, u = me >= o ? incl[me - o] : 0;
      __syncthreads();
      scan[me] += t;
      incl[me] += u;
      __syncthreads();
    }
    if (me == blockDim.x - 1) base = atomicAdd(&ps->top[dst], (unsigned long long)scan[me]);
    __syncthreads();
    const unsigned long long off = base + scan[me] - cap;
    const bool fits = off + cap <= g.pool_cap;
    if (!fits) atomicExch(&ps->error, kErrPoolFull);
    const uint32_t rows = (uint32_t)__syncthreads_count(fits);  // the first ones: offsets ascend
    const uint32_t total = rows ? incl[rows - 1] : 0u;
    if (g.htab) {
      uint32_t* tab = g.htab + 2ull * base;
      const unsigned long long words = rows ? 2ull * scan[rows - 1] : 0ull;
      for (unsigned long long i = me; i < words; i += blockDim.x) tab[i] = kSlotEmpty;
      __syncthreads();
    }
    for (unsigned long long e = me; e < total; e += blockDim.x) {
      uint32_t r = 0;  // rows that end before entry e
#pragma unroll
      for (uint32_t step = 512; step; step >>= 1)
        if (incl[r + step - 1] <= e) r += step;
      const uint32_t i = (uint32_t)e - (r ? incl[r - 1] : 0u), before = r ? scan[r - 1] : 0u;
      const uint2 row = make_uint2((uint32_t)base + before, scan[r] - before);
      const uint32_t y = sp[(uint64_t)s_from[r] + i];
      dp[(uint64_t)row.x + i] = y;
      if (g.htab)
        row_table_insert(g, row, row_entry(y, combo_at(g.dir + (v0 + r) * (g.nc + 1), g.nc, i) % g.n_el, g.hlb));
    }
    __syncthreads();
    if (v < g.n_cap) {
      // a row that finds no room is lost, and the context in error; it must not
      // point into the other pool's slots, which nobody has written
      g.row[v] = fits ? make_uint2((uint32_t)off, cap) : make_uint2(0, 0);
      if (!fits)
        for (uint32_t c = 0; c <= g.nc; c++) g.dir[v * (g.nc + 1) + c] = 0;
      if (g.htab) g.htomb[v] = 0;
    }
    __syncthreads();
  }
  if (last_block(&ps->arrived) && threadIdx.x == 0) {  // every row has moved
    ps->top[src] = 0;
    ps->active = dst;
    ps->compact = 0;
  }
}

__device__ __forceinline__ uint32_t lower_bound_u64(const uint64_t* a, uint32_t lo, uint32_t hi, uint64_t x) {
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Number of the k ascending positions in pos that are at most (below) i.
__device__ __forceinline__ uint32_t count_le(const uint32_t* pos, uint32_t k, uint32_t i) {
  uint32_t lo = 0, hi = k;
#pragma unroll 1
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (pos[mid] <= i) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Row moves by G threads (a warp or a block), eight entries a thread and round:
// a round's entries are all in registers before any is stored, so a move
// within a row is safe when rounds go from the back for a move to the right and
// from the front for a move to the left.  An entry's place follows from its
// rank among the k changed positions, whatever k is: moving the blocks between
// changed positions one after another cost two barriers per change (a batch
// of 65,536 updates changes hub rows in hundreds of places: 634 us inserting
// and 691 us deleting on the 2^22-vertex graph, against 448 and 469 us, the
// time one block takes to move its longest row).
constexpr uint32_t kMoveUnroll = 8;

// Entries [from, deg) of the row at src go to dst + i + (changed positions <= i).
template <int G>
__device__ __forceinline__ void group_insert_move(uint32_t* pool, uint64_t src, uint64_t dst, uint32_t from,
                                                  uint32_t deg, const uint32_t* pos, uint32_t k, uint32_t lane) {
  for (uint32_t end = deg; end > from;) {
    const uint32_t beg = end - from > G * kMoveUnroll ? end - G * kMoveUnroll : from;
    uint32_t val[kMoveUnroll];
#pragma unroll
    for (uint32_t u = 0; u < kMoveUnroll; u++) {
      const uint32_t i = beg + u * G + lane;
      if (i < end) val[u] = pool[src + i];
    }
    group_sync<G>();
#pragma unroll
    for (uint32_t u = 0; u < kMoveUnroll; u++) {
      const uint32_t i = beg + u * G + lane;
      if (i < end) pool[dst + i + count_le(pos, k, i)] = val[u];
    }
    group_sync<G>();
    end = beg;
  }
}

// Entries (pos[0], deg) but those at the changed positions move left by the
// number of changed positions before them.
template <int G>
__device__ __forceinline__ void group_delete_move(uint32_t* pool, uint64_t off, uint32_t deg, const uint32_t* pos,
                                                  uint32_t k, uint32_t lane) {
  for (uint32_t beg = pos[0]; beg < deg; beg += G * kMoveUnroll) {
    uint32_t val[kMoveUnroll];
#pragma unroll
    for (uint32_t u = 0; u < kMoveUnroll; u++) {
      const uint32_t i = beg + u * G + lane;
      if (i < deg) val[u] = pool[off + i];
    }
    group_sync<G>();
#pragma unroll
    for (uint32_t u = 0; u < kMoveUnroll; u++) {
      const uint32_t i = beg + u * G + lane;
      if (i >= deg) continue;
      const uint32_t le = count_le(pos, k, i);
      if (pos[le - 1] != i) pool[off + i - le] = val[u];  // le >= 1: i is not before the first
    }
    group_sync<G>();
  }
}

// lower_bound of x in the sorted range a[lo, hi) by a warp: 32 probes a round.
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t* a, uint32_t lo, uint32_t hi, uint32_t x,
                                                     uint32_t lane) {
  while (hi - lo > 32) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint32_t at = lo + lane * step;
    const uint32_t less = __popc(__ballot_sync(0xffffffffu, at < hi && a[at] < x));
    if (less == 0) return lo;
    const uint32_t last = lo + (less - 1) * step;  // the last probe below x
    hi = min(hi, last + step);
    lo = last + 1;
  }
  return lo + __popc(__ballot_sync(0xffffffffu, lo + lane < hi && a[lo + lane] < x));
}

// Merges each vertex's sorted insert list into its row; G = 32: one warp per
// row of at most kBigRow entries, G = blockDim: one block per longer row.
// Insert j (sorted by combo, then id) goes to row position p_j + j, p_j being
// its lower_bound in the old row; an old entry i shifts by the inserts with
// p_j <= i -- in place, or into a larger row elsewhere.
template <int G>
__device__ __forceinline__ void mut_insert(const VRange* ranges, uint32_t nr, const uint64_t* ins_key,
                                           uint32_t* ins_dst, const DevGraph& g, unsigned long long* s_off,
                                           uint32_t block, uint32_t blocks) {
  const uint32_t lane = threadIdx.x % G;
  const uint32_t groups_per_block = blockDim.x / G;
  PoolState* ps = g.ps;
  uint32_t* pool = g.pools[ps->active];
  for (uint32_t w = block * groups_per_block + threadIdx.x / G; w - threadIdx.x / G < nr;
       w += blocks * groups_per_block) {
    // every thread of a block-sized group walks the same w; warps of a
    // warp-sized group skip ranges of the other kind
    const bool mine = w < nr && ranges[w].pad == (G == 32 ? 0u : 1u);
    if (!mine) continue;
    const VRange r = ranges[w];
    const uint32_t x = r.x, s = r.start, k = r.count;
    uint32_t* dirx = g.dir + (size_t)x * (g.nc + 1);
    const uint32_t deg = dirx[g.nc];
    const uint2 old = g.row[x];
    const uint64_t off = old.x;
    const uint32_t new_deg = deg + k;
    const uint32_t tomb = g.htab ? g.htomb[x] : 0u;  // read by every thread before a build clears it
    uint64_t dst_off = off;
    uint32_t new_cap = 0;
    if (new_deg > old.y) {
      new_cap = grow_cap(new_deg, g.htab);
      if (lane == 0) {
        unsigned long long o = atomicAdd(&ps->top[ps->active], (unsigned long long)new_cap);
        if (o + new_cap > g.pool_cap) { atomicExch(&ps->error, kErrPoolFull); o = ~0ULL; }
        s_off[threadIdx.x / G] = o;
      }
      group_sync<G>();
      dst_off = s_off[threadIdx.x / G];
      group_sync<G>();
      if (dst_off == ~0ULL) continue;  // uniform across the group
    }
    // 1. positions p_j in the old row
    for (uint32_t j = lane; j < k; j += G) {
      const uint64_t key = ins_key[s + j];
      const uint32_t c = g.kb.c_of(key), y = g.kb.y_of(key);
      ins_dst[s + j] = (uint32_t)lower_bound_u32(pool + off, dirx[c], dirx[c + 1], y);
    }
    group_sync<G>();
    // 2. old entries, 3. inserted ones
    group_insert_move<G>(pool, off, dst_off, dst_off == off ? ins_dst[s] : 0u, deg, ins_dst + s, k, lane);
    for (uint32_t j = lane; j < k; j += G) pool[dst_off + ins_dst[s + j] + j] = g.kb.y_of(ins_key[s + j]);
    group_sync<G>();
    // 4. directory: a combo's segment starts after the inserts of smaller combos
    for (uint32_t c = lane; c <= g.nc; c += G) {
      const uint32_t add = lower_bound_u64(ins_key, s, s + k, g.kb.pack(x, 0, 0) + ((uint64_t)c << g.kb.yb)) - s;
      dirx[c] += add;
    }
    const uint2 now = new_cap ? make_uint2((uint32_t)dst_off, new_cap) : old;
    if (lane == 0 && new_cap) g.row[x] = now;
    group_sync<G>();
    // 5. row table: the new entries, or the whole table when the row moved or
    // deleted slots would fill it past three quarters
    if (g.htab) {
      if (new_cap || new_deg + tomb > now.y + now.y / 2) {
        row_table_build<G>(g, pool, x, now, dirx, new_deg, lane);
      } else {
        for (uint32_t j = lane; j < k; j += G) {
          const uint64_t key = ins_key[s + j];
          row_table_insert(g, now, row_entry(g.kb.y_of(key), g.kb.c_of(key) % g.n_el, g.hlb));
        }
      }
      group_sync<G>();
    }
  }
}

// Removes each vertex's sorted delete list from its row in place (G as
// above).  Delete j sits at row position q_j; an old entry moves left by the
// deletes before it.  `del_pos` is scratch of the delete list's length.
template <int G>
__device__ __forceinline__ void mut_delete(const VRange* ranges, uint32_t nr, const uint64_t* del_key,
                                           uint32_t* del_pos, const DevGraph& g, uint32_t block, uint32_t blocks) {
  const uint32_t lane = threadIdx.x % G;
  const uint32_t groups_per_block = blockDim.x / G;
  uint32_t* pool = g.pools[g.ps->active];
  for (uint32_t w = block * groups_per_block + threadIdx.x / G; w - threadIdx.x / G < nr;
       w += blocks * groups_per_block) {
    const bool mine = w < nr && ranges[w].pad == (G == 32 ? 0u : 1u);
    if (!mine) continue;
    const VRange r = ranges[w];
    const uint32_t x = r.x, s = r.start, k = r.count;
    uint32_t* dirx = g.dir + (size_t)x * (g.nc + 1);
    const uint32_t deg = dirx[g.nc];
    const uint2 row = g.row[x];
    const uint64_t off = row.x;
    bool missing = false;
    for (uint32_t j = lane; j < k; j += G) {
      const uint64_t key = del_key[s + j];
      const uint32_t c = g.kb.c_of(key), y = g.kb.y_of(key);
      const uint32_t q = (uint32_t)lower_bound_u32(pool + off, dirx[c], dirx[c + 1], y);
      del_pos[s + j] = q;
      if (q >= dirx[c + 1] || pool[off + q] != y) missing = true;
    }
    // a deleted entry missing from its row: leave the row, report
    if (G == 32) { __syncwarp(); missing = __any_sync(0xffffffffu, missing); }
    else missing = __syncthreads_or(missing);
    if (missing) {
      if (lane == 0) atomicExch(&g.ps->error, kErrRowState);
      continue;
    }
    if (g.htab) {  // only now: the table follows the row
      for (uint32_t j = lane; j < k; j += G) {
        const uint64_t key = del_key[s + j];
        row_table_delete(g, x, row, row_entry(g.kb.y_of(key), g.kb.c_of(key) % g.n_el, g.hlb));
      }
      group_sync<G>();
    }
    const uint32_t tomb = g.htab ? g.htomb[x] : 0u;  // read by every thread well before a build clears it
    group_delete_move<G>(pool, off, deg, del_pos + s, k, lane);
    for (uint32_t c = lane; c <= g.nc; c += G) {
      const uint32_t sub = lower_bound_u64(del_key, s, s + k, g.kb.pack(x, 0, 0) + ((uint64_t)c << g.kb.yb)) - s;
      dirx[c] -= sub;
    }
    group_sync<G>();
    if (tomb > tomb_limit(row.y)) {
      row_table_build<G>(g, pool, x, row, dirx, deg - k, lane);
      group_sync<G>();
    }
  }
}

// Both row kinds in one launch: the first warp_blocks blocks take the rows of
// up to kBigRow entries warp by warp, the others the longer rows.
__global__ void __launch_bounds__(256) k_mut_insert(const VRange* ranges, const unsigned int* n_ranges,
                                                    const uint64_t* ins_key, uint32_t* ins_dst, DevGraph g,
                                                    uint32_t warp_blocks) {
  __shared__ unsigned long long s_off[8];
  if (blockIdx.x < warp_blocks)
    mut_insert<32>(ranges, *n_ranges, ins_key, ins_dst, g, s_off, blockIdx.x, warp_blocks);
  else
    mut_insert<256>(ranges, *n_ranges, ins_key, ins_dst, g, s_off, blockIdx.x - warp_blocks, gridDim.x - warp_blocks);
}
__global__ void __launch_bounds__(256) k_mut_delete(const VRange* ranges, const unsigned int* n_ranges,
                                                    const uint64_t* del_key, uint32_t* del_pos, DevGraph g,
                                                    uint32_t warp_blocks) {
  if (blockIdx.x < warp_blocks)
    mut_delete<32>(ranges, *n_ranges, del_key, del_pos, g, blockIdx.x, warp_blocks);
  else
    mut_delete<256>(ranges, *n_ranges, del_key, del_pos, g, blockIdx.x - warp_blocks, gridDim.x - warp_blocks);
}

void launch_mut_insert(const VRange* ranges, const unsigned int* n_ranges, const uint64_t* ins_key,
                       uint32_t* ins_dst, const DevGraph& g, uint32_t warp_blocks, uint32_t big_blocks,
                       cudaStream_t st) {
  k_mut_insert<<<warp_blocks + big_blocks, 256, 0, st>>>(ranges, n_ranges, ins_key, ins_dst, g, warp_blocks);
}
void launch_mut_delete(const VRange* ranges, const unsigned int* n_ranges, const uint64_t* del_key,
                       uint32_t* del_pos, const DevGraph& g, uint32_t warp_blocks, uint32_t big_blocks,
                       cudaStream_t st) {
  k_mut_delete<<<warp_blocks + big_blocks, 256, 0, st>>>(ranges, n_ranges, del_key, del_pos, g, warp_blocks);
}

// ------------------------------------------------- one update per launch
//
// The plain form runs each edge update on its own.  A batch of one needs no
// sorting, no grouping by edge and no temporal entries: an insertion is
// searched after its edge is added and a deletion before its edge is
// removed, so the graph at search time is the sequential one.  Its
// preparation is one kernel and its row mutation another (plus the
// compaction copy when an insertion's relocation does not fit).

// One warp: the labels an edge may have are looked up side by side (one thread
// trying them in turn took 5.4 us).
__global__ void k_plain_resolve(const csm_update* up, DevGraph g, UpdInfo* info, uint64_t* keys, unsigned int* cnt,
                                unsigned long long* count, unsigned long long* hash, unsigned long long* bytes,
                                unsigned int* stop, unsigned long long* stamp) {
  const uint32_t lane = threadIdx.x;
  if (stamp && lane == 0) {
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    stamp[0] = now;
  }
  const csm_update u = *up;
  PoolState* ps = g.ps;
  const bool ids = u.type == 'e' && u.id1 < g.n && u.id2 < g.n && u.id1 != u.id2;
  const uint32_t x = min(u.id1, u.id2), y = max(u.id1, u.id2);
  uint32_t lx = kNone, ly = kNone;
  if (ids) { lx = g.vlabel[x]; ly = g.vlabel[y]; }
  const bool ok = ids && lx != kNone && ly != kNone;
  if (lane < 16) cnt[lane] = 0;
  uint32_t l0 = kNone;
  if (ok) {
    const uint2 rx = g.row[x];
    const uint32_t* pool = g.pools[ps->active];
    for (uint32_t base = 0; base < g.n_el; base += 32) {
      const uint32_t l = base + lane;
      bool found = false;
      if (l < g.n_el) {
        if (g.htab) {
          found = row_find(g, rx, row_entry(y, l, g.hlb)) != kSlotEmpty;
        } else {
          uint64_t lo, hi;
          segment(g, x, ly * g.n_el + l, lo, hi);
          found = contains_u32(pool, lo, hi, y);
        }
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, found);
      if (hit) { l0 = base + (uint32_t)__ffs((int)hit) - 1u; break; }
    }
  }
  UpdInfo inf;
  inf.v1 = u.id1; inf.v2 = u.id2; inf.label = fold_elabel(g, u.label); inf.flags = 0;
  if (u.type == 'e') {
    if (!ok) inf.flags = UF_INVALID;
    else if (u.is_add)  // an edge that is there: graph unchanged, counted with the given label
      inf.flags = UF_VALID | UF_ADD | (l0 != kNone ? UF_DUP : UF_MUT);
    else if (l0 == kNone)
      inf.flags = UF_VALID | UF_INVALID;  // deleting a missing edge
    else {
      inf.label = l0;  // a deletion counts with the edge's own label
      inf.flags = UF_VALID | UF_MUT;
    }
  }
  unsigned long long need = 0;
  if (lane < 2 && (inf.flags & UF_MUT) && u.is_add) {
    const uint32_t v = lane ? y : x;
    const uint32_t deg = g.dir[(size_t)v * (g.nc + 1) + g.nc];
    if (deg + 1 > g.row[v].y) need = grow_cap(deg + 1, g.htab);
  }
  need += __shfl_xor_sync(0xffffffffu, need, 1);
  if (lane == 0) {
    const bool mut = (inf.flags & UF_MUT) != 0;
    keys[0] = mut ? g.kb.pack(x, ly * g.n_el + inf.label, y) : ~0ULL;
    keys[1] = mut ? g.kb.pack(y, lx * g.n_el + inf.label, x) : ~0ULL;
    count[0] = 0; hash[0] = 0; bytes[0] = 0; stop[0] = 0;
    ps->compact = need > g.pool_cap - ps->top[ps->active] ? 1u : 0u;
    info[0] = inf;
  }
}

// One block per row (the two ends of the edge).
__global__ void __launch_bounds__(256) k_plain_mutate(DevGraph g, const UpdInfo* info, const uint64_t* keys,
                                                      csm_result* out, const unsigned long long* stamp,
                                                      uint32_t mut_bytes) {
  PoolState* ps = g.ps;
  const uint32_t lane = threadIdx.x;
  __shared__ unsigned long long s_off;
  __shared__ uint32_t s_pos;
  const UpdInfo inf = info[0];
  if (inf.flags & UF_MUT) {
    uint32_t* pool = g.pools[ps->active];
    const uint64_t key = keys[blockIdx.x];
    const uint32_t x = g.kb.x_of(key), c = g.kb.c_of(key), y = g.kb.y_of(key);
    uint32_t* dirx = g.dir + (size_t)x * (g.nc + 1);
    const uint32_t deg = dirx[g.nc];
    const uint2 old = g.row[x];
    const uint64_t off = old.x;
    const uint32_t entry = row_entry(y, c % g.n_el, g.hlb);
    const uint32_t tomb = g.htab ? g.htomb[x] : 0u;  // read by every thread before a build clears it
    const bool add = (inf.flags & UF_ADD) != 0;
    uint32_t new_cap = 0;
    if (lane < 32) {
      const uint32_t end = dirx[c + 1];
      const uint32_t p = warp_lower_bound(pool + off, dirx[c], end, y, lane);
      if (lane == 0) s_pos = !add && (p >= end || pool[off + p] != y) ? kNone : p;  // a deleted entry must be there
    }
    if (add && deg + 1 > old.y) {
      new_cap = grow_cap(deg + 1, g.htab);
      if (lane == 0) {
        unsigned long long o = atomicAdd(&ps->top[ps->active], (unsigned long long)new_cap);
        if (o + new_cap > g.pool_cap) { atomicExch(&ps->error, kErrPoolFull); o = ~0ULL; }
        s_off = o;
      }
    }
    __syncthreads();
    const uint32_t p = s_pos;
    const uint64_t dst = new_cap ? s_off : off;
    if (p == kNone) {
      if (lane == 0) atomicExch(&ps->error, kErrRowState);
    } else if (add && dst != ~0ULL) {
      const uint2 now = new_cap ? make_uint2((uint32_t)dst, new_cap) : old;
      group_insert_move<256>(pool, off, dst, new_cap ? 0u : p, deg, &s_pos, 1, lane);
      if (lane == 0) pool[dst + p] = y;
      for (uint32_t cc = c + 1 + lane; cc <= g.nc; cc += 256) dirx[cc] += 1;
      if (lane == 0 && new_cap) g.row[x] = now;
      __syncthreads();
      if (g.htab) {  // the row table follows, as in mut_insert
        if (new_cap || deg + 1 + tomb > now.y + now.y / 2)
          row_table_build<256>(g, pool, x, now, dirx, deg + 1, lane);
        else if (lane == 0)
          row_table_insert(g, now, entry);
      }
    } else if (!add) {
      group_delete_move<256>(pool, off, deg, &s_pos, 1, lane);
      for (uint32_t cc = c + 1 + lane; cc <= g.nc; cc += 256) dirx[cc] -= 1;
      __syncthreads();
      if (g.htab) {
        if (tomb + 1 > tomb_limit(old.y))
          row_table_build<256>(g, pool, x, old, dirx, deg - 1, lane);
        else if (lane == 0)
          row_table_delete(g, x, old, entry);
      }
    }
  }
  if (out && blockIdx.x == 0 && lane == 0) {
    // an update whose label triple matches no query edge: nothing to count
    csm_result r;
    r.pos = 0; r.neg = 0; r.hash = 0;
    r.status = (inf.flags & UF_INVALID) ? CSM_ST_INVALID : CSM_ST_OK;
    r.safe = 1;
    r.work_bytes = (inf.flags & UF_MUT) ? (unsigned long long)mut_bytes : 0ull;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    r.latency_ns = stamp ? t - stamp[0] : 0ull;
    out[0] = r;
  }
}

// Vertex deletion: the packed keys of every directed entry incident to v,
// (v, combo, y) and (y, combo', v), for the deletion kernels.
__global__ void k_vdel_keys(DevGraph g, uint32_t v, uint32_t deg, uint64_t* keys) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= deg) return;
  const uint32_t* pool = g.pools[g.ps->active];
  const uint32_t* dirv = g.dir + (size_t)v * (g.nc + 1);
  const uint32_t y = pool[(uint64_t)g.row[v].x + i];
  const uint32_t c = combo_at(dirv, g.nc, i);
  const uint32_t el = c % g.n_el;
  keys[2 * i] = g.kb.pack(v, c, y);
  keys[2 * i + 1] = g.kb.pack(y, g.vlabel[v] * g.n_el + el, v);
}

// Vertex insertion (Graph::AddVertex, ParaCOSM/CSM/graph/graph.cpp:23-49): sets
// the label of an absent vertex slot.  A deletion of an id beyond the
// vertex slots is invalid; other deletions are applied by the caller.
__global__ void k_vertex_update(const csm_update* ups, uint32_t B, DevGraph g, UpdInfo* info) {
  uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= B) return;
  const csm_update u = ups[s];
  if (u.type != 'v') return;
  UpdInfo inf;
  inf.v1 = u.id1; inf.v2 = 0; inf.label = u.label; inf.flags = 0;
  if (u.is_add && u.id1 < g.n_cap) {
    if (g.vlabel[u.id1] == kNone) g.vlabel[u.id1] = fold_vlabel(g, u.label);
  } else if (u.is_add || u.id1 >= g.n) {
    inf.flags = UF_INVALID;
  }
  info[s] = inf;
}

}  // namespace csm
