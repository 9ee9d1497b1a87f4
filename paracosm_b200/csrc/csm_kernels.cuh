// Kernel entry points of the engine (defined in csm_kernels.cu and
// csm_search.cu), launched by the context in csm_api.cu.
#pragma once
#include "csm_internal.cuh"

namespace csm {

// A run of consecutive entries of one vertex in a sorted packed-key list.
struct VRange {
  uint32_t x, start, count, pad;
};

// ---- load-time CSR build (csm_kernels.cu) ----
__global__ void k_load_edge_keys(const uint32_t* e, uint64_t m, const uint32_t* vlabel, uint32_t n,
                                 uint64_t* key, uint64_t* idx, unsigned long long* bad);
__global__ void k_fold_vlabels(uint32_t* vlabel, uint32_t n, DevGraph g);
__global__ void k_load_directed(const uint64_t* ukey, const uint64_t* uidx, uint64_t m, const uint32_t* e,
                                DevGraph g, uint64_t* dkey);
__global__ void k_load_count(const uint64_t* dkey, uint64_t M, KeyBits kb, uint32_t nc, uint32_t* dir,
                             uint64_t* first, unsigned long long* n_valid);
// Row capacities for a graph with row tables or without, and the sums of both
// (sums[0]: with, sums[1]: without).
__global__ void k_load_caps(const uint32_t* dir, uint32_t n_cap, uint32_t nc, uint32_t tables, uint64_t* cap64,
                            unsigned long long* sums);
__global__ void k_load_rows(const uint32_t* dir, uint32_t n_cap, uint32_t nc, uint32_t tables, uint2* row);
__global__ void k_load_scatter(const uint64_t* dkey, uint64_t M, const uint64_t* first, DevGraph g, uint32_t* pool);
__global__ void k_dir_scan(uint32_t* dir, uint32_t n_cap, uint32_t nc);

// ---- batch preparation ----
// ukey: the update's edge (smaller end, larger end; yb bits each), for sorting;
// cnt[0..15] cleared.
__global__ void k_batch_init(const csm_update* ups, uint32_t B, DevGraph g, uint64_t* ukey, uint32_t* useq,
                             UpdInfo* info, unsigned int* cnt);
struct ResolveOut {
  uint64_t* ins_key; unsigned int* n_ins;
  uint64_t* del_key; unsigned int* n_del;
  uint64_t* t_key; uint64_t* t_span; unsigned int* n_t;
  uint32_t cap;  // capacity of each list
};
__global__ void k_resolve(const uint64_t* skey, const uint32_t* sseq, uint32_t B, DevGraph g,
                          const csm_update* ups, UpdInfo* info, ResolveOut out);
constexpr uint32_t kBigRow = 4096;  // rows longer than this are mutated by a whole block
__global__ void k_ranges(const uint64_t* key, uint32_t cap, KeyBits kb, VRange* ranges, unsigned int* n_ranges,
                         const uint32_t* dir, uint32_t nc);
__global__ void k_temporal_set(uint32_t L, DevGraph g);
__global__ void k_temporal_clear(uint32_t L, DevGraph g);
// Slots of the temporal table (DevGraph::t_tab) for a batch of B updates: a
// power of two, at most a quarter full (two directed entries an update, and a
// head for each of their segments).
__host__ __device__ inline uint32_t temporal_slots(uint32_t B) {
  uint32_t s = 64;
  while (s < 16u * B) s <<= 1;
  return s;
}
__global__ void k_reloc_need(const VRange* ranges, const unsigned int* n_ranges, DevGraph g);
// Lists that k_sort_block sorts, one block each: job.n keys of job.bits bits to
// out (stable; unused slots, all ones, come out as job.bits ones); pos: where to
// put each key's place in the list, or null; val: moved along to val_out, or
// null.  A list fits when n <= kSortMax and bits <= kSortMaxBits.
constexpr uint32_t kSortMax = 9 * 1024;  // the lists of a batch of 4,096
constexpr uint32_t kSortPosBits = 14;    // > log2(kSortMax)
constexpr uint32_t kSortMaxBits = 64 - kSortPosBits;
struct SortJob {
  const uint64_t* key;
  uint64_t* out;
  uint32_t* pos;
  const uint64_t* val;
  uint64_t* val_out;
  uint32_t n, bits;
};
struct SortJobs { SortJob job[3]; };
cudaError_t launch_sort_block(const SortJobs& jobs, uint32_t n_jobs, cudaStream_t st);
__global__ void k_compact_copy(DevGraph g);
void launch_mut_insert(const VRange* ranges, const unsigned int* n_ranges, const uint64_t* ins_key,
                       uint32_t* ins_dst, const DevGraph& g, uint32_t warp_blocks, uint32_t big_blocks,
                       cudaStream_t st);
void launch_mut_delete(const VRange* ranges, const unsigned int* n_ranges, const uint64_t* del_key,
                       uint32_t* del_pos, const DevGraph& g, uint32_t warp_blocks, uint32_t big_blocks,
                       cudaStream_t st);
__global__ void k_vdel_keys(DevGraph g, uint32_t v, uint32_t deg, uint64_t* keys);

// ---- one edge update per launch sequence (the plain form; csm_kernels.cu) ----
// keys[0..1]: the update's two directed entries (sentinels when the graph does
// not change); cnt[0..15], count/hash/bytes/stop[0]: cleared for the search;
// stamp[0] (unless null): the time.
__global__ void k_plain_resolve(const csm_update* up, DevGraph g, UpdInfo* info, uint64_t* keys, unsigned int* cnt,
                                unsigned long long* count, unsigned long long* hash, unsigned long long* bytes,
                                unsigned int* stop, unsigned long long* stamp);
// Applies the update's row insertion or deletion (two 256-thread blocks); with
// `out`, also writes the result of an update that needs no search (latency
// from stamp[0]).
__global__ void k_plain_mutate(DevGraph g, const UpdInfo* info, const uint64_t* keys, csm_result* out,
                               const unsigned long long* stamp, uint32_t mut_bytes);
__global__ void k_vertex_update(const csm_update* ups, uint32_t B, DevGraph g, UpdInfo* info);

// ---- search (csm_search.cu) ----
// Donated search task: a partial match of positions 0..depth (depth 1 = the
// updated edge itself) and the driver range of position depth + 1.
struct DTask {
  uint32_t upd;
  uint16_t anchor;
  uint8_t orient;
  uint8_t depth;
  uint32_t dlo, dn;
  uint32_t sel;  // driver and first join (back entries; LevelSM::dsel, jsel in bits 8 and up)
  uint32_t m[kMaxQ];
  uint32_t pad[3];
};
static_assert(sizeof(DTask) == 160, "DTask is 160 bytes");

// Work queue of the search launches.  Tickets count up across launches: an
// idle warp takes ticket `head` (fetch-and-add) and waits for its record; a
// busy warp hands work over by filling tickets from `tail`, one per unit of
// `hungry` it takes (a signed count of idle warps not yet promised a record),
// so records go to waiting warps in ticket order and tail never passes head.
// `pending` counts this launch's tasks (root and donated) that are not
// finished, and waiting warps exit when it reaches zero.
// The words lie on cache lines of their own: waiting warps read `pending` all
// the time, busy ones read and write the others.
struct SearchQueue {
  alignas(128) unsigned long long head;
  alignas(128) unsigned long long tail;
  alignas(128) unsigned int hungry;
  alignas(128) unsigned int pending;
};

// Cumulative search counters (device memory, read by csm_gpu_stats).
struct SearchStats {
  unsigned long long busy_ns;    // warp time spent inside tasks
  unsigned long long idle_ns;    // warp time spent waiting for handed-over tasks
  unsigned long long iters;      // chunk iterations (32 candidate slots each)
  unsigned long long donations;  // hand-overs (one or more tasks each)
  unsigned long long starved;    // idle warps existed but nothing could be handed over
  unsigned long long checks;     // hand-over checks made by busy warps
  unsigned long long checks_hungry;  // ... that saw idle warps waiting
  unsigned long long root_busy_ns;   // warp time in root tasks (the rest is handed-over tasks)
  unsigned long long last_root_ns;   // max over warps: kernel start -> end of its last root task
  unsigned long long max_task_ns;    // longest single task
  unsigned long long launch_t0;      // globaltimer at the start of the current launch
  // first malformed handed-over record seen: ticket, observed sequence, words 0..4, batch
  unsigned long long bad_ticket, bad_seq;
  unsigned int bad_words[5], bad_batch;
  unsigned int bad_set, pad_;
  // first task stopped by the task time guard: its depth, iterations, update and level cursors
  unsigned int guard_set, guard_d, guard_upd, guard_pad;
  unsigned long long guard_iters;
  unsigned int guard_lv[4 * 16];  // per level 1..16: cnt, cur, total, incl[0]
};

// What the results of a batch's updates are made of.
struct ResultArgs {
  const UpdInfo* info;
  const unsigned long long *count, *hash, *bytes;
  const uint32_t* safe;
  const unsigned int* stop;
  uint64_t cap;
  int want_hash;
  csm_result* out;
  uint32_t mut_bytes;               // bytes of an applied mutation (0 on secondary shards)
  const unsigned long long* stamp;  // non-null: latency from stamp[0]
};

struct SearchParams {
  DevGraph g;
  const Plan* plan;
  const Task* tasks;
  const unsigned int* n_tasks;
  uint32_t task_cap;
  unsigned int* task_next;
  const UpdInfo* info;
  unsigned long long* count;   // per update of the batch
  unsigned long long* hash;    // per update of the batch
  unsigned long long* bytes;   // per update: algorithmic bytes of the expanded nodes
  unsigned int* stop;          // per update: cap reached
  const uint64_t* d2;          // optional candidate filter bitsets [n_q][d2_words]
  uint64_t d2_words;
  uint64_t cap;                // 0 = none
  int homo;
  int want_hash;
  unsigned int* error;
  // work donation (null dq: off)
  SearchQueue* q;
  DTask* dq;                  // ring of qcap slots (a power of two)
  unsigned long long* qseq;   // per-slot sequence numbers
  uint32_t qcap;
  unsigned long long wait_limit_ns;  // idle warps waiting for work
  unsigned long long slot_limit_ns;  // a hand-over waiting for its ring slot
  unsigned long long task_limit_ns;  // one task (a guard: a correct walk always ends)
  uint32_t batch;             // updates in this batch (bound of task update indices)
  SearchStats* sstat;
  unsigned long long deadline_ns;  // per-update time budget from the launch's start; 0 = none
  // hand-over tuning: busy warps look for idle ones every donate_every
  // iterations (a power of two; 0 = every iteration) and split a driver range deep in the
  // tree only when at least split_deep elements remain (0 = 64)
  uint32_t donate_every, split_deep;
  // match-set output (null: off): each embedding found at a leaf is appended
  // as a record of 1 + n_q words (enum_base + its update's batch index, then
  // the data vertex of every query vertex in query-vertex order) while fewer
  // than enum_cap records exist; enum_n counts every embedding found
  uint32_t* enum_buf;
  unsigned long long* enum_n;
  unsigned long long enum_cap;
  uint32_t enum_base, enum_stride;
  // nonzero: count each anchor's independent tail (PlanAnchor::tail_at)
  // instead of enumerating it; only for counts without hashes or match sets.
  // The value is the entries that the first tail stage of a task takes (tail_first)
  uint32_t tail;
  uint32_t levels, warp_bytes;  // SearchShape
  // non-null result.out: the launch's last block writes the batch's results
  // (a launch less; for a few updates, which one block writes in no time)
  ResultArgs result;
  unsigned int* ended;          // blocks that have ended; 0 between launches
};
// Entries of the tail's level that the first tail stage of a task takes; every
// further one takes twice as many, up to 32.  With a cap a few entries may be all
// it takes, and a stage lists every candidate of the tail's members for all of
// its entries: with all 32 from the start, the counting of 1,500 updates capped
// at 10,000 under 24- to 32-vertex queries took 3 to 14 ms, with eight 2 to 6
// (of 24-vertex homomorphisms 2.3 to 3.1 ms, 1.6), where a batch of 4,097 updates
// whose prefixes mostly die takes 1 % longer (with one, 1.2 ms and 3 %).
__host__ __device__ constexpr uint32_t tail_first(uint64_t cap) { return cap ? 8u : 32u; }
constexpr uint32_t kFuseResults = 1024;  // updates of a batch up to which it does
// Per-update counters of a search.
struct Counters {
  unsigned long long *count, *hash, *bytes;
  unsigned int* stop;
};
// Root tasks of B updates; clears their counters.
__global__ void k_seed(uint32_t B, const UpdInfo* info, DevGraph g, const Plan* plan, const uint64_t* d2,
                       uint64_t d2_words, Task* tasks, unsigned int* n_tasks, uint32_t task_cap,
                       uint32_t* safe, unsigned int* error, Counters ctr, uint32_t shard_rank = 0, uint32_t shard_count = 1,
                       uint32_t turboflux_compat = 0, uint32_t dup_zero = 0, SearchQueue* q = nullptr,
                       SearchStats* ss = nullptr);
// mode: 0 plain, 1 match sets, 2 tail counting
struct SearchShape {
  uint32_t levels;      // levels of a warp's walk
  uint32_t warp_bytes;  // shared memory of a warp
  bool general;         // instantiation (search_general)
};
SearchShape search_shape_of(const Plan& plan, int mode, const DevGraph& g);
uint32_t search_max_blocks(const SearchShape& shape, uint32_t warps, int mode);
int search_mode(const SearchParams& p);
// `prepared`: k_seed has prepared the queue.
void launch_search(const SearchParams& p, uint32_t blocks, uint32_t warps, cudaStream_t s, bool prepared = false);
__global__ void k_finalize(uint32_t B, ResultArgs a);
// stop[] values: 1 = the cap was reached, 2 = the deadline passed first
constexpr unsigned int kStopCap = 1u, kStopDeadline = 2u;
__global__ void k_classify(uint64_t n, const csm_update* ups, DevGraph g, const Plan* plan, uint8_t* safe);

}  // namespace csm
