// Host-side helpers shared by the engine's translation units: error text and
// device allocations tracked against the context's HBM budget.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

#include "../../include/csm_gpu.h"

namespace csm {

int set_err(int code, const char* fmt, ...);

struct DevMem {
  std::vector<void*> ptrs;
  uint64_t bytes = 0, budget = 0;
  int alloc(void** p, size_t sz) {
    sz = std::max<size_t>(sz, 16);
    if (budget && bytes + sz > budget)
      return set_err(CSM_ENOMEM, "HBM budget of %llu bytes exceeded", (unsigned long long)budget);
    cudaError_t e = cudaMalloc(p, sz);
    if (e != cudaSuccess) {
      cudaGetLastError();  // a caller that does without must not find it after its next launch
      return set_err(CSM_ENOMEM, "cudaMalloc(%zu): %s", sz, cudaGetErrorString(e));
    }
    ptrs.push_back(*p);
    bytes += sz;
    return CSM_OK;
  }
  void release(void* p, size_t sz) {
    if (!p) return;
    for (size_t i = 0; i < ptrs.size(); i++)
      if (ptrs[i] == p) { ptrs.erase(ptrs.begin() + (long)i); break; }
    cudaFree(p);
    bytes -= std::min<uint64_t>(bytes, std::max<size_t>(sz, 16));
  }
  void free_all() {
    for (void* p : ptrs) cudaFree(p);
    ptrs.clear();
    bytes = 0;
  }
};

// Several arrays in one device allocation (an allocation and its release cost
// 0.1 ms each, and setting a context up took 62 of them).
struct DevBlock {
  std::vector<std::pair<void**, size_t>> parts;  // pointer to set, offset
  size_t total = 0;
  template <class T>
  void add(T*& p, size_t bytes) {
    parts.emplace_back(reinterpret_cast<void**>(&p), total);
    total += (std::max<size_t>(bytes, 16) + 255) & ~(size_t)255;
  }
  int alloc(DevMem& mem, void** base) {
    const int rc = mem.alloc(base, total);
    if (rc) return rc;
    for (auto& q : parts) *q.first = static_cast<unsigned char*>(*base) + q.second;
    return CSM_OK;
  }
};

// Slots of a row pool, and whether the rows have tables.  `with` and `without`:
// slots of the loaded rows with capacities in multiples of four, as tables need
// them, and as they come; `entries_fit`: an id and a label fit in a table entry.
struct PoolPlan {
  bool ok, tables;
  uint64_t cap;
};
inline PoolPlan pool_plan(uint64_t with, uint64_t without, uint32_t max_batch, bool entries_fit) {
  constexpr uint64_t kLimit = 1ull << 32;  // offsets have 32 bits
  const uint64_t room = 16ull * max_batch + (1ull << 20), plain = 2 * without + room;
  if (plain >= kLimit) return {false, false, 0};
  // rounding may not take the room to grow: a pool cut off at the limit has to
  // keep as many free slots as without tables
  const uint64_t cap = std::min(2 * with + room, kLimit - 4);
  if (entries_fit && cap >= with + (plain - without)) return {true, true, cap};
  return {true, false, plain};
}

}  // namespace csm
