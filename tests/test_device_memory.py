"""csm::DevMem, compiled here over a stand-in CUDA runtime whose allocations fail on request: a failed allocation
leaves nothing behind, neither in the accounting nor as the runtime's last error (callers that do without the
memory -- row tables, InitialMatching's seed buffers -- would report it after their next launch)."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

from paracosm_b200 import build

SOURCE = r"""
#include <cassert>
#include <cstdarg>
#include <cstdlib>
#include "csm_host.cuh"
static cudaError_t last = cudaSuccess;
static bool fail = false;
extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
  if (fail) return last = cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "error"; }
namespace csm { int set_err(int code, const char*, ...) { return code; } }
int main() {
  csm::DevMem m;
  m.budget = 1000;
  void *a = nullptr, *b = nullptr;
  if (m.alloc(&a, 600) != CSM_OK || m.bytes != 600) return 1;
  if (m.alloc(&b, 600) != CSM_ENOMEM || m.bytes != 600) return 2;  // the budget
  fail = true;
  if (m.alloc(&b, 100) != CSM_ENOMEM || m.bytes != 600 || m.ptrs.size() != 1) return 3;  // the device
  if (cudaGetLastError() != cudaSuccess) return 4;
  fail = false;
  csm::DevBlock blk;
  int *x = nullptr, *y = nullptr;
  blk.add(x, 4);
  blk.add(y, 4);
  if (blk.alloc(m, &b) != CSM_ENOMEM || x || y) return 5;  // 512 bytes do not fit
  m.release(a, 600);
  if (m.bytes != 0 || blk.alloc(m, &b) != CSM_OK || y - x != 64 || m.bytes != 512) return 6;
  m.free_all();
  return m.bytes != 0;
}
"""


def test_failed_allocations_leave_nothing_behind(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    cuda = Path(os.path.realpath(build.NVCC)).parents[1] / "include"
    subprocess.run([build.CXX, "-std=c++17", f"-I{build.CSRC}", f"-I{cuda}", "-o", str(exe), str(src)], check=True,
                   capture_output=True, text=True)
    assert subprocess.run([str(exe)]).returncode == 0
