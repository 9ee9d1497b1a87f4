"""csm::pool_plan: how large the row pools are and whether rows have tables, compiled here as it stands."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

import pytest

from paracosm_b200 import build

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "csm_host.cuh"
namespace csm { int set_err(int code, const char*, ...) { return code; } }
int main(int, char** a) {
  const csm::PoolPlan p = csm::pool_plan(std::strtoull(a[1], 0, 10), std::strtoull(a[2], 0, 10),
                                         (uint32_t)std::atoi(a[3]), a[4][0] == '1');
  std::printf("%d %d %llu\n", p.ok, p.tables, (unsigned long long)p.cap);
}
extern "C" cudaError_t cudaMalloc(void**, size_t) { return cudaSuccess; }
extern "C" cudaError_t cudaFree(void*) { return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return ""; }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "t.cpp").write_text(MAIN)
    cuda = Path(os.path.realpath(build.NVCC)).parents[1] / "include"
    subprocess.run([build.CXX, "-std=c++17", f"-I{build.CSRC}", f"-I{cuda}", "-o", str(d / "t"), str(d / "t.cpp")],
                   check=True, capture_output=True, text=True)

    def run(rows, degree, batch=65536, fit=True):
        cap = degree + max(2, degree // 4)
        args = [rows * ((cap + 3) // 4 * 4), rows * cap, batch, int(fit)]
        ok, tables, slots = subprocess.check_output([str(d / "t")] + [str(x) for x in args], text=True).split()
        return bool(int(ok)), bool(int(tables)), int(slots)

    return run


ROOM = 16 * 65536 + (1 << 20)


def test_ordinary_graphs_have_tables(plan):
    assert plan(1 << 20, 3) == (True, True, 2 * 8 * (1 << 20) + ROOM)
    assert plan(0, 0, batch=1) == (True, True, 16 + (1 << 20))
    assert plan(1 << 20, 3, fit=False) == (True, False, 2 * 5 * (1 << 20) + ROOM)


def test_rounding_refuses_no_graph(plan):
    """Rows of degree 3 take 5 slots, with tables 8: what fits without tables is loaded."""
    assert plan(1 << 28, 3) == (True, True, (1 << 32) - 4)  # cut off at the limit, with room to grow
    n = 340_000_000  # the limit would leave less room than rows without tables have
    assert plan(n, 3) == (True, False, 10 * n + ROOM)
    most = ((1 << 32) - 1 - ROOM) // 10  # the last that fits at all
    assert plan(most, 3) == (True, False, 10 * most + ROOM)
    assert not plan(most + 1, 3)[0]


@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 7, 9, 33, 1000])
def test_room_to_grow(plan, degree):
    cap = degree + max(2, degree // 4)
    for rows in (1, 1000, 10**6, ((1 << 31) - (1 << 21)) // cap, (1 << 30) // cap, 3 * (1 << 29) // cap):
        ok, tables, slots = plan(rows, degree)
        assert ok and slots < 1 << 32
        used = rows * ((cap + 3) // 4 * 4 if tables else cap)
        assert slots - used >= rows * cap + ROOM
        assert not tables or slots % 4 == 0
