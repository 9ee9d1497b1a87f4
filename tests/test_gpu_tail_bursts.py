"""Tail stages take the entries of the tail's level in bursts when results are capped: entry counts around the
bursts' and a level's sizes, caps below, at and above the counts."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu

# a - b - c with leaves d, d', e at c: the leaves are the tail, c's matches the entries before it
QUERY = ([0, 1, 2, 3, 3, 4], [(0, 1, 0), (1, 2, 0), (2, 3, 0), (2, 4, 0), (2, 5, 0)])


@pytest.mark.parametrize("homo", [False, True])
@pytest.mark.parametrize("mode", ["batched", "plain"])
@pytest.mark.parametrize("entries", [1, 7, 8, 9, 23, 24, 25, 31, 32, 33, 56, 57, 100])
def test_bursts(entries, mode, homo):
    rng = np.random.default_rng(entries)
    d0, e0 = 2 + entries, 2 + entries + 40
    vl = np.array([0, 1] + [2] * entries + [3] * 40 + [4] * 40, np.uint32)
    edges = [(1, 2 + i, 0) for i in range(entries)]
    for i in range(entries):
        for base in (d0, e0):
            edges += [(2 + i, int(v), 0) for v in base + rng.permutation(40)[: int(rng.integers(0, 6))]]
    edges = np.array(edges, np.uint32)
    ups = np.zeros(2, UPDATE_DTYPE)
    ups["type"], ups["id2"], ups["is_add"] = ord("e"), 1, (1, 0)
    true = int(pyoracle.run(*QUERY, vl, edges, ups, homo=homo, want_hash=False)["pos"][0])
    for cap in (0, 1, max(1, true // 2), max(1, true - 1), max(1, true), true + 1, 1_000_000):
        with Engine("parallel_symbi", max_results=cap, mode=mode, homo=homo) as eng:
            eng.set_query(*QUERY)
            eng.load_graph(vl, edges)
            eng.build_index()
            r = eng.run(ups)
            assert eng.initial_match() == 0
        want = min(cap, true) if cap else true
        assert r["pos"][0] == want and r["neg"][1] == want, (cap, true)
        assert (r["status"] == (1 if cap and true >= cap else 0)).all()
