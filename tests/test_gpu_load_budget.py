"""Loading with little device memory: what the row tables add -- themselves, row capacities in multiples of four,
long work lists of the index -- is left out before a graph is refused."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu

QUERY = ([0, 1, 0, 1], [(0, 1, 0), (1, 2, 0), (2, 3, 0), (3, 0, 0)])


def degree_three(n):
    vl = (np.arange(n) % 2).astype(np.uint32)
    i = np.arange(n, dtype=np.uint32)
    h = i[: n // 2]
    edges = np.concatenate([np.stack([i, (i + 1) % n], 1), np.stack([h, h + n // 2], 1)])
    return vl, np.concatenate([edges, 0 * edges[:, :1]], 1).astype(np.uint32)


def stream(rng, n, m):
    """Edges come and go at few vertices, so that rows grow past their capacity."""
    ups = np.zeros(m, UPDATE_DTYPE)
    ups["type"] = ord("e")
    present = set()
    for u in ups:
        a, b = 2 * int(rng.integers(0, 20)), 2 * int(rng.integers(0, 20)) + 1
        if abs(a - b) in (1, n - 1):
            b = (b + 40) % n | 1
        if (a, b) in present and rng.random() < 0.6:
            present.discard((a, b))
        else:
            u["is_add"] = 1
            present.add((a, b))
        u["id1"], u["id2"] = a, b
    return ups


@pytest.mark.parametrize("algo,kw", [("parallel_graphflow", {}), ("parallel_symbi", {}), ("parallel_symbi", {"mode": "plain"})])
def test_tables_and_lists_are_left_out_first(algo, kw):
    n, batch = 100_000, 64
    vl, edges = degree_three(n)
    ups = stream(np.random.default_rng(11), n, 300)
    ref = pyoracle.run(*QUERY, vl, edges, ups)
    assert ref["pos"].sum() > 0

    def run(budget):
        with Engine(algo, want_hash=True, max_batch=batch, hbm_budget_bytes=budget, **kw) as eng:
            eng.set_query(*QUERY)
            eng.load_graph(vl, edges)
            eng.build_index()
            res = eng.run(ups)
            for f in ("pos", "neg", "hash"):
                assert np.array_equal(res[f], ref[f]), f
            st = eng.stats()
            return st["device_bytes"], st["pool_capacity"]

    room = 16 * (1 if kw else batch) + (1 << 20)
    full, slots = run(0)
    assert slots == 2 * 8 * n + room  # five slots a row, rounded to eight
    bare, slots2 = run(full - 4 * slots)
    assert slots2 == 2 * 5 * n + room  # no tables, no rounding
    assert bare < full - 8 * slots
    if algo != "parallel_graphflow":
        lists = 4 * 2 * 4 * 32768
        tight, slots3 = run(bare - lists // 2)
        assert slots3 == slots2 and tight < bare - lists // 2
