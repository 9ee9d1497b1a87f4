"""The row tables and the search over them where they can go wrong: rows around a bucket's and a row's
capacity, rows that move, deleted slots, edge-label counts around the entry's width, the join without tables,
and walks whose candidates fill the waiting buffer.  Counts and hashes are exact (the oracle's)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu


def updates(rows) -> np.ndarray:
    u = np.zeros(len(rows), UPDATE_DTYPE)
    u["type"] = ord("e")
    for i, (add, a, b, l) in enumerate(rows):
        u[i]["is_add"], u[i]["id1"], u[i]["id2"], u[i]["label"] = add, a, b, l
    return u


def hub_case(rng, n_v, hub_deg, n_el, n_updates):
    """A hub joined to hub_deg vertices over a sparse random graph, and a stream that inserts and deletes
    edges at the hub (its row grows past its capacity and loses entries) and elsewhere."""
    vl = rng.integers(0, 3, n_v).astype(np.uint32)
    present = {}
    for v in rng.permutation(np.arange(1, n_v))[:hub_deg]:
        present[(0, int(v))] = int(rng.integers(0, n_el))
    for _ in range(2 * n_v):
        a, b = sorted(int(x) for x in rng.integers(0, n_v, 2))
        if a != b and (a, b) not in present:
            present[(a, b)] = int(rng.integers(0, n_el))
    edges = np.array([(a, b, l) for (a, b), l in present.items()], np.uint32)
    rows = []
    for _ in range(n_updates):
        if rng.random() < 0.45 and present:
            keys = [k for k in present if k[0] == 0] if rng.random() < 0.6 else list(present)
            keys = keys or list(present)
            a, b = keys[int(rng.integers(0, len(keys)))]
            rows.append((0, a, b, present.pop((a, b))))
        else:
            a = 0 if rng.random() < 0.6 else int(rng.integers(0, n_v))
            b = int(rng.integers(0, n_v))
            a, b = min(a, b), max(a, b)
            if a == b:
                continue
            l = int(rng.integers(0, n_el))
            rows.append((1, a, b, l))
            present.setdefault((a, b), l)
    return vl, edges, updates(rows)


QUERY = ([0, 1, 2, 0], [(0, 1, 0), (1, 2, 0), (0, 2, 0), (2, 3, 0)])


def check(vl, edges, ups, qv, qe, algo="parallel_graphflow", **kw):
    ref = pyoracle.run(qv, qe, vl, edges, ups, want_hash=True)
    with Engine(algo, want_hash=True, **kw) as eng:
        eng.set_query(qv, qe)
        eng.load_graph(vl, edges)
        eng.build_index()
        res = eng.run(ups)
        bytes_ = eng.stats()["device_bytes"], eng.stats()["pool_capacity"]
    for f in ("pos", "neg", "hash"):
        assert np.array_equal(res[f], ref[f]), (f, np.nonzero(res[f] != ref[f])[0][:10])
    with Engine(algo, **kw) as eng:  # counts only: the tail of an order is counted
        eng.set_query(qv, qe)
        eng.load_graph(vl, edges)
        eng.build_index()
        res = eng.run(ups)
    assert np.array_equal(res["pos"], ref["pos"]) and np.array_equal(res["neg"], ref["neg"])
    return bytes_


@pytest.mark.parametrize("kw", [{}, {"mode": "plain"}, {"max_batch": 5}, {"max_batch": 64, "graphs": True}],
                         ids=["batched", "plain", "batches of 5", "graphs"])
@pytest.mark.parametrize("hub_deg", [0, 3, 4, 8, 33, 300])
def test_rows_that_grow_move_and_lose_entries(hub_deg, kw):
    rng = np.random.default_rng(100 + hub_deg)
    vl, edges, ups = hub_case(rng, 400, hub_deg, 2, 500)
    check(vl, edges, ups, *QUERY, **kw)  # GraphFlow: the index plugins count a repeated insertion with another label as 0


@pytest.mark.parametrize("n_el", [1, 3, 15, 16, 17, 62])
def test_edge_label_counts(n_el):
    """Each of the query's labels takes part in an entry; 16 and more needed binary searches before."""
    rng = np.random.default_rng(n_el)
    vl, edges, ups = hub_case(rng, 120, 60, n_el, 300)
    m = min(n_el, 62)
    qe = [(i, i + 1, i % m) for i in range(3)] + [(0, 2, (m - 1))]
    # a path per label keeps every label of the data graph in the folding table
    extra = [(3 + i, 4 + i, i % m) for i in range(min(m, 27))]
    qv = [0, 1, 2, 0] + [int(i % 3) for i in range(len(extra))]
    check(vl, edges, ups, qv[:4], qe)
    if extra:
        check(vl, edges, ups[:60], qv, qe + extra)


def test_joins_without_tables():
    """A device-memory budget below the tables' size: the search joins by binary search, with equal results."""
    rng = np.random.default_rng(7)
    n = 300_000
    vl = rng.integers(0, 3, n).astype(np.uint32)
    e = rng.integers(0, n, (800_000, 2))
    e = e[e[:, 0] != e[:, 1]]
    edges = np.concatenate([e, np.zeros((len(e), 1), np.int64)], 1).astype(np.uint32)
    _, first = np.unique(np.minimum(e[:, 0], e[:, 1]) * n + np.maximum(e[:, 0], e[:, 1]), return_index=True)
    edges = edges[np.sort(first)]
    held, edges = edges[:300], edges[300:]
    ups = updates([(1, int(a), int(b), 0) for a, b, _ in held] + [(0, int(a), int(b), 0) for a, b, _ in held[::2]])
    full, cap = check(vl, edges, ups, *QUERY, max_batch=64)
    table = 8 * cap
    with Engine("parallel_graphflow", want_hash=True, max_batch=64, hbm_budget_bytes=full - table // 8) as eng:
        eng.set_query(*QUERY)
        eng.load_graph(vl, edges)
        eng.build_index()
        res = eng.run(ups)
        assert eng.stats()["device_bytes"] < full - table // 2, "the tables were expected not to fit"
    ref = pyoracle.run(*QUERY, vl, edges, ups)
    for f in ("pos", "neg", "hash"):
        assert np.array_equal(res[f], ref[f])


@pytest.mark.parametrize("n", [31, 32, 33, 65, 97])
@pytest.mark.parametrize("homo", [False, True])
def test_waiting_candidates_around_a_warp(n, homo):
    """Two hubs with n common neighbours: every level has about n candidates that pass the first join."""
    vl = np.zeros(n + 2, np.uint32)
    edges = np.array([(h, 2 + i, 0) for h in (0, 1) for i in range(n)], np.uint32)
    qv, qe = [0, 0, 0, 0], [(0, 1, 0), (0, 2, 0), (1, 2, 0), (0, 3, 0), (1, 3, 0)]
    ups = updates([(1, 0, 1, 0), (1, 2, 3, 0), (0, 0, 1, 0)])
    check(vl, edges, ups, qv, qe, homo=False)
    if homo:
        ref = pyoracle.run(qv, qe, vl, edges, ups, homo=True)
        with Engine("parallel_symbi", homo=True) as eng:
            eng.set_query(qv, qe)
            eng.load_graph(vl, edges)
            eng.build_index()
            res = eng.run(ups)
        assert np.array_equal(res["pos"], ref["pos"]) and np.array_equal(res["neg"], ref["neg"])


@pytest.mark.parametrize("warps", [4, 8, 16])
def test_largest_query_fits_every_block_shape(warps):
    """A 32-vertex query: where 16 walks do not fit in a block's shared memory, fewer are taken."""
    rng = np.random.default_rng(3)
    n = 64
    vl = (np.arange(n) % 32).astype(np.uint32)
    edges = np.array([(i, (i + 1) % n, 0) for i in range(n)] + [(i, (i + 2) % n, 0) for i in range(n)], np.uint32)
    qv = list(range(32))
    qe = [(i, i + 1, 0) for i in range(31)] + [(i, i + 2, 0) for i in range(0, 30, 2)]
    ups = updates([(0, 3, 4, 0), (1, 3, 4, 0)] + [(1, int(a), int(b), 0) for a, b in rng.integers(0, n, (20, 2)) if a != b])
    check(vl, edges, ups, qv, qe, warps_per_block=warps)
