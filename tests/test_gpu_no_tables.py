"""Searches of graphs that have no row tables -- a device-memory budget without room for them, or vertex ids and
edge labels too wide for a table entry -- in the forms a search takes.  Exact against the oracle, and against the
same context with tables."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu


def core_case(rng, n, m, core, n_el):
    """A sparse random graph with a dense core, and a stream of insertions and deletions in the core in which
    edges come and go more than once within a batch."""
    vl = rng.integers(0, 2, n).astype(np.uint32)
    e = rng.integers(core, n, (m, 2))
    a, b = np.triu_indices(core, 1)
    keep = rng.random(len(a)) < 0.8
    e = np.concatenate([np.stack([a, b], 1)[keep], e[e[:, 0] != e[:, 1]]])
    key = np.minimum(e[:, 0], e[:, 1]) * n + np.maximum(e[:, 0], e[:, 1])
    e = e[np.sort(np.unique(key, return_index=True)[1])]
    edges = np.concatenate([e, rng.integers(0, n_el, (len(e), 1))], 1).astype(np.uint32)
    present = {(int(x), int(y)): int(l) for x, y, l in edges if x < core and y < core}
    ups = np.zeros(400, UPDATE_DTYPE)
    ups["type"] = ord("e")
    hot = [tuple(sorted(map(int, rng.choice(core, 2, replace=False)))) for _ in range(60)]
    for u in ups:
        x, y = hot[int(rng.integers(0, len(hot)))]
        l = present.pop((x, y), None)
        if l is None:
            l = present[(x, y)] = int(rng.integers(0, n_el))
            u["is_add"] = 1
        u["id1"], u["id2"], u["label"] = x, y, l
    return vl, edges, ups


QUERY = ([0, 1, 0, 1, 0, 0], [(0, 1, 0), (0, 2, 0), (1, 2, 1), (0, 3, 0), (1, 3, 0), (2, 3, 1), (2, 4, 0), (3, 5, 0), (0, 5, 1)])

FORMS = [dict(), dict(want_hash=True), dict(homo=True), dict(max_results=50), dict(tail_enumerate=True),
         dict(mode="plain", want_hash=True), dict(graphs=True)]


def run(algo, vl, edges, ups, query, **kw):
    with Engine(algo, **{"max_batch": 64, **kw}) as eng:
        eng.set_query(*query)
        eng.load_graph(vl, edges)
        eng.build_index()
        init = eng.initial_match()
        res = eng.run(ups)
        return init, res, eng.stats()


def expect(vl, edges, ups, query, res, kw):
    ref = pyoracle.run(*query, vl, edges, ups, max_results=kw.get("max_results", 0), homo=kw.get("homo", False))
    assert ref["pos"].sum() > 0 and ref["neg"].sum() > 0
    for f in ("pos", "neg") + (("hash",) if kw.get("want_hash") else ()):
        assert np.array_equal(res[f], ref[f]), (f, np.nonzero(res[f] != ref[f])[0][:10])


@pytest.mark.parametrize("kw", FORMS, ids=lambda k: " ".join(k) or "counts")
@pytest.mark.parametrize("algo", ["parallel_graphflow", "parallel_symbi"])
def test_no_room_for_tables(algo, kw):
    vl, edges, ups = core_case(np.random.default_rng(5), 300_000, 800_000, 40, 2)
    init, res, st = run(algo, vl, edges, ups, QUERY, **kw)
    table = 8 * st["pool_capacity"]
    init2, res2, st2 = run(algo, vl, edges, ups, QUERY, hbm_budget_bytes=st["device_bytes"] - table // 2, **kw)
    assert st2["device_bytes"] < st["device_bytes"] - table // 2, "the tables were expected not to fit"
    expect(vl, edges, ups, QUERY, res2, kw)
    assert init == init2
    for f in ("pos", "neg", "status"):
        assert np.array_equal(res[f], res2[f])


@pytest.mark.parametrize("headroom", [(1 << 26) - 2000, 1 << 26], ids=["tables", "no tables"])
def test_ids_and_labels_around_an_entry(headroom):
    """17 folded edge labels take five bits: below 2^26 vertices the entries fit, above they do not."""
    vl, edges, ups = core_case(np.random.default_rng(6), 1000, 3000, 30, 16)
    skew = lambda l: np.where(l < 12, l % 4, l)  # most edges carry one of the query's labels
    edges[:, 2], ups["label"] = skew(edges[:, 2]), skew(ups["label"])
    query = ([0, 0, 0, 0], [(0, 1, 0), (1, 2, 1), (0, 2, 2), (2, 3, 3)])
    vl[:] = 0
    with Engine("parallel_graphflow", want_hash=True, max_batch=64, vertex_headroom=headroom) as eng:
        eng.set_query(*query)
        eng.reserve_labels([], np.arange(16))
        eng.load_graph(vl, edges)
        eng.build_index()
        res = eng.run(ups)
    expect(vl, edges, ups, query, res, dict(want_hash=True))
