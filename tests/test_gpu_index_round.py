"""The incremental index round against an index built afresh on the same graph, where its work lists can go
wrong: a flag whose change marks just under, exactly, just over and well over a list's 32,768 vertices, few
and many items per warp, and changed entries on both sides of the seed's two forms (64 entries)."""
from __future__ import annotations

import numpy as np
import pytest

from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu

ALGOS = ["parallel_turboflux", "parallel_symbi", "parallel_calig", "parallel_newsp"]
# a path 0 - 1 - 2 - 3 with a chord: labels 0, 1, 2, 0
QUERY = ([0, 1, 2, 0], [(0, 1, 0), (1, 2, 0), (2, 3, 0)])


def engine(algo, vl, edges, **kw):
    eng = Engine(algo, **kw)
    eng.set_query(*QUERY)
    eng.load_graph(vl, edges)
    eng.build_index()
    return eng


def ups(rows):
    u = np.zeros(len(rows), UPDATE_DTYPE)
    u["type"] = ord("e")
    for i, (add, a, b) in enumerate(rows):
        u[i]["is_add"], u[i]["id1"], u[i]["id2"] = add, a, b
    return u


def assert_same_index(eng, algo, vl, edges):
    a = eng.index(len(vl))
    with engine(algo, vl, edges) as fresh:
        b = fresh.index(len(vl))
    if a["root"] == b["root"] and a["order"] == b["order"]:  # the root follows the label frequencies
        for k in ("d1", "d2"):
            assert np.array_equal(a[k], b[k]), (k, np.argwhere(a[k] != b[k])[:5])
        return 1
    return 0


@pytest.mark.parametrize("mode", ["batched", "plain"])
@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("n", [1, 31, 33, 2000, 32767, 32768, 32769, 40000])
def test_a_hub_that_marks_n_vertices(n, algo, mode):
    """Vertex 0 (label 1) has n neighbours of label 0; its edge to the only label-2 vertex comes and goes."""
    vl = np.concatenate([[1, 2, 0], np.zeros(n, int)]).astype(np.uint32)
    star = np.stack([np.zeros(n, int), 3 + np.arange(n), np.zeros(n, int)], 1)
    base = np.concatenate([star, [[1, 2, 0]]]).astype(np.uint32)
    full = np.concatenate([base, [[0, 1, 0]]]).astype(np.uint32)
    compared = 0
    with engine(algo, vl, base, mode=mode, max_results=10) as eng:
        for add, now in ((1, full), (0, base), (1, full)):
            eng.run(ups([(add, 0, 1)]))
            compared += assert_same_index(eng, algo, vl, now)
    assert compared


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("k", [1, 31, 32, 33, 500])
def test_batches_of_k_updates(k, algo):
    rng = np.random.default_rng(k)
    n = 3000
    vl = rng.integers(0, 3, n).astype(np.uint32)
    e = rng.integers(0, n, (9000, 2))
    e = e[e[:, 0] != e[:, 1]]
    e = np.unique(np.sort(e, 1), axis=0)
    e = e[rng.permutation(len(e))]
    three = np.concatenate([e, np.zeros((len(e), 1), int)], 1).astype(np.uint32)
    held, edges = three[:k], three[k:]
    steps = [(ups([(1, int(a), int(b)) for a, b, _ in held]), three),
             (ups([(0, int(a), int(b)) for a, b, _ in edges[:k]] + [(0, int(a), int(b)) for a, b, _ in held[:1]]),
              np.concatenate([held[1:], edges[k:]]))]
    # the same updates one by one as well: an index built afresh may choose another root
    with engine(algo, vl, edges, max_results=100) as eng, engine(algo, vl, edges, mode="plain", max_results=100) as one:
        for u, now in steps:
            eng.run(u)
            one.run(u)
            a, b = eng.index(n), one.index(n)
            assert np.array_equal(a["d1"], b["d1"]) and np.array_equal(a["d2"], b["d2"])
            assert_same_index(eng, algo, vl, now)
