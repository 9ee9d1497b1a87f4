"""A warp re-evaluates a flag over up to 15 segments at once: the first 32 / segments entries of each together, the
rest one segment after another.  The only supporting entry lies last in its segment, on both sides of that line."""
from __future__ import annotations

import numpy as np
import pytest

from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["parallel_turboflux", "parallel_symbi", "parallel_calig"])
@pytest.mark.parametrize("n", [1, 2, 3, 6, 7, 10, 11, 16, 17, 32, 33, 70])
@pytest.mark.parametrize("arms", [1, 2, 3, 5, 15])
def test_last_entry_supports(arms, n, algo):
    """Query: a centre with `arms` arms of two edges.  Data: a hub with n inner vertices per arm, of which only the
    last has an outer vertex; that edge of the first and of the last arm goes and comes back."""
    qlab = [0] + [1 + a for a in range(arms)] + [arms + 1] * arms
    qedges = [(0, 1 + a, 0) for a in range(arms)] + [(1 + a, 1 + arms + a, 0) for a in range(arms)]
    inner = 1 + np.arange(arms * n).reshape(arms, n)
    outer = 1 + arms * n + np.arange(arms)
    vl = np.concatenate([[0], np.repeat(1 + np.arange(arms), n), np.full(arms, arms + 1)]).astype(np.uint32)
    spokes = [(0, int(v), 0) for v in inner.ravel()]
    ends = [(int(inner[a, -1]), int(outer[a]), 0) for a in range(arms)]
    base = np.array(spokes + ends, np.uint32)
    rows = []
    for a in sorted({0, arms - 1}):
        rows += [(0, *ends[a][:2]), (1, *ends[a][:2])]

    def engine(edges):
        eng = Engine(algo, max_results=100)
        eng.set_query(qlab, qedges)
        eng.load_graph(vl, edges)
        eng.build_index()
        return eng

    with engine(base) as eng:
        for add, x, y in rows:
            u = np.zeros(1, UPDATE_DTYPE)
            u["type"], u["is_add"], u["id1"], u["id2"] = ord("e"), add, x, y
            res = eng.run(u)
            assert (int(res["pos"][0]), int(res["neg"][0])) == (add, 1 - add)
            now = base if add else np.array(spokes + [e for e in ends if e[:2] != (x, y)], np.uint32)
            got = eng.index(len(vl))
            with engine(now) as fresh:
                want = fresh.index(len(vl))
            if (got["root"], got["order"]) == (want["root"], want["order"]):  # it follows the label frequencies
                assert np.array_equal(got["d1"], want["d1"]) and np.array_equal(got["d2"], want["d2"])


@pytest.mark.parametrize("algo", ["parallel_turboflux", "parallel_symbi", "parallel_calig"])
@pytest.mark.parametrize("mode", ["batched", "plain"])
@pytest.mark.parametrize("widths", [[1] * 6, [1, 32, 1, 33, 1, 40], [1, 1, 40, 1, 40, 1], [33, 1, 31, 1, 64, 1],
                                    [104, 1, 33, 33, 1, 2]])
def test_runs_of_short_and_long_steps(widths, mode, algo):
    """Levels of vertices, each wholly joined to the next, under a path query: the edges between the first two levels
    go and come back, so the round's work lists are as long as the levels are wide, short and long in turn."""
    levels, n = [], 0
    for w in widths:
        levels.append(list(range(n, n + w)))
        n += w
    vl = np.repeat(np.arange(len(widths)), widths).astype(np.uint32)
    pairs = [[(x, y, 0) for x in a for y in b] for a, b in zip(levels, levels[1:])]
    base = np.array(sum(pairs, []), np.uint32)
    rest = np.array(sum(pairs[1:], []), np.uint32)
    embeddings = int(np.prod(widths, dtype=np.int64))

    def engine(edges):
        eng = Engine(algo, max_results=10**9, mode=mode)
        eng.set_query(list(range(len(widths))), [(i, i + 1, 0) for i in range(len(widths) - 1)])
        eng.load_graph(vl, edges)
        eng.build_index()
        return eng

    compared = 0
    with engine(base) as eng:
        for add in (0, 1):
            u = np.zeros(len(pairs[0]), UPDATE_DTYPE)
            u["type"], u["is_add"] = ord("e"), add
            u["id1"], u["id2"] = [p[0] for p in pairs[0]], [p[1] for p in pairs[0]]
            res = eng.run(u)
            assert int(res["pos" if add else "neg"].sum()) == embeddings
            got = eng.index(n)
            with engine(base if add else rest) as fresh:
                want = fresh.index(n)
            if (got["root"], got["order"]) == (want["root"], want["order"]):
                compared += 1
                assert np.array_equal(got["d1"], want["d1"]) and np.array_equal(got["d2"], want["d2"])
    assert compared
