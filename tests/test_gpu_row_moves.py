"""Row insertion and deletion at the edges of their rounds (8 entries a thread: 256 a warp, 2,048 a block) and of
the warp / block split of rows (4,096 entries): random changes at the front, the back and everywhere in a hub's
row.  The row is read back through counts: a query edge at the hub per neighbour label and edge label."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu


def case(deg, k, where, seed):
    """Hub 0 (label 0) with `deg` neighbours of labels 1 and 2; k of them leave and k others arrive."""
    rng = np.random.default_rng(seed)
    n = deg + k
    vl = np.concatenate([[0], rng.integers(1, 3, n), [1, 2]]).astype(np.uint32)
    lab = rng.integers(0, 2, n + 1)
    ids = 1 + np.arange(n)
    if where == "front":
        change = ids[:2 * k]
    elif where == "back":
        change = ids[-2 * k:]
    else:
        change = rng.permutation(ids)[:2 * k]
    change = rng.permutation(change)
    arrive, leave = change[:k], change[k:2 * k]
    start = np.setdiff1d(ids, arrive)
    edges = [(0, int(v), int(lab[v])) for v in start] + [(int(ids[0]), n + 1, 0), (n + 1, n + 2, 0)]
    rows = [(1, 0, int(v), int(lab[v])) for v in arrive] + [(0, 0, int(v), 0) for v in leave if v in start]
    u = np.zeros(len(rows), UPDATE_DTYPE)
    u["type"] = ord("e")
    for i, (a, x, y, l) in enumerate(rows):
        u[i]["is_add"], u[i]["id1"], u[i]["id2"], u[i]["label"] = a, x, y, l
    return vl, np.array(edges, np.uint32), u


# a star of two: every change at the hub counts the hub's other neighbours of the second label pair
QUERY = ([0, 1, 2], [(0, 1, 0), (0, 2, 1)])


@pytest.mark.parametrize("mode", ["batched", "plain"])
@pytest.mark.parametrize("where", ["front", "back", "anywhere"])
@pytest.mark.parametrize("deg,k", [(1, 1), (31, 3), (255, 1), (256, 9), (257, 40), (2047, 5), (2049, 64), (4096, 7),
                                   (4097, 300), (10000, 1000)])
def test_rows_after_changes(deg, k, where, mode):
    if mode == "plain" and k > 64:
        k = 64
    vl, edges, ups = case(deg, k, where, deg + k)
    # the changes twice, undone in between, then a probe of every neighbour: delete them all
    back = ups[::-1].copy()
    back["is_add"] ^= 1
    for r in back:  # a re-inserted edge takes its own label
        r["label"] = next((int(l) for a, b, l in edges if a == r["id1"] and b == r["id2"]), r["label"])
    stream = np.concatenate([ups, back, ups])
    ref = pyoracle.run(*QUERY, vl, edges, stream)
    with Engine("parallel_graphflow", mode=mode, want_hash=True) as eng:
        eng.set_query(*QUERY)
        eng.load_graph(vl, edges)
        eng.build_index()
        for part in (stream[:len(ups)], stream[len(ups):2 * len(ups)], stream[2 * len(ups):]):
            first = eng.submitted
            res = eng.run(part)
            for f in ("pos", "neg", "hash"):
                assert np.array_equal(res[f], ref[f][first:first + len(part)]), f
