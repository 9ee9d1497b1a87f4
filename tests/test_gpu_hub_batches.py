"""Batches whose updates meet at one vertex: the presence of a segment's touched entries, around a warp's width and
with edges that come and go several times in the batch.  Counts, hashes and work bytes are the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu

QUERY = ([0, 1, 1, 2], [(0, 1, 0), (0, 2, 1), (1, 2, 0), (0, 3, 0)])


@pytest.mark.parametrize("batch", [65536, 50], ids=["one batch", "batches of 50"])
@pytest.mark.parametrize("kw", [dict(want_hash=True), dict()], ids=["hashes", "counts"])
@pytest.mark.parametrize("spread", [1, 3, 31, 32, 33, 97, 400])
def test_hub_batches(spread, kw, batch):
    """`spread` neighbours of vertex 0 come and go, over two edge labels."""
    rng = np.random.default_rng(spread)
    n = 1 + 2 * spread + 40
    vl = np.ones(n, np.uint32)
    vl[0], vl[-20:] = 0, 2
    present = {}
    for v in range(1, 2 * spread + 1, 2):
        present[v] = int(rng.integers(0, 2))
    edges = [(0, v, l) for v, l in present.items()] + [(0, n - 1 - i, 0) for i in range(5)]
    edges += [(int(a), int(b), 0) for a, b in {tuple(sorted(rng.integers(1, n - 20, 2))) for _ in range(6 * n)} if a != b]
    ups = np.zeros(900, UPDATE_DTYPE)
    ups["type"] = ord("e")
    for i, u in enumerate(ups):
        v = int(rng.integers(1, 2 * spread + 1))
        if i % 9 == 8:
            v = n - 1 - int(rng.integers(0, 20))
            if v in present or v > n - 6:
                v = 1
        u["id2"] = v
        if v in present:
            u["label"] = present.pop(v)
        else:
            u["is_add"] = 1
            u["label"] = present[v] = 0 if v >= n - 20 else int(rng.integers(0, 2))
    edges = np.array(edges, np.uint32)
    ref = pyoracle.run(*QUERY, vl, edges, ups, want_hash=kw.get("want_hash", False))
    assert ref["pos"].sum() > 0 or spread < 3
    with Engine("parallel_graphflow", max_batch=batch, **kw) as eng:
        eng.set_query(*QUERY)
        eng.load_graph(vl, edges)
        eng.build_index()
        res = eng.run(ups)
    for f, g in (("pos", "pos"), ("neg", "neg"), ("work_bytes", "bytes")) + ((("hash", "hash"),) if kw else ()):
        assert np.array_equal(res[f], ref[g]), (f, np.nonzero(res[f] != ref[g])[0][:10])
