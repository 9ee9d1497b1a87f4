"""Batches whose lists are sorted by one block each, against the same updates one by one: list lengths (2 B + 64) and
batch sizes on both sides of 512, 2,048, 4,096 and 9,216, edges that come and go many times (the order of equal keys), and
vertex ids of so many bits that a key leaves no room for its place."""
from __future__ import annotations

import numpy as np
import pytest

from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu

QUERY = ([0, 1, 2, 0], [(0, 1, 0), (1, 2, 1), (2, 3, 0)])


def case(n, b, seed):
    rng = np.random.default_rng(seed)
    m = 3000
    ids = np.sort(rng.choice(n, m, replace=False))
    ids[-1] = n - 1
    vl = np.zeros(n, np.uint32)
    vl[ids] = rng.integers(0, 3, m)
    e = np.unique(np.sort(rng.integers(0, m, (12000, 2)), 1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    edges = np.stack([ids[e[:, 0]], ids[e[:, 1]], rng.integers(0, 2, len(e))], 1).astype(np.uint32)
    u = np.zeros(b, UPDATE_DTYPE)
    u["type"] = ord("e")
    u["is_add"] = rng.integers(0, 2, b)
    hot = rng.integers(0, 20, b)
    pick = np.where(rng.random(b) < 0.3, hot, rng.integers(0, len(edges), b))
    flip = rng.random(b) < 0.5
    x, y = edges[pick, 0].copy(), edges[pick, 1].copy()
    fresh = rng.random(b) < 0.2
    x[fresh], y[fresh] = ids[rng.integers(0, m, fresh.sum())], ids[rng.integers(0, m, fresh.sum())]
    u["id1"], u["id2"] = np.where(flip, x, y), np.where(flip, y, x)
    u["label"] = np.where(fresh, rng.integers(0, 2, b), edges[pick, 2])
    return vl, edges, u


@pytest.mark.parametrize("n,b", [(5000, b) for b in (1, 31, 224, 225, 512, 513, 992, 993, 1024, 1025, 2016, 2017, 2048, 2049, 4096, 4097, 4576,
                                                     4577, 9216, 9217)] + [(1 << 22, 700), (1 << 24, 700)])
def test_batches_against_single_updates(n, b):
    vl, edges, ups = case(n, b, b)
    got = {}
    for mode in ("batched", "plain"):
        with Engine("parallel_graphflow", mode=mode, want_hash=True, max_batch=16384) as eng:
            eng.set_query(*QUERY)
            eng.load_graph(vl, edges)
            eng.build_index()
            got[mode] = np.concatenate([eng.run(ups), eng.run(ups[::-1].copy())])
    assert (got["batched"]["pos"].sum() > 0) or b < 100
    for f in ("pos", "neg", "hash", "status"):
        assert np.array_equal(got["batched"][f], got["plain"][f]), f
