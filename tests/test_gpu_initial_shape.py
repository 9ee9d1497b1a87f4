"""InitialMatching counts the tail of every order, with walks of up to one level more than the batches of a
context that asks for hashes or match sets take: its launch shape is fitted to its own search."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import Engine

pytestmark = pytest.mark.gpu


def layers(n: int, width: int, rng):
    """A path query over n labels (its orders end in the path's two ends, a tail of two) and a layered graph."""
    qv, qe = list(range(n)), [(i, i + 1, 0) for i in range(n - 1)]
    vl = np.repeat(np.arange(n), width).astype(np.uint32)
    edges = [(i * width + a, (i + 1) * width + b, 0) for i in range(n - 1) for a in range(width) for b in range(width)
             if a == b or rng.random() < 0.4]
    return qv, qe, vl, np.array(edges, np.uint32)


@pytest.mark.parametrize("kw", [{}, {"want_hash": True}, {"enum_capacity": 64}], ids=["counts", "hashes", "match sets"])
@pytest.mark.parametrize("n", [21, 22, 23])  # around 16 walks in a block's shared memory
def test_shape_is_that_of_the_counting_search(n, kw):
    qv, qe, vl, edges = layers(n, 3, np.random.default_rng(n))
    want = pyoracle.initial_count(qv, qe, vl, edges)
    assert want > 0
    with Engine("parallel_symbi", warps_per_block=16, max_batch=64, **kw) as eng:
        eng.set_query(qv, qe)
        eng.load_graph(vl, edges)
        eng.build_index()
        before = eng.stats()["device_bytes"]
        assert eng.initial_match() == want
        assert eng.stats()["device_bytes"] == before
