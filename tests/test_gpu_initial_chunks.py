"""InitialMatching's seeds per launch: contexts of every batch size, seed counts below and above one launch's,
and a budget without room for the seeds' own buffers, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle
from paracosm_b200 import Engine

pytestmark = pytest.mark.gpu


def ring(n: int):
    """A ring with chords: 2 n edges between two alternating labels (even n) and one edge label."""
    vl = (np.arange(n) % 2).astype(np.uint32)
    i = np.arange(n, dtype=np.uint32)
    return vl, np.concatenate([np.stack([i, (i + 1) % n, 0 * i], 1), np.stack([i, (i + 3) % n, 0 * i], 1)]).astype(np.uint32)


def count(vl, edges, **kw):
    with Engine("parallel_symbi", **kw) as eng:
        eng.set_query([0, 1, 0], [(0, 1, 0), (1, 2, 0)])
        eng.load_graph(vl, edges)
        eng.build_index()
        before = eng.stats()["device_bytes"]
        c = eng.initial_match()
        assert eng.stats()["device_bytes"] == before
        assert eng.initial_match() == c
        return c, before


@pytest.mark.parametrize("n", [8, 1000, 32768, 32770, 70000])  # n entries 0 -> 1 each side: 2 n seeds, one launch takes 65,536
def test_seed_counts_around_a_launch(n):
    vl, edges = ring(n)
    want = pyoracle.initial_count([0, 1, 0], [(0, 1, 0), (1, 2, 0)], vl, edges)
    for kw in ({}, {"mode": "plain"}, {"max_batch": 333}):
        assert count(vl, edges, **kw)[0] == want, kw


def test_no_room_for_the_seeds_buffers():
    vl, edges = ring(2000)
    want, held = count(vl, edges, max_batch=100)
    tight, _ = count(vl, edges, max_batch=100, hbm_budget_bytes=held + (1 << 20))
    assert tight == want == pyoracle.initial_count([0, 1, 0], [(0, 1, 0), (1, 2, 0)], vl, edges)
