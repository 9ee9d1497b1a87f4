"""A submit that fails on the host when part of it is queued: the device error which that part raised is reported
by the next wait, not hidden by the state of the submit before."""
from __future__ import annotations

import numpy as np
import pytest

from paracosm_b200 import UPDATE_DTYPE, Engine
from paracosm_b200._abi import CsmError

pytestmark = pytest.mark.gpu

HUB = 20_000  # neighbours of vertex 0


def test_device_error_of_a_failed_submit():
    n, batch = 400_000, 4096
    vl = np.zeros(n, np.uint32)
    edges = np.zeros((HUB, 3), np.uint32)
    edges[:, 1] = np.arange(1, HUB + 1)
    # disjoint edges: every insertion takes a new row at both ends, until the pool cannot hold them
    m = 150_000
    ups = np.zeros(m + 1, UPDATE_DTYPE)
    ups["type"] = ord("e")
    ups["id1"][:m] = HUB + 1 + 2 * np.arange(m)
    ups["id2"][:m] = HUB + 2 + 2 * np.arange(m)
    idle = ups.copy()  # deletions of missing edges: buffers of this size, nothing else
    ups["is_add"] = 1
    ups[m] = (ord("v"), 0, 0, 0, 0, 0)  # deleting the hub needs memory that the budget does not have
    query = ([0, 0, 0], [(0, 1, 0), (1, 2, 0), (0, 2, 0)])

    def engine(budget):
        eng = Engine("parallel_graphflow", max_batch=batch, hbm_budget_bytes=budget)
        eng.set_query(*query)
        eng.load_graph(vl, edges)
        eng.build_index()
        eng.run(idle)
        return eng

    with engine(0) as eng:
        held = eng.stats()["device_bytes"]
    with engine(held + 100_000) as eng:
        with pytest.raises(CsmError, match="budget"):
            eng.submit(ups)
        with pytest.raises(CsmError, match="row pool"):
            eng.wait()
        eng.wait()  # reported once
