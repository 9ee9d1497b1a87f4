"""Row tables built afresh when a row moves, for row lengths around what a warp and a block take at once: every
entry is found again, old ones and those inserted with the move, and none that left."""
from __future__ import annotations

import numpy as np
import pytest

from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["batched", "plain"])
@pytest.mark.parametrize("d", [1, 4, 31, 33, 127, 128, 129, 255, 257, 1023, 1024, 1025, 3300, 4100, 5000])
def test_every_entry_is_found_after_a_move(d, mode):
    grow = max(2, d // 4) + 4  # past the capacity that d entries are loaded with
    n = d + grow
    # 0: the row; 1 .. n: its neighbours; z is joined to all of them but one, y to as many others
    z, y = n + 1, n + 2
    vl = np.ones(2 * n + 3, np.uint32)
    vl[0], vl[z], vl[y] = 0, 2, 2
    edges = [(0, v, 0) for v in range(1, d + 1)] + [(z, v, 0) for v in range(1, n)] + [(y, n + 2 + v, 0) for v in range(1, n)]
    rows = [(1, 0, v, 0) for v in range(d + 1, n + 1)]
    rows += [(1, 0, z, 0), (1, 0, y, 0), (0, 0, z, 0), (0, 0, 1, 0), (0, 0, n - 1, 0), (1, 0, z, 0)]
    ups = np.zeros(len(rows), UPDATE_DTYPE)
    ups["type"] = ord("e")
    ups["is_add"], ups["id1"], ups["id2"], ups["label"] = np.array(rows, np.uint32).T
    with Engine("parallel_graphflow", mode=mode) as eng:
        eng.set_query([0, 1, 2], [(0, 1, 0), (1, 2, 0), (0, 2, 0)])
        eng.load_graph(vl, np.array(edges, np.uint32))
        eng.build_index()
        grown = eng.run(ups[:grow])
        assert grown["pos"].sum() == 0
        r = eng.run(ups[grow:])
    assert list(r["pos"][:2]) == [n - 1, 0] and r["neg"][2] == n - 1
    assert r["pos"][5] == n - 3
