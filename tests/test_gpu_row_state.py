"""A batch that cannot be taken out of a row again leaves the row and its table as they were: after "row state"
the joins by table still find what the row holds."""
from __future__ import annotations

import numpy as np
import pytest

from paracosm_b200 import UPDATE_DTYPE, Engine
from paracosm_b200._abi import CsmError

pytestmark = pytest.mark.gpu


def edge(add, a, b):
    return (ord("e"), add, 0, a, b, 0)


def test_row_and_table_agree_after_a_row_that_lacks_an_entry():
    # x = 0 with eight neighbours, e among them; z joined to e; vertices with room for another neighbour
    x, e, z, pairs = 0, 1, 50, 40
    edges = [(x, i, 0) for i in range(1, 9)] + [(e, z, 0)] + [(100 + 2 * i, 101 + 2 * i, 0) for i in range(pairs)]
    first_free, m = 300, 150_000
    vl = np.zeros(first_free + 2 * m, np.uint32)
    fill = np.zeros(m, UPDATE_DTYPE)
    fill["type"], fill["is_add"] = ord("e"), 1
    fill["id1"] = first_free + 2 * np.arange(m)
    fill["id2"] = fill["id1"] + 1
    with Engine("parallel_graphflow", max_batch=4096) as eng:
        eng.set_query([0, 0, 0], [(0, 1, 0), (1, 2, 0), (0, 2, 0)])
        eng.load_graph(vl, np.array(edges, np.uint32))
        eng.build_index()

        def submit(rows):
            return eng.submit(np.array(rows, UPDATE_DTYPE))

        eng.submit(fill)  # a new row at both ends of every edge, until no row can move any more
        with pytest.raises(CsmError, match="row pool"):
            eng.wait()
        for i in range(pairs):  # fill x's row to its capacity
            submit([edge(1, x, 100 + 2 * i)])
            try:
                eng.wait()
            except CsmError:
                break
        else:
            raise AssertionError("x's row was expected to fill up")
        w = 101  # has room, is not joined to x
        submit([edge(1, x, w), edge(0, x, w), edge(0, x, e)])  # (x, w) finds no room in x's row
        with pytest.raises(CsmError, match="row state|row pool"):
            eng.wait()
        s = submit([edge(1, x, z)])  # triangle x, z, e: z's row drives, e is looked up in x's
        with pytest.raises(CsmError, match="row pool"):
            eng.wait()
        assert eng.results(s, 1)["pos"][0] == 6
