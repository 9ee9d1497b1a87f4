"""Contexts with queries of different sizes, a host thread each: the search's shared-memory limit is a property of
the kernel that all contexts of a device share, and no context may lower it for another."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from paracosm_b200 import UPDATE_DTYPE, Engine

pytestmark = pytest.mark.gpu


def path_engine(n):
    """A path query of n labels over four copies of itself, and one edge that comes and goes."""
    vl = np.tile(np.arange(n), 4).astype(np.uint32)
    edges = np.array([(c * n + i, c * n + i + 1, 0) for c in range(4) for i in range(n - 1)], np.uint32)
    eng = Engine("parallel_graphflow", max_batch=64)
    eng.set_query(list(range(n)), [(i, i + 1, 0) for i in range(n - 1)])
    eng.load_graph(vl, edges)
    eng.build_index()
    ups = np.zeros(2, UPDATE_DTYPE)
    ups["type"], ups["id1"], ups["id2"], ups["is_add"] = ord("e"), n // 2, n // 2 + 1, (0, 1)
    return eng, ups


def test_queries_of_different_sizes_side_by_side():
    errors = []

    def work(n):
        try:
            eng, ups = path_engine(n)
            with eng:
                for _ in range(1500):
                    r = eng.run(ups)
                    assert r["neg"][0] == 1 and r["pos"][1] == 1
        except BaseException as e:  # noqa: BLE001
            errors.append((n, repr(e)))

    threads = [threading.Thread(target=work, args=(n,)) for n in (5, 32, 8, 28)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
