"""Levels and tails whose driver segments do not fit in one 32-bit range together.  That takes rows of 2^27
entries; here the search is compiled with a range of 96 elements instead, so that ordinary walks reach it
everywhere.  Counts, hashes and work bytes must be those of the oracle and of the ordinary build."""
from __future__ import annotations

import subprocess

import numpy as np
import pytest

from conftest import golden_cases, load_golden
from oracle import pyoracle
from paracosm_b200 import Engine, _abi, build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def narrow(tmp_path_factory):
    """The engine with a range of 96 elements."""
    d = tmp_path_factory.mktemp("narrow")

    def obj(src):
        done = build.OBJ / (src[:-3] + ".o")
        if src != "csm_search.cu" and done.exists():
            return done
        out = d / (src[:-3] + ".o")
        subprocess.run([build.NVCC] + build.NVFLAGS + ["-DCSM_RANGE_MAX=96u", "-c", str(build.CSRC / src), "-o", str(out)],
                       check=True, capture_output=True)
        return out

    objs = [str(obj(s)) for s in build.CU_SOURCES]
    lib = d / "libcsmgpu_narrow.so"
    subprocess.run([build.NVCC] + build.ARCH + ["-shared", "-ccbin", build.CXX, "-o", str(lib)] + objs + ["-lcudart"],
                   check=True, capture_output=True)
    return _abi.load_library(lib)


def run(g, algo, ups, **kw):
    with Engine(algo, **kw) as eng:
        eng.set_query(g["qv"], g["qe"])
        eng.load_graph(g["vl"], g["e"])
        eng.build_index()
        init = eng.initial_match()
        return init, eng.run(ups)


@pytest.mark.parametrize("kw", [dict(want_hash=True), dict(), dict(mode="plain"), dict(homo=True), dict(max_results=7)],
                         ids=lambda k: " ".join(k) or "counts")
@pytest.mark.parametrize("algo", ["parallel_graphflow", "parallel_symbi"])
@pytest.mark.parametrize("case", golden_cases())
def test_narrow_ranges(narrow, monkeypatch, case, algo, kw):
    g = load_golden(case)
    ups = g["stream"][:150]
    init, want = run(g, algo, ups, **kw)
    monkeypatch.setattr(_abi, "_lib", narrow)
    init2, res = run(g, algo, ups, **kw)
    assert init2 == init
    fields = ["pos", "neg", "status"] + (["hash"] if kw.get("want_hash") else [])
    if not kw.get("max_results"):
        fields.append("work_bytes")  # a walk that stops at a cap may have expanded more or less
    for f in fields:
        assert np.array_equal(res[f], want[f]), (f, np.nonzero(res[f] != want[f])[0][:10])
    if algo == "parallel_graphflow":
        ref = pyoracle.run(g["qv"], g["qe"], g["vl"], g["e"], ups, homo=kw.get("homo", False),
                           max_results=kw.get("max_results", 0))
        for f in ("pos", "neg") + (("hash",) if kw.get("want_hash") else ()):
            assert np.array_equal(res[f], ref[f]), f
