"""An error that a stage reports in any step of a run -- stacked or single,
followed by others or not, replayed from a graph or redone in reference order --
is the run's error.  The errors are written by a stand-in for the stages'
launch functions (status_shim.cpp); nothing fails on the GPU."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

TESTS = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(TESTS)

CHILD = r"""
import ctypes, sys
sys.path[:0] = [{root!r}, {tests!r}]
import torch
shim = ctypes.CDLL({shim!r}, ctypes.RTLD_GLOBAL)
from cageo_gb300 import _build, api
api.lib()
shim.shim_library(_build.LIB.encode())
import numpy as np
from cases import make_case
dem, streams = make_case(96, 80, seed=5)

def failing(stage, call, kw, batch, first, count, graphs=True):
    p = api.Pipeline(dem, streams, error_stddev=1.5, seed=4, use_graphs=graphs, **kw)
    if batch:
        p.set_batch(batch)
    if first:
        p.run(0, first)
    shim.shim_fail(stage, call)
    try:
        p.run(first, count)
        text = "no error"
    except api.CageoError as e:
        text = str(e)
    assert shim.shim_seen() >= call, "the call to fail was not made"
    shim.shim_fail(0, 0)
    # The next run starts afresh (a captured step would hold the stand-in's write).
    p.set_tuning(64, 20)
    p.reset_counts()
    p.run(0, 5)
    got = p.counts()
    p.close()
    q = api.Pipeline(dem, streams, error_stddev=1.5, seed=4, **kw)
    q.set_batch(1)
    q.run(0, 5)
    assert np.array_equal(got, q.counts())
    q.close()
    return text

names = {{1: "pit filling", 2: "flow routing", 3: "flow tracing"}}
for stage in (1, 2, 3):
    for label, args in {cases!r}:
        text = failing(stage, *args)
        assert names[stage] in text, (label, stage, text)
print("statuses ok")
"""

CASES = {
    # (call to fail, pipeline options, batch, realizations before, count, graphs)
    "a batched step, a remainder after it": (1, {}, 2, 0, 3),
    "a batched step, another after it": (1, {}, 2, 0, 4, False),
    "the last batched step, a remainder after it": (2, {}, 2, 0, 5, False),
    "a stack sized by the grid": (1, {}, None, 0, 4),
    "a single realization, others after it": (1, {}, 1, 0, 3, False),
    "the last single realization": (3, {}, 1, 0, 3, False),
    # The captured call carries the error into every replay.
    "a replayed single realization": (2, {}, 1, 0, 3),
    "reference order, another realization after it": (1, {"nodata_dem": 0.0}, 1, 0, 2),
}


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    from cageo_gb300 import _build
    out = str(tmp_path_factory.mktemp("shim") / "status_shim.so")
    lib64 = os.path.join(_build.CUDA_HOME, "lib64")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", _build.INCLUDE, "-I",
                    _build.CSRC, "-I", os.path.join(_build.CUDA_HOME, "include"), "-o", out,
                    os.path.join(TESTS, "status_shim.cpp"), "-L", lib64, "-lcudart", "-ldl"],
                   check=True)
    return out


@pytest.mark.parametrize("case", list(CASES))
def test_error_of_any_step_is_the_runs(cuda, shim, case):
    code = CHILD.format(root=ROOT, tests=TESTS, shim=shim, cases=[(case, CASES[case])])
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "statuses ok" in r.stdout, r.stdout + r.stderr
