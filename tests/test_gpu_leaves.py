"""The leaf level with resident panels on leaves of up to 64 columns (needs a B200): FP64 forward, FP64
backward with and without reach flags, and FP32 backward with all of its row tiles.

The block is wide enough for every one of them by the plan's own rule (leaves_check.cpp runs it on the
host), and ends inside a round of column groups. A few columns of the same engine take the general
kernels: the same factor in the same depth order, so FP64 agrees to 1e-12 of the maximum and mixed to the
1e-5 of test_gpu_fronts.py."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fastcorticalwiring_b200 import engine, mesh as M  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402
from tests.conftest import ROOT  # noqa: E402
from tests.test_fronts_cpu import CSRC, _write  # noqa: E402


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("leaves") / "leaves_check")
    src = [os.path.join(CSRC, f) for f in ("prep.cpp", "symbolic.cpp", "fronts.cpp")]
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o", exe,
                           os.path.join(ROOT, "tests", "leaves_check.cpp"), *src, "-lpthread"])
    return exe


@pytest.mark.parametrize("params,widest", [
    (dict(leaf_size=64, max_width=64, relax=64), 400),  # 512 of 515 leaf tasks hold 33 to 64 columns
    (dict(leaf_size=24, max_width=40, relax=40), 50),   # a mix of leaves
])
def test_resident_leaves_of_64_columns(checker, tmp_path, params, widest):
    g = folded_icosphere(6, seed=4, jitter=0.2)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    block, count, few = 1600, 1590, 16
    path = str(tmp_path / "mesh.bin")
    _write(path, pm.V, pm.F)

    def plan(k):
        args = [params["leaf_size"], params["max_width"], params["relax"]]
        return [int(x) for x in subprocess.check_output([checker, path, str(k), *map(str, args)], text=True).split()]

    tasks, wide, *resident = plan(block)
    assert wide > widest and resident == [1, 1, 1, 1]
    assert plan(64)[2:] == [0, 0, 0, 0]
    src = np.random.default_rng(1).permutation(pm.n_vertices)[:count].astype(np.int32)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=block, pipeline_depth=1, **params)
    try:
        sel = np.linspace(0, count - 1, few).astype(int)
        for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
            ref = eng.compute_distances(src[sel], precision=precision)
            d = eng.compute_distances(src, precision=precision)[sel]
            assert np.max(np.abs(d - ref)) <= tol * np.max(np.abs(ref)), precision
    finally:
        eng.close()
