"""The sweeps' solve plan on the host: fronts, gather lists, tasks and panels (no GPU).

fronts_check.cpp builds the plan of several meshes with the engine's own host code and checks its
invariants: every column and update row written by exactly one task, every update row gathered once
on its vertex's row, panels disjoint and aligned, dependencies only between levels.
"""
import os
import subprocess

import numpy as np
import pytest

from fastcorticalwiring_b200 import mesh as M
from fastcorticalwiring_b200.meshgen import folded_icosphere
from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "fastcorticalwiring_b200", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fronts") / "fronts_check")
    src = [os.path.join(CSRC, f) for f in ("prep.cpp", "symbolic.cpp", "fronts.cpp")]
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o", exe,
                           os.path.join(ROOT, "tests", "fronts_check.cpp"), *src, "-lpthread"])
    return exe


def _write(path, V, F):
    with open(path, "wb") as f:
        np.array([V.shape[0], F.shape[0]], np.int64).tofile(f)
        np.ascontiguousarray(V, np.float64).tofile(f)
        np.ascontiguousarray(F, np.int32).tofile(f)


def _two_pieces(m):
    V = np.concatenate([m.V, 0.4 * m.V])
    return V, np.concatenate([m.F, m.F + m.V.shape[0]])


@pytest.mark.parametrize("leaf,width,relax", [(64, 64, 64), (16, 24, 8), (64, 33, 33)])
def test_plan_invariants(checker, tmp_path, leaf, width, relax):
    paths = []
    for level, cap, jitter in ((2, 0.5, 0.0), (4, 0.1, 0.2), (5, 0.37, 0.1), (6, 0.1, 0.2)):
        g = folded_icosphere(level, seed=level, jitter=jitter, cap_fraction=cap)
        pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
        paths.append(str(tmp_path / f"m{level}.bin"))
        _write(paths[-1], pm.V, pm.F)
        if level == 4:
            paths.append(str(tmp_path / "two.bin"))
            _write(paths[-1], *_two_pieces(pm))
    one = str(tmp_path / "one.bin")
    _write(one, np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]]), np.array([[0, 1, 2]]))
    out = subprocess.check_output([checker, str(leaf), str(width), str(relax), *paths, one], text=True)
    lines = [x.split() for x in out.strip().splitlines()]
    assert [x[0] for x in lines] == ["ok"] * (len(paths) + 1)
    if (leaf, width, relax) == (64, 64, 64):  # merging chains takes levels away where there are chains
        assert int(lines[-2][2]) < int(lines[-2][3])
