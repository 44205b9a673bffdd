"""The fans are the same arrays for any number of threads (no GPU): fans_check.cpp forms them in one
range of vertices, in the number the engine would take, and in 2 to 64, also more than the mesh has
vertices. And the fans of vertices with sharp corners: which they are, and their coefficients."""
import os
import subprocess

import numpy as np
import pytest

from fastcorticalwiring_b200 import mesh as M
from fastcorticalwiring_b200.meshgen import folded_icosphere
from tests.conftest import ROOT
from tests.test_fronts_cpu import CSRC, _write
from tests.test_patches_cpu import book, hub


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fans") / "fans_check")
    src = [os.path.join(CSRC, f) for f in ("prep.cpp", "patches.cpp")]
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o", exe,
                           os.path.join(ROOT, "tests", "fans_check.cpp"), *src, "-lpthread"])
    return exe


def _icosphere(level):
    g = folded_icosphere(level, seed=level, jitter=0.2)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    return pm.V, pm.F


@pytest.mark.parametrize("mesh,sharp", [
    (lambda: _icosphere(6), 0),  # 36,866 vertices: eight ranges by the engine's own rule
    (lambda: _icosphere(4), 0), (lambda: book(5), 0),
    (lambda: hub(60), 0), (lambda: hub(64), 1),    # the hub, from 5.7 degrees on
    (lambda: hub(500), 1001),                      # there the rings' triangles are needles too
    (lambda: (np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]]), np.array([[0, 1, 2]], np.int32)), 0),
], ids=["L6", "L4", "book", "hub60", "hub64", "hub500", "triangle"])
def test_fans_do_not_depend_on_the_threads(checker, tmp_path, mesh, sharp):
    V, F = mesh()
    path = str(tmp_path / "mesh.bin")
    _write(path, V, F)
    out = subprocess.check_output([checker, path], text=True).split()
    assert out[0] == "ok" and int(out[1]) > 3 * len(F)
    assert int(out[2]) == sharp
