"""The divergence's fans and patches on the host (no GPU): patches_check.cpp builds them with the
engine's own code on regular, ragged, non-manifold and hub meshes and checks that every face enters
each of its vertices' fans once with the right coefficients, and that a patch's rows name the mesh's
vertices."""
import os
import subprocess

import numpy as np
import pytest

from fastcorticalwiring_b200 import mesh as M
from fastcorticalwiring_b200.meshgen import folded_icosphere
from tests.conftest import ROOT
from tests.test_fronts_cpu import CSRC, _write


def book(pages=3, n=6):
    """Sheets joined along one edge line: its edges have `pages` faces."""
    V, F = [], []
    spine = list(range(n))
    V += [(float(i), 0.0, 0.0) for i in range(n)]
    for p in range(pages):
        a = 2.0 * np.pi * p / pages
        first = len(V)
        V += [(float(i) + 0.3, np.cos(a), np.sin(a)) for i in range(n)]
        for i in range(n - 1):
            F += [(spine[i], spine[i + 1], first + i), (spine[i + 1], first + i + 1, first + i)]
    return np.array(V), np.array(F, np.int32)


def hub(n):
    """A disc whose centre has n neighbours, with a second ring of faces."""
    t = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(t), np.sin(t), 0.1 * np.sin(3 * t)], 1)
    V = np.concatenate([[[0.0, 0, 0.2]], ring, 1.2 * ring])
    F = []
    for i in range(n):
        j = (i + 1) % n
        F += [(0, 1 + i, 1 + j), (1 + i, 1 + n + i, 1 + j), (1 + j, 1 + n + i, 1 + n + j)]
    return V, np.array(F, np.int32)


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("patches") / "patches_check")
    src = [os.path.join(CSRC, f) for f in ("prep.cpp", "patches.cpp")]
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o", exe,
                           os.path.join(ROOT, "tests", "patches_check.cpp"), *src, "-lpthread"])
    return exe


def test_fans_and_patches(checker, tmp_path):
    meshes = []
    for level, cap, jitter in ((2, 0.5, 0.0), (4, 0.1, 0.2), (5, 0.37, 0.1)):
        g = folded_icosphere(level, seed=level, jitter=jitter, cap_fraction=cap)
        pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
        meshes.append((pm.V, pm.F))
    meshes += [book(3), book(5), hub(20), hub(107), hub(108), hub(400)]
    meshes.append((np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]]), np.array([[0, 1, 2]], np.int32)))
    paths = []
    for i, (V, F) in enumerate(meshes):
        paths.append(str(tmp_path / f"{i}.bin"))
        _write(paths[-1], V, F)
    out = [x.split() for x in subprocess.check_output([checker, *paths], text=True).strip().splitlines()]
    assert [x[0] for x in out] == ["ok"] * len(meshes)
    assert [int(x[2]) for x in out[5:9]] == [0, 0, 1, 1]  # the centre of 108 and 400 neighbours is gathered
