"""The patch-wise divergence at its edges (needs a B200): meshes smaller than a patch, non-manifold
edges (fans that end), a vertex with more neighbours than a patch holds, edges tens of diffusion
lengths long (faces whose gradient leaves the fans' common scale), and column counts of one and
several slices.

FP64: bit-identical to the oracle's face loop, given the same u. Mixed: the fields against the
oracle's, 1e-5 of the maximum as in test_gpu_fronts.py (not on the hub, whose needle triangles take
FP32 itself past that: the form evaluated per face and corner is 1.4e-5 off there, the fans 1.2e-5).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from fastcorticalwiring_b200 import _lib, engine, mesh as M  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402
from tests.test_patches_cpu import book, hub  # noqa: E402


def _ico(level, cap, jitter):
    g = folded_icosphere(level, seed=7, jitter=jitter, cap_fraction=cap)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    return pm.V, pm.F


MESHES = {
    "edges of 54 diffusion lengths": lambda: _ico(1, 0.2, 0.0),
    "edges of 30 diffusion lengths": lambda: _ico(2, 0.1, 0.1),
    "jittered": lambda: _ico(4, 0.3, 0.2),
    "non-manifold": lambda: book(4, 40),
    "hub": lambda: hub(300),
}


@pytest.mark.parametrize("name", sorted(MESHES))
def test_divergence(name):
    import torch

    V, F = MESHES[name]()
    V = np.ascontiguousarray(V, np.float64)
    n = V.shape[0]
    ho = oracle.HeatOracle(V, F)
    eng = engine.HeatEngine(V, F, block_k=192, pipeline_depth=1)
    try:
        for k in (1, 64, 150):
            src = np.random.default_rng(k).integers(0, n, k)
            u = ho.heat(src)
            if k > 2:
                u[:, 1] = 0.0            # every face's gradient vanishes
                u[n // 2:, 2] *= 1e-200  # subnormal and zero differences
            ud = torch.tensor(u, dtype=torch.float64, device="cuda").contiguous()
            div = torch.empty_like(ud)
            _lib.check(_lib.load().fcw_divergence_device(eng.handle, ctypes.c_void_p(ud.data_ptr()), k,
                                                         ctypes.c_void_p(div.data_ptr()), None))
            eng.synchronize(0)
            assert np.array_equal(div.cpu().numpy(), ho.divergence(u)), k
        src = np.random.default_rng(5).integers(0, n, 130).astype(np.int32)
        ref = ho.distances(src)
        top = np.max(np.abs(ref))
        for precision, tol in (("fp64", 1e-10), ("mixed", 1e-5)):
            if (precision, name) == ("mixed", "hub"):
                continue
            d = eng.compute_distances(src, precision=precision)
            assert np.max(np.abs(d - ref)) <= tol * top, precision
    finally:
        eng.close()
