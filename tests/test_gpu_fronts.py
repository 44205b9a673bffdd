"""The batched sweeps over fronts at the sizes where their tiles end (needs a B200).

Fields of a few sources against the oracle's, for block widths that take the 64- and 128-column
tiles, a ragged number of sources, meshes whose fronts stay under 64 columns and meshes with wide
fronts (assembled right-hand sides, 32- and 64-row tasks), and narrow factorisations (many small
supernodes, so fronts are long chains). Tolerances: the FP64 fields agree with another
factorisation to 1e-10 of the maximum (as test_gpu_parity.py), the mixed ones to 1e-5: FP32 rounding
(6e-8) times the grounded operator's amplification, measured under 1e-6 on these meshes' order.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from fastcorticalwiring_b200 import engine, mesh as M  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402


@pytest.mark.parametrize("level,cap,jitter,params", [
    (3, 0.6, 0.2, {}),                                           # a couple of fronts
    (4, 0.33, 0.1, {}),                                          # no wide front
    (5, 0.1, 0.2, {}),                                           # wide fronts at the root
    (5, 0.21, 0.0, dict(leaf_size=16, max_width=20, relax=8)),   # long chains
])
@pytest.mark.parametrize("count", [1, 64, 100, 129, 320])
def test_fields_match_oracle(level, cap, jitter, params, count):
    g = folded_icosphere(level, seed=2, jitter=jitter, cap_fraction=cap)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    rng = np.random.default_rng(count)
    src = rng.permutation(pm.n_vertices)[:count].astype(np.int32)
    if src.size < count:  # a mesh of fewer vertices: sources may repeat
        src = np.concatenate([src, rng.integers(0, pm.n_vertices, count - src.size).astype(np.int32)])
    eng = engine.HeatEngine(pm.V, pm.F, block_k=384, pipeline_depth=1, **params)
    try:
        sel = np.unique(np.concatenate([np.arange(min(count, 6)), [count // 2, count - 1]]))
        ref = oracle.HeatOracle(pm.V, pm.F).distances(src[sel])
        top = np.max(np.abs(ref))
        for precision, tol in (("fp64", 1e-10), ("mixed", 1e-5)):
            d = eng.compute_distances(src, precision=precision)[sel]
            assert np.max(np.abs(d - ref)) <= tol * top, precision
    finally:
        eng.close()
