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
from fastcorticalwiring_b200 import _lib, engine, mesh as M  # noqa: E402
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


@pytest.mark.parametrize("block_k,count", [(64, 1), (320, 320), (320, 500), (128, 129)])
def test_source_order_changes_nothing(block_k, count):
    """Blocks are solved in elimination order: each source's results, repeated sources' too, are the
    same wherever it stands in the list (fields bit for bit; records to the near lists' order of
    summation, FP64)."""
    g = folded_icosphere(4, seed=5, jitter=0.1, cap_fraction=0.2)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    rng = np.random.default_rng(3)
    src = rng.integers(0, pm.n_vertices, count).astype(np.int32)
    src[count // 2] = src[0]
    perm = rng.permutation(count)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=block_k, pipeline_depth=2)
    try:
        targets = pm.targets(M.RUNNER_SCALES)
        for precision in ("fp64", "mixed"):
            a = eng.compute_distances(src, precision=precision)
            b = eng.compute_distances(src[perm], precision=precision)
            assert np.array_equal(a[perm], b)
            assert np.array_equal(a[count // 2], a[0])
            if count == 1 and precision == "fp64":
                continue  # one FP64 source takes a chain of its own
            ra = eng.compute_metrics(src, targets, 2, precision=precision)
            rb = eng.compute_metrics(src[perm], targets, 2, precision=precision)
            np.testing.assert_allclose(ra[perm], rb, rtol=1e-12, equal_nan=True)
    finally:
        eng.close()


@pytest.mark.parametrize("count,params", [
    (1000, dict(leaf_size=16, max_width=20, relax=8)),  # thousands of leaves: both sweeps, reach flags too
    (600, {}),                                          # 64-column leaves, a ragged number of column groups
])
def test_resident_leaves_match_general_sweeps(count, params):
    """Many leaves and columns keep the leaves' panels in shared memory; a few columns of the same
    engine take the general kernels. Same factor, same depth order: FP64 to 1e-12 of the maximum, mixed
    to the 1e-5 above."""
    g = folded_icosphere(6, seed=4, jitter=0.2)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    src = np.random.default_rng(count).permutation(pm.n_vertices)[:count].astype(np.int32)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=1024, pipeline_depth=1, **params)
    try:
        sel = np.arange(7, count, 97)
        for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
            ref = eng.compute_distances(src[sel], precision=precision)
            d = eng.compute_distances(src, precision=precision)[sel]
            assert np.max(np.abs(d - ref)) <= tol * np.max(np.abs(ref)), precision
    finally:
        eng.close()


def test_invalid_source_is_refused():
    g = folded_icosphere(3, seed=1)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=64, pipeline_depth=1)
    try:
        for bad in (-1, pm.n_vertices):
            with pytest.raises(_lib.FCWError) as e:
                eng.compute_distances(np.array([0, bad, 1], np.int32))
            assert e.value.code == _lib.FCW_E_INVALID
        assert eng.compute_distances(np.array([1], np.int32))[0, 1] == 0.0
    finally:
        eng.close()
