"""The per-source kernel and the shift statistics where their launches change shape (needs a B200): one
source per SM, two, more; vertex tiles of 128 to 1024; targets of most of the surface, whose near faces
are too many for the staged list; against the oracle on a few sources (FP64 1e-9, mixed 1e-4 relative,
MSD 1e-5, as test_gpu_parity.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from fastcorticalwiring_b200 import engine, mesh as M  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402


@pytest.fixture(scope="module")
def mesh():
    g = folded_icosphere(5, seed=4, jitter=0.1, cap_fraction=0.15)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=1024, pipeline_depth=1)
    yield pm, eng, oracle.HeatOracle(pm.V, pm.F)
    eng.close()


@pytest.mark.parametrize("scales", [M.RUNNER_SCALES, (0.01, 0.4, 0.97)])
@pytest.mark.parametrize("count", [1, 64, 148, 192, 297, 900])
def test_metrics_match_oracle(mesh, count, scales):
    pm, eng, ho = mesh
    src = np.random.default_rng(count).permutation(pm.n_vertices)[:count].astype(np.int32)
    targets = pm.targets(scales)
    sel = np.unique([0, count // 2, count - 1])
    phi = ho.distances(src[sel])
    for precision, tol in (("fp64", 1e-9), ("mixed", 1e-4)):
        r = engine.split_records(eng.compute_metrics(src, targets, 2, precision=precision), len(scales), 2)
        for i, j in enumerate(sel):
            ref = oracle.source_metrics(phi[i], int(src[j]), pm, targets, n_between=2)
            assert bool(r["bad"][j]) == ref["bad"]
            assert r["neg"][j] == ref["neg"] and r["viol"][j] == ref["viol"]
            if ref["bad"]:
                continue
            for k in ("radii", "perim", "extra_r", "extra_a"):
                np.testing.assert_allclose(r[k][j], ref[k], rtol=tol, err_msg=f"{precision} {k}")
            for k in ("msd_u", "msd_w"):
                np.testing.assert_allclose(r[k][j], ref[k], rtol=max(tol / 10, 1e-9))
            np.testing.assert_allclose(r["dist_b"][j], ref["dist_b"], rtol=tol)


@pytest.fixture(scope="module")
def large():
    g = folded_icosphere(6, seed=4, jitter=0.1)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=512, pipeline_depth=1)
    yield pm, eng
    eng.close()


@pytest.mark.parametrize("n_targets", [1, 4, 7, 8, 12, 15, 16, 32])
def test_teams_match_one_warp_per_target(large, n_targets):
    """A few sources on a large mesh evaluate each target with four, two or (from 16 targets) one warp;
    a large block of the same sources takes a warp per target. Same bracket and Newton steps; sums differ
    in order only (1e-9 relative, as above)."""
    pm, eng = large
    src = np.random.default_rng(n_targets).permutation(pm.n_vertices)[:400].astype(np.int32)
    targets = pm.targets(np.geomspace(0.002, 0.1, n_targets))
    for precision in ("fp64", "mixed"):
        many = engine.split_records(eng.compute_metrics(src, targets, 3, precision=precision), n_targets, 3)
        for few in (1, 9):
            r = engine.split_records(eng.compute_metrics(src[:few], targets, 3, precision=precision), n_targets, 3)
            for k in ("radii", "perim", "extra_r", "extra_a"):
                np.testing.assert_allclose(r[k], many[k][:few], rtol=1e-9, err_msg=f"{precision} {k}")
            assert np.array_equal(r["n_eval"], many["n_eval"][:few])


def test_far_from_the_origin():
    """The chord test's FP32 form must not decide where the coordinates' magnitude swamps it: health
    counts on a mesh moved 1e6 mm away are the oracle's."""
    g = folded_icosphere(4, seed=3, jitter=0.2)  # some fields violate the chord bound
    V = g.vertices + np.array([1e6, -2e6, 3e5])
    pm = M.prepare(V, g.faces, g.cortex_mask)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=256, pipeline_depth=1)
    try:
        src = np.arange(256, dtype=np.int32)
        fields = eng.compute_distances(src, precision="fp64")
        r = engine.split_records(eng.compute_metrics(src, pm.targets([0.01, 0.02]), 0, precision="fp64"), 2, 0)
        for j in range(src.size):
            neg, viol, bad = oracle.field_health(fields[j], pm.V, int(src[j]), pm.health_h)
            assert (r["neg"][j], r["viol"][j], bool(r["bad"][j])) == (neg, viol, bad)
    finally:
        eng.close()
