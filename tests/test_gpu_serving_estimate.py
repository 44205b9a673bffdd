"""The serving loop's memory estimate against engines as they are built (needs a B200), over sizes, block
widths and the options that add arrays."""
import pytest

pytestmark = pytest.mark.gpu

from fastcorticalwiring_b200 import engine, mesh as M, serving as S  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402


@pytest.mark.parametrize("level,cap", [(2, 0.5), (4, 0.1), (5, 0.37), (6, 0.1)])
def test_estimate_is_an_upper_one(level, cap):
    g = folded_icosphere(level, seed=level, jitter=0.2, cap_fraction=cap)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    n = pm.n_vertices
    for opts in ({}, dict(tc_sweeps=1, refine=1), dict(robust=1), dict(leaf_size=256),
                 dict(leaf_size=16, max_width=20, relax=8)):
        for block_k, depth in ((64, 1), (320, 2)):
            eng = engine.HeatEngine(pm.V, pm.F, block_k=block_k, pipeline_depth=depth, **opts)
            held = eng.info()["device_bytes"]
            eng.close()
            kept = {k: v for k, v in opts.items() if k in ("tc_sweeps", "refine", "leaf_size")}
            est = S.estimate_device_bytes(n, 2 * n, block_k, depth, 0, S._stride(12, 3), **kept)
            assert held <= est, (opts, block_k)
