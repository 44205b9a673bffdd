"""The mixed divergence at sharp corners (needs a B200): needle triangles around a hub, whose long edges
are nearly parallel at it.

Two refinement steps take the FP32 factor's error out of the fields, which leaves the divergence's. Bound:
2e-6 of the maximum against the oracle; a restatement in numpy with FP32 coefficients and differences is at
most 4e-7 off at 107 to 500 needles, 1.8e-5 without the sharp corners' form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from fastcorticalwiring_b200 import engine  # noqa: E402
from tests.test_patches_cpu import hub  # noqa: E402


@pytest.mark.parametrize("needles", [64, 107, 108, 300, 500])
@pytest.mark.parametrize("count", [1, 130])
def test_mixed_fields_around_needles(needles, count):
    V, F = hub(needles)
    V = np.ascontiguousarray(V, np.float64)
    src = np.random.default_rng(5).integers(0, V.shape[0], count).astype(np.int32)
    ref = oracle.HeatOracle(V, F).distances(src)
    eng = engine.HeatEngine(V, F, block_k=192, pipeline_depth=1, refine=2)
    try:
        d = eng.compute_distances(src, precision="mixed")
        assert np.max(np.abs(d - ref)) <= 2e-6 * np.max(np.abs(ref))
    finally:
        eng.close()
