"""The mixed divergence of vertices with more neighbours than a patch holds (needs a B200): those are
gathered from memory, a warp each (k_div_mixed_big), on both sides of the patch's limit.

A patch holds 108 rows, a vertex's own among them. The mesh is a hub of needle triangles, which take FP32
itself past the 1e-5 of test_gpu_divergence.py: evaluated per face and corner the form is 1.4e-5 off at
300 neighbours. Bound here: 2e-5 of the maximum, against the oracle's fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from fastcorticalwiring_b200 import engine  # noqa: E402
from tests.test_patches_cpu import hub  # noqa: E402


@pytest.mark.parametrize("neighbours", [106, 107, 108, 300])
@pytest.mark.parametrize("count", [1, 130])
def test_mixed_fields_around_a_hub(neighbours, count):
    V, F = hub(neighbours)
    V = np.ascontiguousarray(V, np.float64)
    n = V.shape[0]
    src = np.random.default_rng(5).integers(0, n, count).astype(np.int32)
    src[0] = int(np.argmax(np.bincount(np.asarray(F).ravel(), minlength=n)))  # the hub itself
    ref = oracle.HeatOracle(V, F).distances(src)
    eng = engine.HeatEngine(V, F, block_k=192, pipeline_depth=1)
    try:
        d = eng.compute_distances(src, precision="mixed")
        assert np.max(np.abs(d - ref)) <= 2e-5 * np.max(np.abs(ref))
    finally:
        eng.close()
