"""Several engines of different sizes on one device (needs a B200): what the first one set up has to hold
after the others were made ready."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fastcorticalwiring_b200 import engine, mesh as M  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402


def _engine(level):
    g = folded_icosphere(level, seed=3, jitter=0.1)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    return engine.HeatEngine(pm.V, pm.F, block_k=64, pipeline_depth=1)


@pytest.mark.parametrize("graphs", [True, False])
def test_single_source_calls_after_a_smaller_engine(graphs):
    """The single-source sweeps' shared memory depends on the engine's largest front; a smaller engine's
    first call must not take it away from a larger one, captured or launched directly, nor from its stage
    timeline."""
    large, small = _engine(6), _engine(3)
    try:
        sources = [0, large.n_vertices // 2]
        want = [large.compute_distance(s) for s in sources]
        small.compute_distance(1)
        large.graphs(graphs)
        for s, d in zip(sources, want):
            assert np.array_equal(large.compute_distance(s), d)
        large.profile(True)
        assert np.array_equal(large.compute_distance(sources[0]), want[0])
        assert large.stage_times()[0]["poisson_bwd"] > 0
    finally:
        large.close()
        small.close()
