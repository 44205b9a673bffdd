"""Heat solves in a row on small trees of fronts (needs a B200): each block has its own reach flags (which
fronts lie on its sources' paths), and the backward sweep of a tree of few levels reads them soon after
they are written. FP64 fields against the oracle's to 1e-10 of the maximum (as test_gpu_fronts.py), and
bit for bit the same every time a block comes round again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from fastcorticalwiring_b200 import engine, mesh as M  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402


def _ico(level, cap):
    g = folded_icosphere(level, seed=3, jitter=0.1, cap_fraction=cap)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    return np.asarray(pm.V, np.float64), np.asarray(pm.F)


@pytest.mark.parametrize("level,cap", [(2, 0.5), (3, 0.3), (4, 0.2)])
@pytest.mark.parametrize("graphs", [True, False])
def test_blocks_of_changing_reach(level, cap, graphs):
    V, F = _ico(level, cap)
    n = V.shape[0]
    eng = engine.HeatEngine(V, F, block_k=64, pipeline_depth=1)
    ho = oracle.HeatOracle(V, F)
    try:
        eng.graphs(graphs)
        order = np.argsort(V[:, 2])  # blocks from opposite ends of the mesh take different paths
        blocks = [order[:3], order[-3:], order[n // 2:n // 2 + 1], order[:: max(1, n // 60)][:60]]
        blocks = [np.ascontiguousarray(b, np.int32) for b in blocks]
        want = [ho.distances(b) for b in blocks]
        first = [eng.compute_distances(b, precision="fp64") for b in blocks]
        for got, ref in zip(first, want):
            assert np.max(np.abs(got - ref)) <= 1e-10 * np.max(np.abs(ref))
        for _ in range(50):
            for b, ref in zip(blocks, first):
                assert np.array_equal(eng.compute_distances(b, precision="fp64"), ref)
    finally:
        eng.close()
