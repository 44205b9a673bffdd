"""Calls of growing and shrinking sizes on one engine (needs a B200): the host-buffer entry points keep
device staging between calls, and each call's launch chain is captured and replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fastcorticalwiring_b200 import engine, mesh as M  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fields_after_a_larger_call(precision):
    """A few fields, more of them (the staging is allocated anew), and the same few again: the replayed
    chain must write the fields where the copy to the host reads them."""
    g = folded_icosphere(4, seed=2, jitter=0.1)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    rng = np.random.default_rng(0)
    few, more, other = (rng.permutation(pm.n_vertices)[:k].astype(np.int32) for k in (37, 100, 37))
    eng = engine.HeatEngine(pm.V, pm.F, block_k=128, pipeline_depth=2)
    try:
        first = eng.compute_distances(few, precision=precision)
        eng.compute_distances(more, precision=precision)
        assert np.array_equal(eng.compute_distances(few, precision=precision), first)
        a = eng.compute_distances(other, precision=precision)  # and with other sources
        eng.graphs(False)
        assert np.array_equal(eng.compute_distances(other, precision=precision), a)
    finally:
        eng.close()


@pytest.mark.parametrize("count", [2, 63, 65, 1000, 2049, 4096])
def test_sources_sorted_in_place(count):
    """The host-buffer call sorts its sources where they were copied to, up to the largest block: every
    field is the one its source has alone."""
    g = folded_icosphere(2, seed=2, jitter=0.1)
    pm = M.prepare(g.vertices, g.faces, g.cortex_mask)
    src = np.random.default_rng(count).integers(0, pm.n_vertices, count).astype(np.int32)
    eng = engine.HeatEngine(pm.V, pm.F, block_k=4096, pipeline_depth=1)
    try:
        alone = eng.compute_distances(np.arange(pm.n_vertices, dtype=np.int32), precision="fp64")
        d = eng.compute_distances(src, precision="fp64")
        # a column's sums do not depend on the block it is in, but the kernels' split of a block may
        assert np.max(np.abs(d - alone[src])) <= 1e-12 * np.max(np.abs(alone))
        assert np.array_equal(d[np.arange(count), src], np.zeros(count))
    finally:
        eng.close()
