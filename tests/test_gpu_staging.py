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
