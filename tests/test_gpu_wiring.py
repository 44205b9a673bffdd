"""WiringAnalysis through fcw_compute_wiring against the same run through records and host assembly
(needs a B200): several blocks with a ragged last one, a lone last source, flagged fields, a boundary
cap, no samples between scales, one scale and 32. The device packs the same records: float32 maps and
samples agree to one float32 rounding (the records' sums differ in their last bits), flags and row
lengths exactly."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fastcorticalwiring_b200 import analysis as A  # noqa: E402
from fastcorticalwiring_b200.meshgen import folded_icosphere  # noqa: E402


class _RecordsOnly:
    def __init__(self, eng):
        self.compute_metrics, self.assemble_samples = eng.compute_metrics, eng.assemble_samples


@pytest.fixture(scope="module")
def an():
    m = folded_icosphere(4, seed=3, jitter=0.2)  # some of its fields are flagged
    a = A.WiringAnalysis(m.vertices, m.faces, m.cortex_mask, engine_kwargs=dict(block_k=128))
    a.quiet = True
    yield a
    a.distance_engine.engine.close()


def _run(a, **kw):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        a.compute_all_wiring_costs(**kw)
    out = {k: v.copy() for k, v in a.get_metric_arrays().items()}
    out.update(flag=a.field_flag.copy(), indptr=a.sample_indptr.copy(), radii=a.sample_radii_flat.copy(),
               areas=a.sample_areas_flat.copy())
    return out, a.n_flagged_fields


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("count,block,kw", [
    (None, 16384, {}),
    (700, 300, dict(boundary_cap_fraction=0.02)),
    (301, 300, dict(scale=[0.01], n_samples_between_scales=0)),  # the last block is one source
    (129, 64, dict(scale=list(np.geomspace(0.001, 0.08, 32)), n_samples_between_scales=8)),
    (0, 64, {}),
])
def test_wiring_matches_records(an, precision, count, block, kw):
    an.precision, an.block_sources = precision, block
    subset = None if count is None else np.random.default_rng(1).permutation(an.sub_to_orig)[:count].tolist()
    got, flagged = _run(an, vertex_subset=subset, **kw)
    whole = an.distance_engine
    an.distance_engine = type("E", (), {"engine": _RecordsOnly(whole.engine), "name": "b200"})()
    try:
        want, flagged_want = _run(an, vertex_subset=subset, **kw)
    finally:
        an.distance_engine = whole
    assert flagged == flagged_want and (count is not None or flagged > 0)
    for k in ("flag", "indptr"):
        assert np.array_equal(got[k], want[k]), k
    for k, v in want.items():
        np.testing.assert_allclose(got[k], v, rtol=2.0 ** -23, atol=0, equal_nan=True, err_msg=k)


def test_subset_forms(an):
    """Lists, tuples and arrays of integers take the vectorised path, anything else the loop; both skip
    what is not a cortical vertex."""
    ids = [int(x) for x in an.sub_to_orig[:50]]
    medial = int(np.flatnonzero(~an.cortex_mask_full)[0])
    base = an._sources([str(x) for x in ids])
    for form in (ids, tuple(ids), np.array(ids), np.array(ids, np.int32), ids + [medial, -5, 10 ** 7, ids[0]],
                 np.array(ids, np.float64), [float(x) for x in ids] + [None, "x"], iter(ids), [10 ** 30] + ids):
        assert np.array_equal(an._sources(form), base)
