"""Host-side rules of the wiring analysis' fast paths, without a device."""
import types

import numpy as np
import pytest

from fastcorticalwiring_b200.analysis import WiringAnalysis


class _Ids(list):
    """A list that iterates as something else than it holds."""

    def __iter__(self):
        return iter([3, 4])


def _analysis(n=12):
    a = object.__new__(WiringAnalysis)
    a.mesh = types.SimpleNamespace(bfs=np.arange(n)[::-1], n_vertices=n)
    a.n_vertices_full = n
    a.cortex_mask_full = np.ones(n, bool)
    a.orig_to_sub = np.arange(n)
    return a


@pytest.mark.parametrize("form", [
    np.ma.MaskedArray([1, 2, 3, 7], mask=[0, 1, 0, 1]),  # masked vertices are not asked for
    np.ma.MaskedArray([1, 2, 3, 7]),
    _Ids([5, 6]),
])
def test_subset_subclasses_are_read_element_by_element(form):
    want = set()
    for x in form:
        try:
            want.add(int(x))
        except Exception:
            continue
    assert set(_analysis()._sources(form).tolist()) == want
