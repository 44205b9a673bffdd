"""Host-side rules of the wiring analysis' fast paths, without a device."""
import types

import numpy as np
import pytest

from fastcorticalwiring_b200 import engine
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


def _bad_arrays():
    k, n = 5, 8
    maps, flags = np.zeros((k, n), np.float32), np.zeros(n, np.uint8)
    locked_maps, locked_flags = maps.copy(), flags.copy()
    locked_maps.flags.writeable = locked_flags.flags.writeable = False
    yield "every second flag", maps, np.zeros(2 * n, np.uint8)[::2]
    yield "flags backwards", maps, flags[::-1]
    yield "flags of another shape", maps, flags.reshape(2, 4)
    yield "read-only flags", maps, locked_flags
    yield "read-only maps", locked_maps, flags
    yield "maps by columns", np.asfortranarray(maps), flags
    yield "maps of more dimensions", np.zeros((k, n, 2), np.float32), flags
    yield "FP64 maps", maps.astype(np.float64), flags
    yield "too few flags", maps, flags[:-1]


@pytest.mark.parametrize("name,maps,flags", list(_bad_arrays()), ids=lambda x: x if isinstance(x, str) else "")
def test_arrays_that_cannot_be_written_in_place_are_refused(name, maps, flags):
    """The library writes both arrays through their first element's address."""
    eng = object.__new__(engine.HeatEngine)
    eng._h = None
    with pytest.raises(ValueError):
        eng.compute_wiring([0, 1], [1.0], [2, 3], maps, flags)
