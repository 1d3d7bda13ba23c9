"""Values that are not finite are refused on both sides of the size from which the
device checks its copy of the arguments (24,000 values: 4,800 markers of five), at the
first and the last value of every argument; nothing is written, and the context serves
the next call."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [4800, 4801, 20000])
def test_nonfinite_arguments(built_lib, collops_mod, N):
    v, w = gaussian_markers(N, 1.0, 0.6, seed=3)
    bp = uniform_bp(-8.0, 8.0, 16)
    ws = collops_mod.build_workspace(
        collops_mod.SimParameters(bp1=bp, bp2=bp, collision_model="lb"))
    ref = np.zeros_like(v, order="F")
    collops_mod.picard_map(ws, ref, v, v, w, 1.0, 0.02)
    for bad in (np.nan, np.inf, -np.inf):
        for arg in range(3):
            for end in (0, -1):
                a = [v.copy(order="F"), v.copy(order="F"), w.copy()]
                a[arg][(end,) * a[arg].ndim] = bad
                out = np.full_like(v, 7.0, order="F")
                with pytest.raises(collops_mod.CollopsError):
                    collops_mod.picard_map(ws, out, a[0], a[1], a[2], 1.0, 0.02)
                assert np.all(out == 7.0)
    out = np.zeros_like(v, order="F")
    collops_mod.picard_map(ws, out, v, v, w, 1.0, 0.02)
    ws.close()
    assert np.array_equal(out, ref)
