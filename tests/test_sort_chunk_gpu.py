"""The marker sort on both sides of the size from which its chunks are larger, and at the
smaller sizes of a context that has grown beyond it: the projection and the Picard map of
the same markers give the same bits in either order of the sizes, and the projection is that
of the CPU oracle.

Tolerance: sums of N terms in another order, 1e-11 of the largest value.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu

SIZES = [40959, 40960, 40961, 49152, 255, 70000, 40960]


def test_chunk_sizes(built_lib, collops_mod, oracle_mod):
    bp = uniform_bp(-8.0, 8.0, 20)
    om = oracle_mod.OracleMesh(bp, bp, 6)

    def run(ws, N):
        v, w = gaussian_markers(N, 1.2, 0.6, seed=N)
        f, out = np.zeros(ws.n_dofs), np.zeros((N, 2), order="F")
        collops_mod.l2_project_gpu(ws, f, v, w)
        collops_mod.picard_map(ws, out, np.asfortranarray(v + 0.01), v, w, 1.0, 0.02)
        fr = om.l2_project(v, w)
        assert np.max(np.abs(f - fr)) <= 1e-11 * np.max(np.abs(fr))
        return f, out

    def fresh():
        return collops_mod.build_workspace(
            collops_mod.SimParameters(bp1=bp, bp2=bp, collision_model="lb"))

    ws = fresh()
    for N in SIZES:
        one = fresh()
        for a, b in zip(run(ws, N), run(one, N)):
            assert np.array_equal(a, b)
        one.close()
    ws.close()
