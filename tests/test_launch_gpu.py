"""The chain of a map on both sides of the sizes up to which its markers are sorted in
smaller chunks and its grids start early, and at its smallest: calls in quick succession
on alternating inputs give the results of the first call every time, and the projection
that of the CPU oracle. The quadrature for each number of Gauss points.

Tolerance of the projection: sums of N terms in another order, 1e-11 of the largest value.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 257, 2048, 16384, 16385, 20000, 20001])
def test_repeated_maps(built_lib, collops_mod, oracle_mod, N):
    bp = uniform_bp(-8.0, 8.0, 20)
    om = oracle_mod.OracleMesh(bp, bp, 6, use_logsq=True)
    ws = collops_mod.build_workspace(
        collops_mod.SimParameters(bp1=bp, bp2=bp, collision_model="lb", use_logsq=True))
    cases = []
    for seed in (1, 2):
        v, w = gaussian_markers(N, 1.2, 0.6, seed=seed)
        v_in = np.asfortranarray(v + 0.01)
        f = np.zeros(ws.n_dofs)
        collops_mod.l2_project_gpu(ws, f, v, w)
        S0 = om.entropy(om.l2_project(v, w))
        out = np.zeros_like(v, order="F")
        collops_mod.picard_map(ws, out, v_in, v, w, S0, 0.02)
        fr = om.l2_project(v, w)
        assert np.max(np.abs(f - fr)) <= 1e-11 * np.max(np.abs(fr))
        cases.append((v, w, v_in, S0, f, out))
    for _ in range(20):
        for v, w, v_in, S0, f, out in cases:
            f2, out2 = np.zeros_like(f), np.zeros_like(out, order="F")
            collops_mod.picard_map(ws, out2, v_in, v, w, S0, 0.02)
            collops_mod.l2_project_gpu(ws, f2, v, w)
            assert np.array_equal(f2, f) and np.array_equal(out2, out, equal_nan=True)
    ws.close()


@pytest.mark.parametrize("n_quad", [1, 2, 5, 7, 8])
@pytest.mark.parametrize("n_el", [1, 3, 17])
def test_quadrature(built_lib, collops_mod, oracle_mod, n_quad, n_el):
    """Every number of Gauss points that divides a block of 256 differently, on meshes of
    one element, of less than a block's elements and of a remainder. Both sides add the
    same terms of a positive field, in another order: 1e-12."""
    bp = uniform_bp(-6.0, 6.0, n_el)
    om = oracle_mod.OracleMesh(bp, bp, n_quad)
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp, N_QUAD=n_quad))
    rng = np.random.default_rng(n_el)
    f = rng.uniform(0.1, 1.0, ws.n_dofs)
    r = np.zeros(ws.n_dofs)
    collops_mod.compute_r_gpu(ws, r, f)
    S = collops_mod.compute_entropy_gpu(ws, f)
    ws.close()
    ref = om.compute_r(f)
    assert np.max(np.abs(r - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert abs(S - om.entropy(f)) <= 1e-12 * np.sum(np.abs(ref * f))
