"""The element quadrature where its blocks take different numbers of elements (one to all
that fit), with a remainder in the last block, for one job and for the two of a map,
against the CPU oracle. Both sides add the same terms of a positive field, in another
order: 1e-12; a map's velocities 1e-11, as for the other maps."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_quad", [2, 6])
@pytest.mark.parametrize("n_el", [13, 24, 37, 48, 49])
def test_elements_per_block(built_lib, collops_mod, oracle_mod, n_el, n_quad):
    bp = uniform_bp(-6.0, 6.0, n_el)
    om = oracle_mod.OracleMesh(bp, bp, n_quad)
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp, N_QUAD=n_quad))
    f = np.random.default_rng(n_el).uniform(0.1, 1.0, ws.n_dofs)
    r = np.zeros(ws.n_dofs)
    collops_mod.compute_r_gpu(ws, r, f)
    S = collops_mod.compute_entropy_gpu(ws, f)
    ref = om.compute_r(f)
    assert np.max(np.abs(r - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert abs(S - om.entropy(f)) <= 1e-12 * np.sum(np.abs(ref * f))
    v, w = gaussian_markers(20000, 1.0, 0.8, seed=1)
    v_in = np.asfortranarray(0.99 * v)
    out = np.zeros_like(v, order="F")
    collops_mod.picard_map(ws, out, v_in, v, w, 1.0, 1e-4)
    ws.close()
    vr = om.picard_map(oracle_mod.Opts(), v_in, v, w, 1.0, 1e-4)
    assert np.max(np.abs(out - vr)) <= 1e-11 * np.max(np.abs(vr))
