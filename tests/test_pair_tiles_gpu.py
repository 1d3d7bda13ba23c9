"""The packed pair kernels (two source tiles per step) against the CPU oracle where
a row of tile pairs ends: odd and even numbers of tiles, a single last tile, more
than one chunk of a row, and weights that differ from tile to tile.

Tolerances: FP32 terms carry about 2^-22 and their sums over a 256-marker tile
about sqrt(256) 2^-24 of a partial sum, 1e-6 of the result; the bound is ten times
that. Double-single terms carry 1e-13; the bound of 1e-9 on vdot is the one the
double-single map has elsewhere. A missing or doubled tile pair shows above 1e-4.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu


def _weights(kind, N, rng):
    w = np.full(N, 1.0 / N)
    if kind == "random":
        w *= rng.uniform(0.1, 2.0, N)
    elif kind == "half":      # tiles of one weight beside tiles of another
        w[N // 2:] *= 1.5
    return w


@pytest.mark.parametrize("weights", ["equal", "random"])
@pytest.mark.parametrize("N", [1000, 1281, 1537, 4353, 8705])
def test_fp32_sum(built_lib, collops_mod, oracle_mod, N, weights):
    v, _ = gaussian_markers(N, 1.2, 0.6, seed=N)
    rng = np.random.default_rng(N)
    w = _weights(weights, N, rng)
    v[5] = v[N // 2]          # coincident
    G = np.asfortranarray(-v / [1.44, 0.36] + 0.3 * np.sin(2 * v[:, ::-1]))
    bp = uniform_bp(-8.0, 8.0, 16)
    om = oracle_mod.OracleMesh(bp, bp, 6)
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp, gpu_fp32=True))
    dv = np.zeros((N, 2), order="F")
    collops_mod.compute_collision_gpu32(ws, dv, v, w, G)
    ws.close()
    ref = om.collision(v, w, G)
    assert np.max(np.abs(dv - ref)) / np.max(np.abs(ref)) < 1e-5


@pytest.mark.parametrize("weights", ["equal", "random", "half"])
@pytest.mark.parametrize("N", [513, 640, 1000, 2176, 4353])
def test_double_single_map(built_lib, collops_mod, oracle_mod, N, weights):
    v, _ = gaussian_markers(N, 1.2, 0.6, seed=N)
    rng = np.random.default_rng(N)
    w = _weights(weights, N, rng)
    bp = uniform_bp(-8.0, 8.0, 12)
    om = oracle_mod.OracleMesh(bp, bp, 6, use_logsq=True)
    o = oracle_mod.Opts()
    dt = 0.05
    S0 = om.entropy(om.l2_project(v, w))
    v_in = np.asfortranarray(v + 0.01 * rng.standard_normal(v.shape))
    ws = collops_mod.build_workspace(
        collops_mod.SimParameters(bp1=bp, bp2=bp, use_logsq=True))
    out = np.zeros_like(v, order="F")
    collops_mod.picard_map(ws, out, v_in, v, w, S0, dt, precision="mixed_ds")
    ws.close()
    ref = om.picard_map(o, v_in, v, w, S0, dt)
    assert np.max(np.abs(out - ref)) / np.max(np.abs(ref - v)) < 1e-9
