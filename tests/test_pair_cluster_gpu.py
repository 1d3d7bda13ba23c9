"""Markers within the reach of the FP64 form of the fixed-point pair sum: clusters that
span two tiles, so that the targets of a warp add to one source's sum in successive steps,
against the CPU oracle.

Tolerance: close pairs are taken in FP64, and dominate the sums here: |d| from 1e-8 to
1e-6 with |G_a - G_g| of order 1. Both sides add N such terms of both signs, an error of
about sqrt(N) 2^-53 of their size, 3e-15 at N = 700; the bound is ten times that. The
sums are a few times smaller than their terms' sizes together, another factor of ten.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu

TOL = 3e-13


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("N,size", [(500, 40), (700, 150), (13000, 300)])
@pytest.mark.parametrize("weights", ["equal", "random"])
def test_cluster(built_lib, collops_mod, oracle_mod, N, size, weights):
    v, w = gaussian_markers(N, 1.2, 0.7, seed=N)
    rng = np.random.default_rng(N + size)
    v[:size] = (0.3, -0.2) + 4e-7 * rng.standard_normal((size, 2))
    v[size // 2] = v[0]                                   # coincident
    if weights == "random":
        w = rng.uniform(0.2, 1.8, N) / N
    G = np.asfortranarray(-v + rng.standard_normal(v.shape))
    bp = uniform_bp(-6.0, 6.0, 8)
    om = oracle_mod.OracleMesh(bp, bp, 6)
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp))
    runs = []
    for _ in range(3):
        F, A = np.zeros((N, 2), order="F"), np.zeros((N, 3), order="F")
        collops_mod.compute_collision_metric_gpu(ws, F, A, v, w, G)
        dv = np.zeros((N, 2), order="F")
        collops_mod.compute_collision_gpu(ws, dv, v, w, G)
        runs.append((F, A, dv))
    ws.close()
    Fr, Ar = om.collision_metric(v, w, G)
    for F, A, dv in runs:
        assert np.array_equal(F, runs[0][0]) and np.array_equal(A, runs[0][1])
        assert np.array_equal(dv, runs[0][2])
    F, A, dv = runs[0]
    assert rel(F, Fr) < TOL and rel(A, Ar) < TOL and rel(dv, Fr) < TOL
