"""The fixed-point pair sum and metric (co_pair_fixed.cu) against the CPU oracle:
tile edges and remainders of both tile widths (32 and 128 markers; the wider from
about 12,600 markers on), equal and unequal weights (zero among them), markers
outside the domain, coincident and close pairs, and the exactness of its scalings.

Tolerance: the oracle adds N FP64 terms one after another, an error of about
sqrt(N) 2^-53 of the sum for terms of both signs (1.3e-14 at N = 13,000); the
bound is ten times that.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu

TOL = 1.3e-13


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def _case(N, weights, seed=5, lo=-6.0, hi=6.0):
    v, w = gaussian_markers(N, 1.6, 0.7, seed=seed)   # some 20 in 10^5 outside [-6, 6]
    rng = np.random.default_rng(seed)
    v[3] = (7.0, 0.1)
    v[N // 2] = (0.2, -6.0)
    v[10] = v[11]                                    # coincident
    v[20] = v[21] + (1e-13, 0.0)                      # inside the guard
    v[30] = v[31] + (3e-10, -1e-10)                   # FP64 form
    v[40] = v[41] + (2e-6, 2e-6)
    v[50] = v[51] + (1e-5, 0.0)
    if weights == "random":
        w = rng.uniform(0.1, 2.0, N) / N
        w[::17] = 0.0
    G = np.asfortranarray(-v / [2.56, 0.49] + 0.3 * np.sin(2 * v[:, ::-1])
                          + 0.1 * rng.standard_normal(v.shape))
    v += 0.5 * (lo + hi)
    return v, w, G, uniform_bp(lo, hi, 16)


@pytest.mark.parametrize("weights", ["equal", "random"])
@pytest.mark.parametrize("N", [385, 416, 417, 1000, 12543, 12673])
def test_sum_and_metric(built_lib, collops_mod, oracle_mod, N, weights):
    v, w, G, bp = _case(N, weights)
    om = oracle_mod.OracleMesh(bp, bp, 6)
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp))
    dv, F, A = (np.zeros((N, k), order="F") for k in (2, 2, 3))
    collops_mod.compute_collision_gpu(ws, dv, v, w, G)
    collops_mod.compute_collision_metric_gpu(ws, F, A, v, w, G)
    ws.close()
    Fr, Ar = om.collision_metric(v, w, G)
    assert rel(dv, Fr) < TOL and rel(F, Fr) < TOL and rel(A, Ar) < TOL
    scale = np.sum(w[:, None] * np.abs(dv))
    assert abs(np.sum(w * dv[:, 0])) < 1e-14 * scale
    assert abs(np.sum(w * dv[:, 1])) < 1e-14 * scale


@pytest.mark.parametrize("lo,hi", [(1000.0, 1012.0), (-30.0, -18.0), (-6.0, 6.0)])
def test_scalings_are_exact(built_lib, collops_mod, oracle_mod, lo, hi):
    """Powers of two in G and w pass through unrounded; a domain far from 0 is as
    accurate as one around it."""
    N = 700
    v, w, G, bp = _case(N, "random", lo=lo, hi=hi)
    om = oracle_mod.OracleMesh(bp, bp, 6)

    def run(w, G):
        ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp))
        out = np.zeros((N, 2), order="F")
        collops_mod.compute_collision_gpu(ws, out, v, w, G)
        ws.close()
        return out

    ref = run(w, G)
    assert rel(ref, om.collision(v, w, G)) < TOL
    assert np.array_equal(run(w * 2.0 ** -300, G) * 2.0 ** 300, ref)
    assert np.array_equal(run(w, G * 2.0 ** 400) * 2.0 ** -400, ref)


@pytest.mark.parametrize("max_iter,tol,done", [(200, 1e-9, True), (70, 0.0, False)])
def test_solve_restarts(built_lib, collops_mod, oracle_mod, max_iter, tol, done):
    """step_anderson! starts on the fixed-point sums and, where they do not converge
    soon, again from the same guess in FP64: both ends against the oracle. The solve
    stops at 1e-9 of |v|, or after 70 maps well below that; bound 1e-8."""
    N = 700
    v, w = gaussian_markers(N, 1.0, 0.6, seed=9)
    bp = uniform_bp(-6.0, 6.0, 8)
    om = oracle_mod.OracleMesh(bp, bp, 6)
    o = oracle_mod.Opts(m=5, max_iter=max_iter, tol=tol, abs_floor=0.0, damping=0.7,
                        stag_window=1000)
    S0 = om.entropy(om.l2_project(v, w))
    guess = om.predictor(o, v, w, 0.01)
    ref = om.step_anderson(o, guess, v, w, S0, 0.01)
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp))
    out = guess.copy(order="F")
    it = collops_mod.step_anderson(ws, out, v, w, S0, 0.01, m=5, max_iter=max_iter, tol=tol,
                                   abs_floor=0.0, damping=0.7, stag_window=1000)
    ws.close()
    assert (it[0] < max_iter) is done
    assert rel(out, ref[0]) < 1e-8
