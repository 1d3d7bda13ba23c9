"""The attempt of step_anderson! on fixed-point pair sums: when it is made, when it ends,
and that the FP64 solve after it starts from the caller's guess. Counted by the maps; a
solve that cannot converge (tol and abs_floor 0) makes no attempt and gives the bits that
a solve after a failed attempt has to reproduce."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu

N = 700
DT = 0.01


class Case:
    def __init__(self, collops, oracle, weights="equal"):
        self.c = collops
        self.v, self.w = gaussian_markers(N, 1.0, 0.6, seed=9)
        if weights == "decades":
            self.w = self.w * 10.0 ** (-12 * np.random.default_rng(2).random(N))
        bp = uniform_bp(-6.0, 6.0, 8)
        om = oracle.OracleMesh(bp, bp, 6)
        self.S0 = om.entropy(om.l2_project(self.v, self.w))
        self.guess = np.asfortranarray(self.v * 0.999)
        self.ws = collops.build_workspace(collops.SimParameters(bp1=bp, bp2=bp))

    def solve(self, max_iter, tol, abs_floor=0.0, **kw):
        """(solution, iterations, residual, FP64 maps including the attempt's)"""
        out = self.guess.copy(order="F")
        assert self.c.load_library().co_profile(self.ws.h, 1) == 0
        it = self.c.step_anderson(self.ws, out, self.v, self.w, self.S0, DT, m=5,
                                  max_iter=max_iter, tol=tol, abs_floor=abs_floor,
                                  stag_window=1000, **kw)
        p = self.c.CoProfile()
        assert self.ws.lib.co_profile_read(self.ws.h, C.byref(p)) == 0
        return out, it[0], it[1], p.maps64


def test_converging_solve_needs_no_restart(built_lib, collops_mod, oracle_mod):
    k = Case(collops_mod, oracle_mod)
    _, it, _, maps = k.solve(200, 1e-12)
    k.ws.close()
    assert it < 48 and maps == it


@pytest.mark.parametrize("max_iter,attempt", [(7, 0), (8, 6), (30, 6)])
def test_hopeless_attempt_ends_early(built_lib, collops_mod, oracle_mod, max_iter, attempt):
    """A tolerance far below what FP64 can reach: given up at the sixth iteration."""
    k = Case(collops_mod, oracle_mod)
    ref, _, _, maps0 = k.solve(max_iter, 0.0)
    out, it, _, maps = k.solve(max_iter, 1e-200)
    k.ws.close()
    assert maps0 == max_iter and it == max_iter and maps == max_iter + attempt
    assert np.array_equal(out, ref)


def test_attempt_ends_at_its_limit(built_lib, collops_mod, oracle_mod):
    """Damped Picard steps converge at a steady rate: 60 to a floor set by the residual
    of the 60th, on pace throughout, so the attempt runs to its limit of 48."""
    k = Case(collops_mod, oracle_mod)
    kw = dict(damping=0.05, use_anderson=False)
    ref, _, res, maps0 = k.solve(60, 0.0, **kw)
    out, it, _, maps = k.solve(200, 0.0, abs_floor=res * (1 + 1e-9), **kw)
    k.ws.close()
    assert maps0 == 60 and it == 60 and maps == 48 + 60
    assert np.array_equal(out, ref)


def test_wide_operands_end_the_attempt(built_lib, collops_mod, oracle_mod):
    """Weights over twelve decades: the operands are left to FP64 arithmetic, and the solve
    starts again on the FP64 kernels after one map."""
    k = Case(collops_mod, oracle_mod, "decades")
    ref, _, _, maps0 = k.solve(12, 0.0)
    out, it, _, maps = k.solve(12, 1e-200)
    k.ws.close()
    assert maps0 == 12 and maps == 13
    assert np.array_equal(out, ref)
