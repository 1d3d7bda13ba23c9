"""The guard of the pair sum (|d|^2 < 1e-24 is skipped, functions.jl:224) in every FP64 form:
pairs on both sides of it against the CPU oracle. Their terms, of size 1e12, dominate both
sums: a form that draws the line elsewhere is off by all of its value.

Tolerance: one dominant term, a dozen roundings of 2^-53: 1e-14.
"""
from __future__ import annotations

import struct

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

@pytest.mark.gpu
@pytest.mark.parametrize("gap", [0.9e-12, 1.1e-12, 2e-12, 3.1e-12, 3.3e-12])
@pytest.mark.parametrize("form", ["small", "onesided", "fixed", "wide", "noalloc"])
def test_guard(built_lib, collops_mod, oracle_mod, form, gap):
    import torch

    N = 300 if form == "small" else 1000
    v, w = gaussian_markers(N, 1.0, 0.6, seed=2)
    rng = np.random.default_rng(3)
    G = np.asfortranarray(rng.standard_normal((N, 2)))
    v[1] = v[0] + (gap, 0.0)
    v[N - 1] = v[N // 2] + (0.0, gap)
    if form == "wide":
        w[7], G[7] = 0.0, 1e9
    bp = uniform_bp(-6.0, 6.0, 8)
    ref, Ar = oracle_mod.OracleMesh(bp, bp, 6).collision_metric(v, w, G)
    ws = collops_mod.build_workspace(
        collops_mod.SimParameters(bp1=bp, bp2=bp, pair_onesided=form == "onesided"))
    out, F, A = (np.zeros((N, k), order="F") for k in (2, 2, 3))
    if form == "noalloc":
        t = [torch.from_numpy(np.ascontiguousarray(a.T)).cuda() for a in (v, w, G, out)]
        assert ws.lib.co_collision_noalloc(*(a.data_ptr() for a in t), N, bp[0], bp[-1], bp[0],
                                           bp[-1], None) == 0
        torch.cuda.synchronize()
        out = t[3].cpu().numpy().T
    else:
        collops_mod.compute_collision_gpu(ws, out, v, w, G)
        collops_mod.compute_collision_metric_gpu(ws, F, A, v, w, G)
        assert np.max(np.abs(A - Ar)) <= 1e-14 * np.max(np.abs(Ar))
    ws.close()
    near = [0, 1, N // 2, N - 1]
    size = np.max(np.abs(ref[near]))
    assert (size > 1e6) == (gap > 1e-12)
    if gap > 1e-12:
        assert np.max(np.abs(out[near] - ref[near])) <= 1e-14 * size
    else:
        assert np.max(np.abs(out[near])) < 1e6


def test_the_constant():
    import os

    import build
    text = open(os.path.join(build.CSRC, "co_pair64.cuh")).read()
    bits = struct.unpack("<q", struct.pack("<d", 1e-24))[0]
    assert f"#define CO_R2_MIN_BITS 0x{bits:X}LL" in text
