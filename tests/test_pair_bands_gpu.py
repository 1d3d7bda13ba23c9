"""The fixed-point pair sum in bands of tile pairs: F with the metric at sizes where the
partials of all tile pairs would not fit the buffer's 2^30 bytes (from about 82,000
markers on), one band less and one more, against sums in extended precision, and the
memory the call leaves allocated.

Tolerance: a term is rounded to at most 6 units of 2^-53 of its size; the partials of a
marker, one per tile pair, are added in 8 chains and the bands in one: with nt / 16 / 8
adds a chain, 8 chains and 4 bands, 5 + nt / 128 + 12 units of the sum of the sizes.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [81000, 84000, 120001])
def test_bands(built_lib, collops_mod, N):
    import torch

    v, w = gaussian_markers(N, 1.0, 0.6, seed=N)     # all inside [-8, 8]
    rng = np.random.default_rng(1)
    w = rng.uniform(0.2, 1.8, N) / N
    G = np.asfortranarray(-v / [1.0, 0.36] + 0.05 * rng.standard_normal(v.shape))
    bp = uniform_bp(-8.0, 8.0, 32)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp))
    F, A, F2 = (np.zeros((N, k), order="F") for k in (2, 3, 2))
    collops_mod.compute_collision_metric_gpu(ws, F, A, v, w, G)
    used = free - torch.cuda.mem_get_info()[0]
    collops_mod.compute_collision_gpu(ws, F2, v, w, G)
    ws.close()
    assert used < 2 ** 30 + 2 ** 28 + N * 1500     # partials of both sides, marker buffers
    L = np.longdouble
    unit = (17 + N / 128 / 128) * 2.0 ** -53
    for g in rng.integers(0, N, 6):
        d, q = v[g].astype(L) - v.astype(L), G.astype(L) - G[g].astype(L)
        r = np.sqrt((d * d).sum(1))
        r[g] = np.inf
        k = w.astype(L) / r ** 3
        c = k * (q[:, 0] * d[:, 1] - q[:, 1] * d[:, 0])
        Fr = np.array([(c * d[:, 1]).sum(), -(c * d[:, 0]).sum()])
        Ar = np.array([(k * d[:, 1] ** 2).sum(), -(k * d[:, 0] * d[:, 1]).sum(),
                       (k * d[:, 0] ** 2).sum()])
        sf, sa = (w * np.sqrt((q * q).sum(1)) / r).sum(), (w / r).sum()
        assert np.all(np.abs(F[g] - Fr) <= unit * sf)
        assert np.all(np.abs(F2[g] - Fr) <= unit * sf)
        assert np.all(np.abs(A[g] - Ar) <= unit * sa)
