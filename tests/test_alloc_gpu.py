"""A call that needs more device memory than there is returns CO_ERR_NOMEM and leaves the
context usable: the next, smaller call allocates what it needs and gives the result of the
same call before. Requests are sized beyond the whole memory of the GPU at hand, so that
nothing runs on the buffers of the failed call."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import gaussian_markers, uniform_bp

pytestmark = pytest.mark.gpu

CO_ERR_NOMEM = 6


def _small(collops, ws, v, w):
    out = np.zeros_like(v, order="F")
    collops.picard_map(ws, out, v, v, w, 1.0, 0.02, precision="mixed_ds")
    G, F, A = np.asfortranarray(-v), np.zeros_like(v, order="F"), np.zeros((len(w), 3), order="F")
    collops.compute_collision_metric_gpu(ws, F, A, v, w, G)
    return np.concatenate([out, F, A], axis=1)


def _setup(collops):
    bp = uniform_bp(-8.0, 8.0, 16)
    v, w = gaussian_markers(2048, 1.0, 0.6, seed=3)
    ws = collops.build_workspace(collops.SimParameters(bp1=bp, bp2=bp))
    return ws, v, w, _small(collops, ws, v, w)


def test_partials(built_lib, collops_mod):
    """Pair partials of 2.2 million markers: N^2 / 16 bytes and an eighth more, 340 GB."""
    import torch

    if torch.cuda.mem_get_info()[1] > 320e9:
        pytest.skip("the partials would fit")
    ws, v, w, ref = _setup(collops_mod)
    V, W = gaussian_markers(2200000, 1.0, 0.6, seed=4)
    with pytest.raises(collops_mod.CollopsError) as e:
        collops_mod.picard_map(ws, np.zeros_like(V, order="F"), V, V, W, 1.0, 0.02,
                               precision="mixed_ds")
    assert e.value.status == CO_ERR_NOMEM
    assert np.array_equal(_small(collops_mod, ws, v, w), ref)
    ws.close()


def test_marker_buffers(built_lib, collops_mod):
    """The first fourteen marker buffers, of 16 bytes a marker, a tenth beyond the memory."""
    import torch

    N = int(1.1 * torch.cuda.mem_get_info()[1] / (14 * 16))
    if N > 2 ** 31 - 512:
        pytest.skip("no int holds so many markers")

    ws, v, w, ref = _setup(collops_mod)
    x = torch.zeros(16, dtype=torch.float64, device="cuda")   # not read: the call fails first
    o = ws.p.opts()
    rc = ws.lib.co_predictor_dev(ws.h, C.byref(o), x.data_ptr(), x.data_ptr(),
                                             x.data_ptr(), N, 0.02)
    assert rc == CO_ERR_NOMEM
    assert np.array_equal(_small(collops_mod, ws, v, w), ref)
    ws.close()
