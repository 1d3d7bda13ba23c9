"""The network kernels at the edges of their tiles: one sample, one tile less or more
than full, a last tile of one sample, and more tiles than blocks.

Tolerances: FP32 sums of up to 64 terms through four layers, 1e-5 of the largest
output, times ten; per-sample gradients likewise, summed over the batch in FP32
(2e-3 in the 2-norm, as for the gradient check of the whole network).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in", [9, 15])
@pytest.mark.parametrize("B", [1, 63, 64, 65, 129, 9729])
def test_tile_edges(built_lib, collops_mod, B, n_in):
    import torch
    from collops import learned
    from oracle import mlp as om
    net = learned.MLP(seed=4, n_in=n_in)
    p = net.get_params()
    rng = np.random.default_rng(B)
    X = rng.standard_normal((B, n_in)).astype(np.float32)
    T = rng.standard_normal((B, 2)).astype(np.float32)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    Y = torch.full((B + 1, 2), 7.0, dtype=torch.float32, device="cuda")
    net.forward(Xd, Y[:B])
    y_ref, _ = om.forward(p, X.astype(np.float64), n_in)
    y = Y.cpu().numpy()
    assert np.max(np.abs(y[:B] - y_ref)) <= 1e-4 * max(1.0, np.max(np.abs(y_ref)))
    assert np.all(y[B:] == 7.0)
    loss_ref, g_ref = om.loss_and_grad(p, X, T, n_in)
    g, loss = net.gradients(Xd, Td)
    g2, loss2 = net.gradients(Xd, Td)
    net.close()
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref
    assert np.linalg.norm(g - g_ref) <= 2e-3 * np.linalg.norm(g_ref)
    assert loss == loss2 and np.array_equal(g, g2)
