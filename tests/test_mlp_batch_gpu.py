"""A training batch whose last sample indices are the largest an int holds: 2^31 - 1
samples, all alike, against a batch of one tile of the same samples (the mean of the loss
and of the gradients does not depend on their number).

Tolerances: the loss is summed in FP64 (1e-5 as for the other batches); a gradient is
summed in FP32 over 64 samples and then over 2^31 / 64 / 152 = 220,753 tiles of a block,
one after another, an error of at most 220,753 x 2^-24 = 1.3e-2 of its size.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_largest_batch(built_lib, collops_mod):
    import torch
    from collops import learned

    net = learned.MLP(seed=4, n_in=1, n_out=1)
    B = 2 ** 31 - 1
    X = torch.full((B, 1), 0.5, dtype=torch.float32, device="cuda")
    T = torch.full((B, 1), 1.0, dtype=torch.float32, device="cuda")
    g, loss = net.gradients(X, T)
    g1, loss1 = net.gradients(X[:64], T[:64])
    net.close()
    assert abs(loss - loss1) <= 1e-5 * loss1
    assert np.max(np.abs(g - g1)) <= 1.3e-2 * np.max(np.abs(g1))
