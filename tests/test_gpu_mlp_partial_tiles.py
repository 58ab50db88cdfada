"""Batches that do not fill the training kernel's tiles of 128 samples: what the
network gives for anything but the batch's samples does not reach the
gradient, here with weights for which it overflows at the input zero.

Tolerance: 2e-5 of the largest gradient entry, as in test_gpu_mlp_tiles.py (FP32
sums after three 64-term layers); the large products cancel exactly.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu
W2 = 12 * 64 + 64  # offset of the second layer's weights


@pytest.mark.parametrize("batch", [1, 5, 127, 128, 130])
def test_overflow_at_zero_input(ctx, batch):
    import torch

    import highreg

    rng = np.random.default_rng(batch)
    X = rng.standard_normal((batch, 12)).astype(np.float32)
    X[:, 0] = -1.0
    T = rng.standard_normal((batch, 3)).astype(np.float32)
    m = highreg.MLP(ctx, seed=3)
    p = m.params()
    # first feature of layer 1: 3e38 (x_0 + 1), zero for every sample; without
    # input 3e38, which overflows in layer 2
    p[0:12 * 64:64] = 0.0
    p[0] = p[12 * 64] = 3e38
    p[W2:W2 + 64] = 10.0
    m.set_params(p)
    loss, g = m.gradient(torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda(), batch)
    lo, go = mlp_oracle.loss_and_grad(p.astype(np.float64), X, T, np.zeros(12), np.ones(12), 1.0)
    assert abs(loss - lo) <= 1e-5 * lo
    assert np.abs(g - go).max() <= 2e-5 * np.abs(go).max()
