"""The training kernel at batches around its tile of 128 samples, against the
FP64 oracle.

Tolerance: every gradient entry is an FP32 sum of at most `batch` terms after
three 64-term layers; rounding gives a few 1e-6 of the largest entry, 2e-5 is
asked (the smallest reductions are exact sums of a handful of terms).
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 63, 127, 128, 129, 300, 1025])
def test_gradient_at_tile_edges(ctx, batch):
    import torch

    import highreg

    rng = np.random.default_rng(batch)
    X = rng.standard_normal((batch, 12)).astype(np.float32)
    T = rng.standard_normal((batch, 3)).astype(np.float32)
    mean, std = rng.normal(0, 0.1, 12).astype(np.float32), rng.uniform(0.8, 1.2, 12).astype(np.float32)
    m = highreg.MLP(ctx, seed=batch)
    m.set_normalization(mean, std, 1.3)
    p = m.params().astype(np.float64)
    loss, g = m.gradient(torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda(), batch)
    lo, go = mlp_oracle.loss_and_grad(p, X, T, mean.astype(np.float64), std.astype(np.float64), 1.3)
    assert abs(loss - lo) <= 1e-5 * lo
    assert np.abs(g - go).max() <= 2e-5 * np.abs(go).max()
