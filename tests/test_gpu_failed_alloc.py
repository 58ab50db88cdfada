"""A training step whose workspace does not fit the GPU fails with an error, and
the steps after it work: they give the loss of a network that made none.
Tolerance: none, the same steps."""
import numpy as np
import pytest

import highreg

pytestmark = pytest.mark.gpu


def test_training_goes_on_after_a_batch_too_large(ctx):
    import torch

    rng = np.random.default_rng(5)
    X = torch.from_numpy(rng.standard_normal((500, 12)).astype(np.float32)).cuda()
    T = torch.from_numpy(rng.standard_normal((500, 3)).astype(np.float32)).cuda()
    nets = [highreg.MLP(ctx, seed=1) for _ in range(2)]
    nets[0].train_step(X, T, 300, 1e-3, seed=9)
    nets[1].train_step(X, T, 300, 1e-3, seed=9)
    with pytest.raises(highreg.HrError):
        nets[0].train_step(X, T, 1 << 30, 1e-3, seed=9)  # 2^23 tiles of 37 kB
    for batch in (200, 300, 400):
        a, b = (m.train_step(X, T, batch, 1e-3, seed=9, want_loss=True) for m in nets)
        assert a == b
    assert np.array_equal(nets[0].params(), nets[1].params())
