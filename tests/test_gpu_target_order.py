"""A target's off-surface stresslet sum in FP64 depends on the other targets of the
call and on their order at rounding level only (a warp takes a pair beyond 8
delta in one of two forms for all its targets).

Tolerance: 1e-12 of the largest value, as for the same sums against the oracle.
"""
import numpy as np
import pytest

from test_gpu_eval64 import DEL, TOL, _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nt", [(65, 65), (515, 300), (1000, 1000)])
def test_permuted_and_fewer_targets(ctx, nq, nt):
    c = _case(nq, nt, nq + 3 * nt)
    D = 0.25 * DEL  # most pairs of the near targets are beyond 8 delta
    b = np.where(np.arange(nt) % 8 == 7, 9.0 * D, 0.25 * c["b"])
    x0, n0, f0 = (c[k].reshape(-1, 3) for k in ("x0", "n0", "f0"))
    xt = x0 + b[:, None] * n0
    a = (D, c["xq"], c["nrm"], c["area"], c["f"])
    rng = np.random.default_rng(nq)

    def sums(i):
        return ctx.dl_offsurf(*a, xt[i].ravel(), b[i], x0[i].ravel(), n0[i].ravel(), f0[i].ravel(), mode=0)

    every = np.arange(nt)
    whole = sums(every).reshape(-1, 3)
    for i in (rng.permutation(nt), np.sort(rng.choice(nt, nt // 3, replace=False)), every[-1:]):
        assert np.abs(sums(i).reshape(-1, 3) - whole[i]).max() < TOL * np.abs(whole).max()
