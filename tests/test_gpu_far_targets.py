"""Targets beyond 8 delta of the surface take the plain kernels, which read
neither the nearest point nor its normal (2S/KITC.cpp:856-882, 970-995): what
those arrays hold there, as where no nearest point was searched, changes
nothing.

Tolerance: none, the same bits.
"""
import numpy as np
import pytest

import highreg
from test_gpu_eval64 import DEL, _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nt", [(3, 33), (65, 64), (515, 300)])
@pytest.mark.parametrize("unset", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("precision", [highreg.HR_FP64, highreg.HR_MIXED, highreg.HR_FP32])
def test_unset_nearest_point_of_far_targets(ctx, nq, nt, unset, precision):
    c = _case(nq, nt, nq + nt)
    far = np.abs(c["b"]) > 8 * DEL
    assert far.any() and not far.all()

    def with_(v):
        x0, n0 = c["x0"].reshape(-1, 3).copy(), c["n0"].reshape(-1, 3).copy()
        x0[far], n0[far] = v, v
        return x0.ravel(), n0.ravel()

    a = (DEL, c["xq"], c["nrm"], c["area"], c["f"])
    for mode in (dict(mode=0), dict(mode=1, P=4, N0=60)):
        outs = [ctx.dl_offsurf(*a, c["xt"], c["b"], x0, n0, c["f0"], precision=precision, **mode)
                for x0, n0 in (with_(0.0), with_(unset))]
        assert np.isfinite(outs[0]).all()
        assert np.array_equal(outs[0], outs[1])
    # the treecode's proxies take f0.n0 of every target, the direct Stokeslet sum only of near ones
    outs = [ctx.sl_offsurf(*a, c["xt"], c["b"], n0, c["f0"], precision=precision, mode=0)
            for _, n0 in (with_(0.0), with_(unset))]
    assert np.isfinite(outs[0]).all()
    assert np.array_equal(outs[0], outs[1])
