"""The direct sums do not depend on the unit of length: lengths scaled by a power
of two, from delta = 1e-10 to 1e29, against the oracle. (The treecode's root box
is of fixed size, 2S/KITC.cpp:30.)

Tolerance: max |gpu - oracle| <= 1e-12 * max |oracle|, as for the other FP64
sums; scaling by a power of two adds no rounding.
"""
import numpy as np
import pytest

from test_gpu_eval64 import DEL, TOL, _case
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nt", [(33, 64), (513, 97)])
@pytest.mark.parametrize("power", [-30, 0, 30, 45, 60, 100])
def test_scaled_lengths(ctx, oracle, nq, nt, power):
    c = _case(nq, nt, 100 * nq + nt)
    s = 2.0 ** power
    a = (s * DEL, s * c["xq"], c["nrm"], c["area"], c["f"])
    xt, b, x0 = s * c["xt"], s * c["b"], s * c["x0"]
    assert rel_err(ctx.sl_onsurf(*a, mode=0), oracle.sl_onsurf_direct(*a)) < TOL
    assert rel_err(ctx.dl_onsurf(*a, mode=0), oracle.dl_onsurf_direct(*a)) < TOL
    out = ctx.sl_offsurf(*a, xt, b, c["n0"], c["f0"], mode=0)
    assert rel_err(out, oracle.sl_offsurf_direct(*a, xt, b, c["f0"], c["n0"])) < TOL
    # the stresslet's jump g0 does not scale: compare the sums without it
    out = ctx.dl_offsurf(*a, xt, b, x0, c["n0"], c["f0"], mode=0)
    ref = oracle.dl_offsurf_direct(*a, xt, b, x0, c["n0"], c["f0"])
    sums = np.repeat(c["b"] > 1e-6 * DEL, 3)
    assert rel_err(out, ref) < TOL
    assert rel_err(out[sums], ref[sums]) < TOL
    b = np.minimum(b, 7.9 * s * DEL)
    a += (xt, b, c["f0"], c["n0"])
    assert rel_err(ctx.e2g_sl_7ord(*a), oracle.e2g_sl_7ord(*a)) < TOL
    assert rel_err(ctx.e2g_p_7ord(*a), oracle.e2g_p_7ord(*a)) < TOL
