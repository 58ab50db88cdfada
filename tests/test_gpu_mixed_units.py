"""The reduced-precision two-surface sums at the edges of their tiles and half
blocks, with odd source counts (half-filled pairs) and treecode degrees from 1
to 15 (rows of an odd and an even number of proxies), against the FP64 oracle.

Tolerance: 3e-5 of the largest value. A pair's FP32 operations cost some 25
roundings of 6e-8; coordinates relative to the block's origin, up to 1.5 long,
are off by 9e-8, which the kernels at distances from delta = 0.1 amplify to at
most 5e-6 of a term; random signs let both grow as the sums themselves do.
"""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_eval64 import DEL, SIZES, _case

import highreg

pytestmark = pytest.mark.gpu
TOL = 3e-5


@pytest.mark.parametrize("nq,nt", SIZES)
def test_direct_sums(ctx, oracle, nq, nt):
    c = _case(nq, nt, 100 * nq + nt)
    a = (DEL, c["xq"], c["nrm"], c["area"], c["f"])
    m = dict(mode=0, precision=highreg.HR_MIXED)
    assert rel_err(ctx.sl_onsurf(*a, **m), oracle.sl_onsurf_direct(*a)) < TOL
    assert rel_err(ctx.dl_onsurf(*a, **m), oracle.dl_onsurf_direct(*a)) < TOL
    out = ctx.sl_offsurf(*a, c["xt"], c["b"], c["n0"], c["f0"], **m)
    assert rel_err(out, oracle.sl_offsurf_direct(*a, c["xt"], c["b"], c["f0"], c["n0"])) < TOL
    out = ctx.dl_offsurf(*a, c["xt"], c["b"], c["x0"], c["n0"], c["f0"], **m)
    assert rel_err(out, oracle.dl_offsurf_direct(*a, c["xt"], c["b"], c["x0"], c["n0"], c["f0"])) < TOL


@pytest.mark.parametrize("P", [1, 2, 4, 5, 6, 7, 10, 15])
def test_treecode_degrees(ctx, oracle, g2s, P):
    rng = np.random.default_rng(P)
    N0, D = 120, float(g2s["DEL"])
    for kind, on in ((0, True), (1, False), (2, True), (3, False)):
        s, t = (0, 0) if on else (1, 0)
        xq, nrm, area, ctr = g2s["xq%d" % s], g2s["nrm%d" % s], g2s["area%d" % s], g2s["ctr%d" % s]
        q = rng.standard_normal(len(xq))
        opt = dict(mode=1, P=P, N0=N0, theta=0.6, ctr=ctr, precision=highreg.HR_MIXED)
        if on:
            ref, _ = oracle.kitc(kind, P, N0, 0.6, ctr, D, xq, nrm, area, q)
            out = (ctx.sl_onsurf if kind == 0 else ctx.dl_onsurf)(D, xq, nrm, area, q, **opt)
        else:
            xt, b, x0, n0 = g2s["xq0"], g2s["b0"], g2s["x00"], g2s["n00"]
            q0 = rng.standard_normal(len(xt))
            ref, _ = oracle.kitc(kind, P, N0, 0.6, ctr, D, xq, nrm, area, q, xt=xt, b=b, x0=x0, n0=n0, dens0=q0)
            out = (ctx.sl_offsurf(D, xq, nrm, area, q, xt, b, n0, q0, **opt) if kind == 1 else
                   ctx.dl_offsurf(D, xq, nrm, area, q, xt, b, x0, n0, q0, **opt))
        assert rel_err(out, ref) < TOL
