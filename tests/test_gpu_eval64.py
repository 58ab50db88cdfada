"""The FP64 boundary-sum kernels at the edges of their tiles, half blocks and
smoothing pieces, and at treecode degrees from 1 to 15, against the oracle.

Tolerance: max |gpu - oracle| <= 1e-12 * max |oracle|, as for the other FP64
sums: a pair's terms agree to a few ulp (1e-15 relative), and sums of at most a
few thousand of them in another order stay far below 1e-12 of the largest.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-12
DEL = 0.1


def _unit(rng, n):
    v = rng.standard_normal((n, 3))
    return v / np.linalg.norm(v, axis=1)[:, None]


def _case(nq, nt, seed):
    """Sources on a sphere, targets off it (b is the distance to the sphere):
    some right above a source at a distance next to a smoothing piece's edge or
    to a switch to the plain kernel, one on a source, some far."""
    rng = np.random.default_rng(seed)
    n = _unit(rng, nq)
    x = 0.7 * n
    n0 = _unit(rng, nt)
    b = DEL * rng.uniform(-6.5, 7.9, nt)
    for i, s in enumerate([0.0, 0.125, 0.375, 50.999, 51.001, 63.999, 64.001]):
        if i < nt:  # s = b^2 / delta^2 above source i mod nq
            n0[i] = n[i % nq]
            b[i] = DEL * np.sqrt(s)
    x0 = 0.7 * n0
    far = np.arange(nt) % 8 == 7
    b[far] = 9.0 * DEL
    xt = x0 + b[:, None] * n0
    if nt > 0:
        xt[0] = x[0]  # exactly
    f0 = rng.standard_normal((nt, 3))
    return dict(xq=x.ravel(), nrm=n.ravel(), area=rng.uniform(0.5, 1.5, nq) / nq, f=rng.standard_normal(3 * nq),
                xt=xt.ravel(), b=b, x0=x0.ravel(), n0=n0.ravel(), f0=f0.ravel())


SIZES = [(1, 1), (2, 31), (31, 33), (33, 64), (65, 65), (127, 129), (513, 97), (1000, 300)]


@pytest.mark.parametrize("nq,nt", SIZES)
def test_direct_sums(ctx, oracle, nq, nt):
    c = _case(nq, nt, 100 * nq + nt)
    a = (DEL, c["xq"], c["nrm"], c["area"], c["f"])
    assert rel_err(ctx.sl_onsurf(*a, mode=0), oracle.sl_onsurf_direct(*a)) < TOL
    assert rel_err(ctx.dl_onsurf(*a, mode=0), oracle.dl_onsurf_direct(*a)) < TOL
    out = ctx.sl_offsurf(*a, c["xt"], c["b"], c["n0"], c["f0"], mode=0)
    assert rel_err(out, oracle.sl_offsurf_direct(*a, c["xt"], c["b"], c["f0"], c["n0"])) < TOL
    out = ctx.dl_offsurf(*a, c["xt"], c["b"], c["x0"], c["n0"], c["f0"], mode=0)
    assert rel_err(out, oracle.dl_offsurf_direct(*a, c["xt"], c["b"], c["x0"], c["n0"], c["f0"])) < TOL


@pytest.mark.parametrize("nq,nt", SIZES)
def test_extend_to_grid_sums(ctx, oracle, nq, nt):
    c = _case(nq, nt, 100 * nq + nt + 7)
    away = c["xt"] + np.tile([2.0, 0.0, 0.0], nt)
    p = (c["xq"], c["area"], c["f"], away)
    assert rel_err(ctx.e2g_sl_away(*p), oracle.e2g_sl_away(*p)) < TOL
    assert rel_err(ctx.e2g_p_away(*p), oracle.e2g_p_away(*p)) < TOL
    b = np.minimum(c["b"], 7.9 * DEL)
    a = (DEL, c["xq"], c["nrm"], c["area"], c["f"], c["xt"], b, c["f0"], c["n0"])
    assert rel_err(ctx.e2g_sl_7ord(*a), oracle.e2g_sl_7ord(*a)) < TOL
    assert rel_err(ctx.e2g_p_7ord(*a), oracle.e2g_p_7ord(*a)) < TOL


@pytest.mark.parametrize("P", [1, 2, 4, 7, 10, 15])
def test_treecode_degrees(ctx, oracle, g2s, P):
    rng = np.random.default_rng(P)
    N0, D = 120, float(g2s["DEL"])
    for kind, on in ((0, True), (1, False), (2, True), (3, False)):
        s, t = (0, 0) if on else (1, 0)
        xq, nrm, area, ctr = g2s["xq%d" % s], g2s["nrm%d" % s], g2s["area%d" % s], g2s["ctr%d" % s]
        q = rng.standard_normal(len(xq))
        opt = dict(mode=1, P=P, N0=N0, theta=0.6, ctr=ctr)
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
