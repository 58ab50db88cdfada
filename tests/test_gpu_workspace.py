"""Stateless calls share a workspace kept by their context: calls of other
sizes and kinds before do not change a result, and arrays around the limits of
the staged copies (1 MB direct, chunks of an eighth from 512 KB to 16 MB)
arrive whole.

Tolerances: after other calls on the same context the same call gives the same
bits (same kernels, same order). A long array against the same targets in
separate short calls: 1e-12 of the largest value, as for other FP64 sums in
another order.
"""
import numpy as np
import pytest

import highreg
from conftest import rel_err

pytestmark = pytest.mark.gpu


def _sources(nq, seed):
    rng = np.random.default_rng(seed)
    n = rng.standard_normal((nq, 3))
    n /= np.linalg.norm(n, axis=1)[:, None]
    return (0.7 * n).ravel(), n.ravel(), rng.uniform(0.5, 1.5, nq) / nq, rng.standard_normal(3 * nq)


def test_other_calls_before_change_nothing():
    def calls(ctx, which):
        out = {}
        for nq in which:
            xq, nrm, area, f = _sources(nq, nq)
            out[nq] = [ctx.sl_onsurf(0.1, xq, nrm, area, f, mode=0), ctx.dl_onsurf(0.1, xq, nrm, area, f, mode=1, P=3, N0=50),
                       ctx.e2g_sl_away(xq, area, f, xq + 2.0), ctx.dst_poisson3d(7, f[:343] if nq >= 115 else np.ones(343))]
        return out

    ctx = highreg.Context(0)
    a = calls(ctx, [200, 5000, 30, 1])
    b = calls(ctx, [1, 30, 200, 5000])
    for nq in a:
        alone = highreg.Context(0)
        c = calls(alone, [nq])[nq]
        alone.close()
        for u, v, w in zip(a[nq], b[nq], c):
            assert np.array_equal(u, v) and np.array_equal(u, w)
    ctx.close()


@pytest.mark.parametrize("nt", [43690, 43691, 87400, 700001])
def test_long_arrays(ctx, nt):
    xq, nrm, area, f = _sources(40, 3)
    rng = np.random.default_rng(nt)
    xt = (2.0 + rng.uniform(0, 1, (nt, 3))).ravel()
    u, p = ctx.e2g_sl_away(xq, area, f, xt), ctx.e2g_p_away(xq, area, f, xt)
    for i0 in (0, nt // 2 - 500, nt - 1000):
        s = xt[3 * i0:3 * i0 + 3000]
        assert rel_err(u[3 * i0:3 * i0 + 3000], ctx.e2g_sl_away(xq, area, f, s)) < 1e-12
        assert rel_err(p[i0:i0 + 1000], ctx.e2g_p_away(xq, area, f, s)) < 1e-12
    # every value, against the sum written out
    d = xt.reshape(-1, 1, 3) - xq.reshape(1, -1, 3) if nt < 100000 else None
    if d is not None:
        r2 = (d * d).sum(-1)
        fd = (d * f.reshape(1, -1, 3)).sum(-1)
        q = (area[None, :] * fd * r2 ** -1.5).sum(1)
        k = np.argmax(np.abs(q))
        assert np.max(np.abs(p - q * (p[k] / q[k]))) < 1e-12 * np.max(np.abs(p))
