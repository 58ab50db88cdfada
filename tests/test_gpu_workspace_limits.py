"""Every value of long stateless sums against the sums written out, and calls that
need more than the workspace keeps (256 MB of device, 32 MB of page-locked
memory), where some buffers are its own and others not.

Tolerance: 1e-12 of the largest value (FP64 sums of at most half a million
terms in another order, each term to a few ulp: below 1e-13); the same call before
and after others: the same bits.
"""
import math

import numpy as np
import pytest

import highreg

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _sources(nq, seed):
    rng = np.random.default_rng(seed)
    n = rng.standard_normal((nq, 3))
    n /= np.linalg.norm(n, axis=1)[:, None]
    return (0.7 * n).ravel(), n.ravel(), rng.uniform(0.5, 1.5, nq) / nq, rng.standard_normal(3 * nq)


def _written_out(xq, area, f, xt):
    """Plain Stokeslet and pressure sums, targets in slabs."""
    x, q, t = xq.reshape(-1, 3), f.reshape(-1, 3), xt.reshape(-1, 3)
    u, p = np.empty_like(t), np.empty(len(t))
    step = max(1, 4000000 // len(x))
    for i in range(0, len(t), step):
        d = t[i:i + step, None, :] - x[None, :, :]
        r = np.sqrt((d * d).sum(-1))
        fd = (d * q).sum(-1) * area / r ** 3
        u[i:i + step] = ((area / r) @ q + (d * fd[..., None]).sum(1)) / (8 * math.pi)
        p[i:i + step] = fd.sum(1) / (4 * math.pi)
    return u.ravel(), p


def _close(a, b):
    assert np.abs(a - b).max() < TOL * np.abs(b).max()


def _small(ctx):
    xq, nrm, area, f = _sources(300, 1)
    return np.concatenate([ctx.dl_onsurf(0.1, xq, nrm, area, f, mode=0), ctx.e2g_p_away(xq, area, f, xq + 2.0)])


@pytest.mark.parametrize("nt", [43690, 43691, 87400, 700001])
def test_every_value_of_long_arrays(ctx, nt):
    xq, _, area, f = _sources(40, 3)
    xt = (2.0 + np.random.default_rng(nt).uniform(0, 1, (nt, 3))).ravel()
    u, p = _written_out(xq, area, f, xt)
    _close(ctx.e2g_sl_away(xq, area, f, xt), u)
    _close(ctx.e2g_p_away(xq, area, f, xt), p)


def test_more_than_the_device_limit():
    ctx = highreg.Context(0)
    nt = 4000000  # targets and results 96 MB each, partial sums 128 MB
    xq, _, area, f = _sources(5, 4)
    xt = (2.0 + np.random.default_rng(4).uniform(0, 1, (nt, 3))).ravel()
    before = _small(ctx)
    u, p = _written_out(xq, area, f, xt)
    for _ in range(2):  # the second call on the workspace that the first left
        _close(ctx.e2g_sl_away(xq, area, f, xt), u)
        assert np.array_equal(_small(ctx), before)
        _close(ctx.e2g_p_away(xq, area, f, xt), p)
        assert np.array_equal(_small(ctx), before)
    ctx.close()


def test_more_than_the_page_locked_limit():
    ctx = highreg.Context(0)
    nq, nt = 524288, 87381  # seven arrays of 4 MB, three of 2 MB and smaller ones, collected for one copy
    xq, nrm, area, f = _sources(nq, 5)
    rng = np.random.default_rng(6)
    n0 = rng.standard_normal((nt, 3))
    n0 /= np.linalg.norm(n0, axis=1)[:, None]
    D = 0.01
    b = np.full(nt, 9.0 * D) + rng.uniform(0, 1, nt)  # beyond 8 delta: the plain Stokeslet
    xt = ((0.7 + b)[:, None] * n0).ravel()
    before = _small(ctx)
    at = np.sort(rng.choice(nt, 60, replace=False))
    u, _ = _written_out(xq, area, f, xt.reshape(-1, 3)[at].ravel())
    for _ in range(2):
        out = ctx.sl_offsurf(D, xq, nrm, area, f, xt, b, n0.ravel(), rng.standard_normal(3 * nt), mode=0)
        _close(out.reshape(-1, 3)[at].ravel(), u)
        assert np.array_equal(_small(ctx), before)
    ctx.close()
