"""The Poisson transform from one array to another: the input stays as it is, and
the result has the bits of the transform in place."""
import ctypes

import numpy as np
import pytest

import highreg

pytestmark = pytest.mark.gpu


def _call(ctx, n, src, dst):
    p = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in (src, dst)]
    ctx._check(highreg.lib().hr_dst_poisson3d_to(ctx.p, n, *p))


@pytest.mark.parametrize("n", [1, 7, 45, 63, 95])
def test_out_of_place(ctx, n):
    f = np.random.default_rng(n).standard_normal((n, n, n))
    keep, place, out = f.copy(), f.copy(), np.full((n, n, n), np.nan)
    ctx._check(highreg.lib().hr_dst_poisson3d(ctx.p, n, place.ctypes.data_as(ctypes.POINTER(ctypes.c_double))))
    _call(ctx, n, f, out)
    assert np.array_equal(f, keep) and np.array_equal(out, place)
    both = f.copy()
    _call(ctx, n, both, both)
    assert np.array_equal(both, place)
    for a in (f, f.ravel(), f[::-1][::-1], np.asfortranarray(f)):
        b = a.copy()
        r = ctx.dst_poisson3d(n, a)
        assert r is not a and r.shape == a.shape and np.array_equal(r.ravel(), place.ravel()) and np.array_equal(a, b)
    longer = np.concatenate([f.ravel(), [3.0, 4.0]])
    r = ctx.dst_poisson3d(n, longer)
    assert np.array_equal(r[:-2], place.ravel()) and np.array_equal(r[-2:], [3.0, 4.0])
