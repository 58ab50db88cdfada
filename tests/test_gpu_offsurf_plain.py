"""The off-surface stresslet's pairs beyond 8 delta: targets with subtraction
take them as plain stresslets of g - g0 where the target is x0 + b n0 with unit
n0; where it is not, the subtraction form is summed as it stands. Against the
oracle, which has only that form.

Tolerance: max |gpu - oracle| <= 1e-12 * max |oracle|, as for the other FP64
sums. With a target within 1e-13 delta of x0 + b n0 the two forms of a pair
beyond 8 delta differ by at most 5e-13 / 8 of the term.
"""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_eval64 import DEL, _case

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("nq,nt", [(3, 33), (66, 65), (515, 97), (1000, 300)])
@pytest.mark.parametrize("form", ["exact", "shifted foot", "longer normal", "one of many"])
def test_far_pairs_of_near_targets(ctx, oracle, nq, nt, form):
    c = _case(nq, nt, 10 * nq + nt)
    # a smaller delta: most pairs of the near targets are beyond 8 delta
    D = 0.25 * DEL
    far = np.arange(nt) % 8 == 7
    b = np.where(far, 9.0 * D, 0.25 * c["b"])
    x0, n0 = c["x0"].reshape(-1, 3), c["n0"].reshape(-1, 3).copy()
    xt = (x0 + b[:, None] * n0).ravel()
    x0 = x0.copy()
    if form == "shifted foot":
        x0 += 1e-3 * D
    elif form == "longer normal":
        n0 *= 1.0 + 1e-3
    elif form == "one of many":
        x0[nt // 2] += 1e-2 * D
    a = (D, c["xq"], c["nrm"], c["area"], c["f"])
    out = ctx.dl_offsurf(*a, xt, b, x0.ravel(), n0.ravel(), c["f0"], mode=0)
    assert rel_err(out, oracle.dl_offsurf_direct(*a, xt, b, x0.ravel(), n0.ravel(), c["f0"])) < TOL
