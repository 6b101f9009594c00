"""Resident 1D runs of few steps: with fewer than six (second order and many blocks: nine) the chunks are not split
into parts, from there on they are. Any row of such calls leaves the bits of the one-launch-per-sweep schedule."""
import numpy as np
import pytest

from test_gpu_resident import _ctx_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [97, 1500, 5000, 20011])
@pytest.mark.parametrize("order,limiter", [(1, 0), (2, 1)])
@pytest.mark.parametrize("prec", ["mixed_f64", "mixed_kahan"])
def test_short_calls(shll, prec, order, limiter, n):
    p = shll.params(1, order, nx=n, precision=prec, limiter=limiter, ic_rho_l=30.0 if order == 1 else 8.0, ic_x_d=0.41)
    calls = [1, 6, 5, 16, 2, 8, 9, 40, 3]
    a, ta, _ = _ctx_run(shll, p, calls, resident=False)
    b, tb, launches = _ctx_run(shll, p, calls, resident=True)
    assert launches == (3 if order == 1 else 2) * len(calls)
    assert np.array_equal(a, b) and np.array_equal(ta, tb)
