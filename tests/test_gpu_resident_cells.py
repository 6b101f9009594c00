"""Resident runs with one cell per thread (small windows) and two (large ones) against the
one-launch-per-sweep schedule, which has two everywhere: bit for bit, at the largest tubes whose chunks
are still split in two (windows below the limit) and the next size (whole chunks), and at windows that
end inside a warp."""
import numpy as np
import pytest

from test_gpu_resident import _ctx_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["mixed_f64", "mixed_kahan"])
@pytest.mark.parametrize("order,limiter,n", [
    (1, 0, 76 * 480), (1, 0, 76 * 480 + 1), (2, 0, 76 * 448), (2, 1, 76 * 448 + 1), (2, 0, 20011), (1, 0, 7777),
    (2, 1, 641), (1, 0, 97)])
def test_cells_per_thread_keep_the_bits(shll, order, limiter, n, prec):
    ratio, temp = (30.0, 1.3) if order == 1 else (8.0, 0.9)
    p = shll.params(1, order, nx=n, precision=prec, limiter=limiter, ic_rho_l=ratio, ic_T_l=temp, ic_x_d=0.6)
    calls = [16 * 21 + 3, 16]
    a, ta, _ = _ctx_run(shll, p, calls, resident=False)
    b, tb, _ = _ctx_run(shll, p, calls, resident=True)
    assert np.array_equal(a, b) and np.array_equal(ta, tb)
