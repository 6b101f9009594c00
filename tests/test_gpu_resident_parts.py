"""Resident runs whose chunks are split into parts (few chunks, several blocks each) against the
one-launch-per-sweep schedule, which splits nothing: bit for bit, at the sizes where the split changes
(two chunks of a few cells, parts of just the halo width, many parts, no part left over)."""
import numpy as np
import pytest

from test_gpu_resident import _batch_run, _ctx_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 65, 130, 300, 513, 1000, 3001, 10007, 33000])
@pytest.mark.parametrize("order,limiter", [(1, 0), (2, 0), (2, 1)])
@pytest.mark.parametrize("prec,fold", [("mixed_f64", 0), ("mixed_kahan", 64), ("mixed_f64", 12)])
def test_parts_match_launch_per_sweep(shll, prec, fold, order, limiter, n):
    # a strong tube where the scheme allows it (first order): its chunks change to the pair flux and back
    ratio, temp = (50.0, 1.5) if order == 1 else (8.0, 0.9)
    p = shll.params(1, order, nx=n, precision=prec, limiter=limiter, fold_steps=fold, ic_rho_l=ratio, ic_T_l=temp,
                    ic_x_d=0.41)
    calls = [16 * 30 + 5, 64, 7]   # partial last sweeps, fold windows cut by a run's end
    a, ta, _ = _ctx_run(shll, p, calls, resident=False)
    b, tb, launches = _ctx_run(shll, p, calls, resident=True)
    if n >= 300:
        assert launches <= 9       # (resident)
    assert np.array_equal(a, b) and np.array_equal(ta, tb)


@pytest.mark.parametrize("order", [1, 2])
def test_parts_with_the_pair_flux_everywhere(shll, order):
    shll.set_pair_flux(2)
    try:
        p = shll.params(1, order, nx=2500, precision="mixed_f64", ic_rho_l=8.0)
        a, ta, _ = _ctx_run(shll, p, [150], resident=False)
        b, tb, _ = _ctx_run(shll, p, [150], resident=True)
    finally:
        shll.set_pair_flux(1)
    assert np.array_equal(a, b) and np.array_equal(ta, tb)


def test_parts_of_several_tubes(shll):
    items = [shll.params(1, 2, nx=n, precision="mixed_f64", ic_rho_l=r, t_end=0.02) for n, r in
             ((400, 3.0), (1700, 8.0), (901, 5.0), (3300, 2.0))]
    a, ta, _ = _batch_run(shll, items, resident=False)
    b, tb, _ = _batch_run(shll, items, resident=True)
    assert all(np.array_equal(x, y) for x, y in zip(a, b)) and np.array_equal(ta, tb)
