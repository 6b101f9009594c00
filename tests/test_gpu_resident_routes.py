"""Resident 1D runs: that they are what runs at the sizes where their form changes (whole chunks and parts, one
cell per thread and two), counted by launches, and that each form keeps the bits of the one-launch-per-sweep
schedule, with a grid constant that is a power of two and one that is not (then every interface term is a pair)."""
import numpy as np
import pytest

from test_gpu_resident import _batch_run, _ctx_run

pytestmark = pytest.mark.gpu


def sm_count():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


# (order, limiter, cells from the number of SMs): the largest tube whose chunks are split in two and the next
# (windows of one cell per thread, then of two), one chunk per SM, parts of many sizes
TUBES = [(1, 0, lambda sms: sms // 2 * 480), (1, 0, lambda sms: sms // 2 * 480 + 1), (1, 0, lambda sms: sms * 480),
         (2, 0, lambda sms: sms // 2 * 448), (2, 1, lambda sms: sms // 2 * 448 + 1), (2, 1, lambda sms: sms * 448),
         (2, 0, lambda sms: 20011), (1, 0, lambda sms: 7777), (2, 1, lambda sms: 641), (1, 0, lambda sms: 97)]


@pytest.mark.parametrize("prec", ["mixed_f64", "mixed_kahan"])
@pytest.mark.parametrize("cfl", [0.25, 0.3])
@pytest.mark.parametrize("order,limiter,cells", TUBES)
def test_tubes(shll, order, limiter, cells, cfl, prec):
    n = cells(sm_count())
    ratio, temp = (30.0, 1.3) if order == 1 else (8.0, 0.9)
    p = shll.params(1, order, nx=n, precision=prec, limiter=limiter, cfl=cfl, fold_steps=64, ic_rho_l=ratio, ic_T_l=temp,
                    ic_x_d=0.6)
    calls = [16 * 21 + 3, 16]
    a, ta, la = _ctx_run(shll, p, calls, resident=False)
    b, tb, lb = _ctx_run(shll, p, calls, resident=True)
    assert lb == (3 if order == 1 else 2) * len(calls) and la > 20
    assert np.array_equal(a, b) and np.array_equal(ta, tb)


@pytest.mark.parametrize("order,n", [(1, 514), (1, 560), (1, 576), (1, 578), (1, 700), (1, 890), (2, 512), (2, 514), (2, 700), (2, 830)])
def test_batches_with_windows_between(shll, order, n):
    """Two chunks per tube and just more of them than half the SMs: windows of 289 to 479 cells, which no single tube has."""
    tubes = sm_count() // 4 + 2
    items = [shll.params(1, order, nx=n, precision="mixed_f64", fold_steps=64, n_steps=150, cfl=0.25 if n % 4 else 0.2,
                         ic_rho_l=3.0 + 0.1 * t, ic_x_d=0.3 + 0.01 * t) for t in range(tubes)]
    a, ta, la = _batch_run(shll, items, resident=False)
    b, tb, lb = _batch_run(shll, items, resident=True)
    assert lb <= 3 and la > lb
    assert all(np.array_equal(x, y) for x, y in zip(a, b)) and np.array_equal(ta, tb)
