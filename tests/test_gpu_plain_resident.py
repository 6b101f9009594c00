"""1D runs of the plain arithmetic with several steps per launch: bit for bit the CPU oracle (exact
modes), within 1e-10 of it in FP64 with fused multiply-add (the bar of that mode), at the edges of
the chunking: fewer cells than SMs, uneven chunks, windows that reach over many chunks, the last
short sweep, and tubes too long to be resident."""
import time

import numpy as np
import pytest

from helpers import max_rel_scaled

pytestmark = pytest.mark.gpu

# cells and steps: 2 and 3 cells; one cell per chunk or fewer; uneven chunks; several sweeps and a
# short last one; one block per SM with wide windows; more cells than resident windows hold
SIZES = [(2, 70), (3, 200), (151, 130), (153, 131), (311, 2), (311, 3), (2000, 257), (9001, 101), (65536, 90),
         (80001, 21)]


@pytest.mark.parametrize("n,steps", SIZES)
@pytest.mark.parametrize("order,limiter", [(1, 0), (2, 0), (2, 1)])
@pytest.mark.parametrize("prec", ["f64_exact", "f32_exact", "f64"])
def test_matches_oracle(shll, oracle, prec, order, limiter, n, steps):
    bits = 32 if prec == "f32_exact" else 64
    kw = dict(limiter=limiter, cfl=0.25 if n % 2 == 0 else 0.2, n_steps=steps)   # (a factor that is no power of two)
    cfg = oracle.make_cfg(dim=1, order=order, nx=n, real_bits=bits, **kw)
    _, ref, cons = oracle.run(cfg, oracle.ic_sod(n))
    ctx = shll.Context(shll.params(1, order, nx=n, precision=prec, **kw))
    ctx.init_state()
    assert ctx.run() == steps
    out, got = ctx.primitives(), ctx.conserved()
    ctx.close()
    if prec == "f64":
        assert max_rel_scaled(out, ref) <= 1e-10
    else:
        assert np.array_equal(out, ref) and np.array_equal(got, cons)


@pytest.mark.parametrize("prec", ["f64_exact", "f32_exact"])
def test_any_split_of_a_run_is_the_same(shll, prec):
    """Runs split into 1, 2, 5 and many steps end in the same bits (buffers change hands per sweep)."""
    outs = []
    for parts in ([400], [1, 2, 5, 392], [133, 134, 133], [1] * 7 + [393]):
        ctx = shll.Context(shll.params(1, 2, nx=1237, precision=prec))
        ctx.init_state()
        for s in parts:
            ctx.step(s)
        assert ctx.steps_taken == 400
        outs.append((ctx.primitives(), ctx.conserved()))
        ctx.close()
    for o in outs[1:]:
        assert np.array_equal(o[0], outs[0][0]) and np.array_equal(o[1], outs[0][1])


def test_wait_runs_out_and_is_reported(shll, oracle):
    """A chunk that never publishes its progress (host-side hook): the others' bounded waits end the run
    with SHLL_ERR_TIMEOUT, and the next run on the device is right."""
    n, steps = 1024, 300
    cfg = oracle.make_cfg(dim=1, order=1, nx=n, n_steps=steps)
    _, ref, _ = oracle.run(cfg, oracle.ic_sod(n))
    p = shll.params(1, 1, nx=n, precision="f64_exact", n_steps=steps)
    shll.debug_stall_chunk(3)
    try:
        ctx = shll.Context(p)
        ctx.init_state()
        t0 = time.time()
        with pytest.raises(shll.ShllError) as e:
            ctx.run()
        assert e.value.status == shll.ERR_TIMEOUT and time.time() - t0 < 10
    finally:
        shll.debug_stall_chunk(-1)
    ctx.close()
    ctx = shll.Context(p)
    ctx.init_state()
    ctx.run()
    assert np.array_equal(ctx.primitives(), ref)
    ctx.close()
