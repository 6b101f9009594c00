"""Plain contexts: restoring a checkpoint clears the error flags that a failed run raised, so that the same
context runs on from it (an expired wait in a 1D run; a run that ended in a non-positive temperature)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,order", [("f64_exact", 1), ("f32_exact", 2), ("f64", 1)])
def test_restore_after_an_expired_wait(shll, oracle, prec, order):
    n, steps = 1024, 300
    bits = 32 if prec == "f32_exact" else 64
    ctx = shll.Context(shll.params(1, order, nx=n, precision=prec, n_steps=steps))
    ctx.init_state()
    ctx.step(40)
    ctx.checkpoint()
    shll.debug_stall_chunk(3)
    try:
        with pytest.raises(shll.ShllError) as e:
            ctx.run()
        assert e.value.status == shll.ERR_TIMEOUT
    finally:
        shll.debug_stall_chunk(-1)
    ctx.restore()
    assert ctx.steps_taken == 40
    assert ctx.run() == steps
    got = ctx.primitives()
    ctx.close()
    if prec == "f64":
        ctx = shll.Context(shll.params(1, order, nx=n, precision=prec, n_steps=steps))
        ctx.init_state()
        ctx.run()
        ref = ctx.primitives()
        ctx.close()
    else:
        _, ref, _ = oracle.run(oracle.make_cfg(dim=1, order=order, nx=n, real_bits=bits, n_steps=steps), oracle.ic_sod(n))
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("dim", [1, 2])
def test_restore_after_a_breakdown(shll, dim):
    """A step far beyond the stable one makes a temperature negative; the state from before it is whole."""
    kw = dict(nx=200) if dim == 1 else dict(nx=40, ny=36, ic_kind=shll.IC_QUADRANTS2D)
    ctx = shll.Context(shll.params(dim, 1, precision="f64_exact", cfl=40.0, n_steps=60, **kw))
    ctx.init_state()
    before = ctx.primitives()
    ctx.checkpoint()
    with pytest.raises(shll.ShllError) as e:
        ctx.run()
    assert e.value.status == shll.ERR_NUMERIC
    ctx.restore()
    assert np.array_equal(ctx.primitives(), before)
    ctx.compute_P_from_U()
    ctx.close()
