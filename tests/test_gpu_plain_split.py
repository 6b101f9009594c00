"""Fused FP64 runs of 1D tubes: any split of a run into calls ends in the same bits.  Single steps, short
calls and long ones take kernels and windows of their own (one or four threads per cell by the tube's size)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma,R,cfl", [(1.4, 1.0, 0.25), (1.3, 0.9, 0.2)])
@pytest.mark.parametrize("n,order,limiter", [(3, 1, 0), (300, 1, 0), (300, 2, 1), (1237, 2, 0), (3001, 1, 0), (9001, 2, 1)])
def test_any_split_of_a_fused_run_is_the_same(shll, n, order, limiter, gamma, R, cfl):
    outs = []
    for parts in ([400], [1] * 400, [1, 2, 5, 392], [3] * 133 + [1]):
        ctx = shll.Context(shll.params(1, order, nx=n, precision="f64", limiter=limiter, gamma=gamma, R=R, cfl=cfl))
        ctx.init_state()
        for s in parts:
            ctx.step(s)
        assert ctx.steps_taken == 400
        outs.append((ctx.primitives(), ctx.conserved()))
        ctx.close()
    for o in outs[1:]:
        assert np.array_equal(o[0], outs[0][0]) and np.array_equal(o[1], outs[0][1])
