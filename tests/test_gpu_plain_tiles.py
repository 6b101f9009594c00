"""Bit-exact 2D steps against the CPU oracle, bit for bit, at sizes that take different tile heights and
cut tiles in both directions (the tile height follows from the number of tiles and SMs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 65), (37, 33), (256, 256), (301, 277), (609, 31), (95, 700)]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("order,limiter", [(1, 0), (2, 0), (2, 1)])
@pytest.mark.parametrize("prec", ["f64_exact", "f32_exact"])
def test_tiles_match_oracle(shll, oracle, prec, order, limiter, nx, ny):
    bits = 64 if prec == "f64_exact" else 32
    steps = 7
    prim = oracle.ic_quadrants2d(nx, ny, bits)
    cfg = oracle.make_cfg(dim=2, order=order, nx=nx, ny=ny, real_bits=bits, limiter=limiter, ly=ny / nx, n_steps=steps)
    _, ref, cons = oracle.run(cfg, prim)
    ctx = shll.Context(shll.params(2, order, nx=nx, ny=ny, precision=prec, limiter=limiter, ly=ny / nx, n_steps=steps,
                                   ic_kind=shll.IC_QUADRANTS2D))
    ctx.init_state()
    assert ctx.run() == steps
    out, got = ctx.primitives(), ctx.conserved()
    ctx.close()
    assert np.array_equal(got, cons) and np.array_equal(out, ref)
