"""Plain 2D domains with more tile rows than a grid's y axis holds (65535; 6-row tiles from 393211 cells
along x, 8-row ones from 524281): fused and staged steps against the CPU oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("f32_exact", 1, 393211, 2), ("f32_exact", 1, 400000, 16), ("f32_exact", 2, 524281, 3), ("f64_exact", 1, 1400000, 2)]


@pytest.mark.parametrize("prec,order,nx,ny", CASES)
def test_tall_domains(shll, oracle, prec, order, nx, ny):
    bits = 32 if prec == "f32_exact" else 64
    prim = oracle.ic_quadrants2d(nx, ny, bits)
    cfg = oracle.make_cfg(dim=2, order=order, nx=nx, ny=ny, real_bits=bits, ly=ny / nx, n_steps=2)
    _, ref, cons = oracle.run(cfg, prim)
    ctx = shll.Context(shll.params(2, order, nx=nx, ny=ny, precision=prec, ly=ny / nx, n_steps=2,
                                   ic_kind=shll.IC_QUADRANTS2D))
    ctx.init_state()
    ctx.run()
    assert np.array_equal(ctx.conserved(), cons) and np.array_equal(ctx.primitives(), ref)
    ctx.init_state()
    for _ in range(2):
        ctx.compute_F_from_P()
        ctx.update_U_from_F()
        ctx.compute_P_from_U()
    assert np.array_equal(ctx.conserved(), cons) and np.array_equal(ctx.primitives(), ref)
    ctx.close()
