"""The reference's separate stages in 2D on domains of several tiles: Compute_F_from_P, Update_U_from_F and
Compute_P_from_U against the CPU oracle's steps, bit for bit, and the fused steps likewise: tiles cut in either
direction, both limiters, grid constants that are and are not powers of two, and transverse momenta so small
that the products of their slopes underflow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one tile; cut and whole tiles in both directions; a single cell past a tile column (33, 65) and past rows of 6, 8
# and 14 (9 x 7, 65, 29)
SIZES = [(5, 3), (9, 33), (65, 64), (29, 65), (130, 101), (63, 257)]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("order,limiter", [(1, 0), (2, 0), (2, 1)])
@pytest.mark.parametrize("prec", ["f64_exact", "f32_exact"])
@pytest.mark.parametrize("cfl,tiny", [(0.25, False), (0.2, False), (0.25, True)])
def test_stages_and_fused_steps(shll, oracle, prec, order, limiter, nx, ny, cfl, tiny):
    bits, steps = 32 if prec == "f32_exact" else 64, 3
    rng = np.random.default_rng(nx * ny)
    prim = np.stack([1 + rng.uniform(size=nx * ny), 0.3 * rng.normal(size=nx * ny), 0.3 * rng.normal(size=nx * ny),
                     1 + rng.uniform(size=nx * ny)])
    if tiny:   # (the product of two slopes near or below the smallest subnormal; all else is the same along y)
        for q in (0, 1, 3):
            prim[q] = np.repeat(prim[q].reshape(nx, ny)[:, 0], ny)
        prim[2] = rng.normal(size=nx * ny) * 10.0 ** rng.uniform(-21 if bits == 32 else -165, -20 if bits == 32 else -150, nx * ny)
    kw = dict(limiter=limiter, cfl=cfl, n_steps=steps, ly=ny / nx)
    _, ref, cons = oracle.run(oracle.make_cfg(dim=2, order=order, nx=nx, ny=ny, real_bits=bits, **kw), prim)
    ctx = shll.Context(shll.params(2, order, nx=nx, ny=ny, precision=prec, ic_kind=shll.IC_QUADRANTS2D, **kw))
    for staged in (True, False):
        ctx.set_primitives(prim[0], prim[1], prim[3], v=prim[2])
        if staged:
            for _ in range(steps):
                ctx.compute_F_from_P()
                ctx.update_U_from_F()
                ctx.compute_P_from_U()
        else:
            ctx.run()
        assert np.array_equal(ctx.conserved(), cons) and np.array_equal(ctx.primitives(), ref), staged
    ctx.close()
