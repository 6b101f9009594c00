"""Bit-exact modes against the CPU oracle where their integer division, square root and power-of-two
scaling (and the float mode's FP32 forms of double expressions) leave their main path: subnormal and
huge magnitudes, velocities that are zero or underflow when squared, factors that are no power of
two.  Bit for bit, so no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (density scale, temperature scale): ordinary, and products at both ends of the type's range
SCALES = {"f64_exact": [(1.0, 1.0), (1e-100, 1e-203), (1e120, 1e100), (3e-290, 2.0)],
          "f32_exact": [(1.0, 1.0), (1e-20, 1e-16), (1e14, 1e12), (1e-33, 2.0)]}


def field(rng, n, dim, rho, T):
    prim = np.zeros((2 + dim, n))
    prim[0] = rho * (1 + 0.2 * rng.uniform(-1, 1, n))
    prim[-1] = T * (1 + 0.2 * rng.uniform(-1, 1, n))
    for k in range(1, 1 + dim):
        u = 0.4 * np.sqrt(T) * rng.uniform(-1, 1, n)
        u[: n // 4] = 0.0
        u[n // 4: n // 3] *= 1e-25     # squares vanish beside the energy (and underflow at small scales)
        prim[k] = u
    return prim


@pytest.mark.parametrize("dim,order,limiter", [(1, 1, 0), (1, 2, 0), (1, 2, 1), (2, 1, 0), (2, 2, 0), (2, 2, 1)])
@pytest.mark.parametrize("gamma,R,cfl", [(1.4, 1.0, 0.25), (1.3, 0.9, 0.2)])
@pytest.mark.parametrize("prec", ["f64_exact", "f32_exact"])
def test_extreme_magnitudes_bitwise(shll, oracle, prec, gamma, R, cfl, dim, order, limiter):
    nx, ny = (301, 1) if dim == 1 else (21, 37)
    bits = 64 if prec == "f64_exact" else 32
    for q, (rho, T) in enumerate(SCALES[prec]):
        prim = field(np.random.default_rng(q), nx * ny, dim, rho, T)
        if bits == 32:
            prim = prim.astype(np.float32).astype(np.float64)
        # (a step short enough for the scale's velocities: the time step itself does not know them)
        step = cfl / max(1.0, np.sqrt(T)) if T <= 4 else cfl * 0.25 / np.sqrt(T)
        cfg = oracle.make_cfg(dim=dim, order=order, nx=nx, ny=ny, real_bits=bits, gamma=gamma, R=R, cfl=step,
                              limiter=limiter, n_steps=4)
        steps, ref, cons = oracle.run(cfg, prim)
        p = shll.params(dim, order, nx=nx, ny=ny, precision=prec, gamma=gamma, R=R, cfl=step, limiter=limiter,
                        n_steps=4, ic_kind=shll.IC_USER)
        ctx = shll.Context(p)
        ctx.set_primitives(prim[0], prim[1], prim[-1], v=prim[2] if dim == 2 else None)
        assert ctx.run() == steps == 4
        out, got = ctx.primitives(), ctx.conserved()
        ctx.close()
        assert np.array_equal(got, cons) and np.array_equal(out, ref), (rho, T, np.abs(out - ref).max())
