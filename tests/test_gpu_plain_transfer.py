"""Host <-> device transfers of the plain contexts: primitives handed over replace the state as main() forms it
(base_shll.c:202-205) or, refused, leave it; handed back they are the state's; and neither needs device memory
beside the state.  Sizes below and above the largest with staging planes of their own (float), and an odd
number of steps before, which leaves the state in the other buffer."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [("f64_exact", 1, 3000, 1), ("f64_exact", 2, 96, 80), ("f32_exact", 1, 3000, 1), ("f32_exact", 2, 96, 80),
         ("f32_exact", 1, 700003, 1), ("f32_exact", 2, 801, 797), ("f64", 2, 401, 397)]


def make(shll, prec, dim, nx, ny, **kw):
    if dim == 2:
        kw.update(ny=ny, ic_kind=shll.IC_QUADRANTS2D)
    return shll.Context(shll.params(dim, 1, nx=nx, precision=prec, **kw))


def primitives(oracle, prec, dim, nx, ny):
    rng = np.random.default_rng(nx)
    if dim == 1:
        prim = oracle.ic_sod(nx)
    else:
        prim = oracle.ic_quadrants2d(nx, ny, 32 if prec == "f32_exact" else 64)
    return prim * (1 + 0.01 * rng.uniform(size=prim.shape))


def hand_over(ctx, prim):
    if prim.shape[0] == 3:
        ctx.set_primitives(prim[0], prim[1], prim[2])
    else:
        ctx.set_primitives(prim[0], prim[1], prim[3], v=prim[2])


@pytest.mark.parametrize("prec,dim,nx,ny", SIZES)
def test_handed_over_state_runs_as_the_oracle(shll, oracle, prec, dim, nx, ny):
    bits = 32 if prec == "f32_exact" else 64
    prim = primitives(oracle, prec, dim, nx, ny)
    ctx = make(shll, prec, dim, nx, ny, n_steps=5)
    ctx.init_state()
    ctx.step(3)
    hand_over(ctx, prim)
    assert ctx.steps_taken == 0
    cfg = dict(dim=dim, order=1, nx=nx, real_bits=bits, n_steps=5)
    if dim == 2:
        cfg.update(ny=ny)
    _, ref, cons = oracle.run(oracle.make_cfg(**cfg), prim)
    ctx.run()
    out, got = ctx.primitives(), ctx.conserved()
    again = ctx.primitives()
    ctx.close()
    assert np.array_equal(out, again)
    if prec == "f64":
        assert np.max(np.abs(out - ref)) <= 1e-10 * np.max(np.abs(ref))
    else:
        assert np.array_equal(out, ref) and np.array_equal(got, cons)


@pytest.mark.parametrize("prec,dim,nx,ny", SIZES)
def test_refused_state_leaves_the_one_that_is_there(shll, oracle, prec, dim, nx, ny):
    n = nx * ny
    ctx = make(shll, prec, dim, nx, ny, n_steps=8)
    ctx.init_state()
    ctx.step(3)
    before, cons = ctx.primitives(), ctx.conserved()
    good = primitives(oracle, prec, dim, nx, ny)
    for plane, cell, value in ((0, n - 1, 0.0), (good.shape[0] - 1, n // 2, -1.0), (0, n // 3, np.nan)):
        bad = good.copy()
        bad[plane, cell] = value
        bad[good.shape[0] - 1, n - 1] = -0.0
        with pytest.raises(shll.ShllError) as e:
            hand_over(ctx, bad)
        assert e.value.status == shll.ERR_ARG and f"cell {cell}:" in str(e.value)
        assert ctx.steps_taken == 3
        assert np.array_equal(ctx.primitives(), before) and np.array_equal(ctx.conserved(), cons)
    ctx.run()
    out = ctx.primitives()
    ctx.close()
    ctx = make(shll, prec, dim, nx, ny, n_steps=8)
    ctx.init_state()
    ctx.run()
    assert np.array_equal(out, ctx.primitives())
    ctx.close()


@pytest.mark.parametrize("prec", ["f64_exact", "f32_exact"])
@pytest.mark.parametrize("dim,nx,ny", [(1, 40, 1), (1, 9000, 1), (2, 30, 20), (2, 120, 90)])
def test_planes_apart_and_adjoining(shll, oracle, prec, dim, nx, ny):
    """Planes in one buffer (a single copy), in separate ones, and some left out when handed back."""
    prim = primitives(oracle, prec, dim, nx, ny)
    ctx = make(shll, prec, dim, nx, ny)
    hand_over(ctx, prim)
    whole = ctx.primitives()
    apart = [p.copy() for p in prim]
    if dim == 1:
        ctx.set_primitives(apart[0], apart[1], apart[2])
    else:
        ctx.set_primitives(apart[0], apart[1], apart[3], v=apart[2])
    assert np.array_equal(ctx.primitives(), whole)
    for left_out in range(-1, dim + 2):
        out = [np.full(nx * ny, -7.0) for _ in prim]
        ptr = [None if k == left_out else o.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for k, o in enumerate(out)]
        args = ptr if dim == 2 else [ptr[0], ptr[1], None, ptr[2]]
        assert shll.lib().shll_get_primitives(ctx.h, *args) == shll.OK
        for k, o in enumerate(out):
            assert np.all(o == -7.0) if k == left_out else np.array_equal(o, whole[k])
    ctx.close()


@pytest.mark.parametrize("prec,dim,nx,ny", [("f64_exact", 2, 1400, 1400), ("f32_exact", 2, 1400, 1400), ("f32_exact", 1, 2700000, 1)])
def test_device_memory_is_the_state(shll, oracle, prec, dim, nx, ny):
    torch = pytest.importorskip("torch")
    nv, real = (3, 4)[dim - 1], 4 if prec == "f32_exact" else 8
    make(shll, prec, dim, 64, 64).close()   # (the device's context and the modules)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx = make(shll, prec, dim, nx, ny)
    hand_over(ctx, primitives(oracle, prec, dim, nx, ny))
    ctx.primitives()
    used = free - torch.cuda.mem_get_info()[0]
    ctx.close()
    state = nx * ny * real * (3 * nv + 1)   # two state buffers, primitives and sound speed
    assert used <= state + (8 << 20)
