"""The workloads that the solver's speed is judged on, each one whole run through the public API.

A pass is what a user's program does with a problem: hand the initial primitives over from (pinned)
host memory, run the time loop, and take the final primitives back into (pinned) host memory.  A
context or batch, with its device memory, is created once per problem and kept, as such a program
keeps it.  Everything is at the library's defaults: no tuning runs, no switches.

The initial data are Riemann problems of the sizes and strengths that the repository's own
configurations, tests and benchmark use (gamma 1.4, R 1, kinetic CFL 0.25 throughout), drawn from
the seed, as strong as the scheme itself stays positive on at every size here: in 1D density ratios
of 2 to 50 for first-order tubes of the mixed engine, else 2 to 10 (on much stronger tubes the
reference's second order breaks down); in 2D 2 to 20 (box) or 2 to 50 (circle), and the reference's
four shocks and quadrants with their states varied by up to a per cent.

Families ("kind" of a case):
  tube     one 1D shock tube (order 1: reflective walls, order 2: limited slopes, outflow walls)
  plane    one 2D domain: "box" and "circle" (first order), "shocks" and "quadrants" (second order)
  stages   the reference's separate stage calls, one step of the time loop after another
  tubes    a batch of independent tubes of uneven sizes, half first order, half second order
  planes   a batch of independent first-order 2D domains of uneven sizes
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GAMMA, R, CFL = 1.4, 1.0, 0.25
CV = R / (GAMMA - 1.0)
MC_ALPHA = 1.25
T_END = {"tube": 0.2, "box": 0.1, "circle": 0.1, "shocks": 0.8, "quadrants": 0.3}


def _api():
    name = "shll_gb300"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(ROOT, "shll-sve-cfd_gb300", name + ".py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def listed():
    return [
        # the default problem of base_shll.c, in the library's default arithmetic: the smallest call,
        # 410 steps of a tube that fills two blocks
        {"name": "tube256_f64", "kind": "tube", "n": 256, "order": 1, "limiter": 0, "prec": "f64"},
        # the published program on 1024 cells, in its own float arithmetic (1639 steps)
        {"name": "tube1024_f32", "kind": "tube", "n": 1024, "order": 1, "limiter": 0, "prec": "f32_exact"},
        # the bit-exact FP64 oracle of a second-order tube, an odd size (4802 steps)
        {"name": "tube3001_f64_exact_o2", "kind": "tube", "n": 3001, "order": 2, "limiter": 0, "prec": "f64_exact"},
        # base_shll_2d.c's default problem (205 steps) in FP64
        {"name": "box256_f64", "kind": "plane", "ic": "box", "nx": 256, "ny": 256, "order": 1, "limiter": 0,
         "prec": "f64", "steps": 0},
        # 2nd_order_base_shll.c's four-shock problem in the published float arithmetic, ragged sides
        {"name": "shocks301x277_f32", "kind": "plane", "ic": "shocks", "nx": 301, "ny": 277, "order": 2, "limiter": 0,
         "prec": "f32_exact", "steps": 600},
        # a program that calls the reference's stages one by one (flux, update, primitives), FP64
        {"name": "stages512x480_f64", "kind": "stages", "ic": "quadrants", "nx": 512, "ny": 480, "order": 2, "limiter": 0,
         "prec": "f64", "steps": 40},
        # one long second-order tube on the mixed engine, the whole run (104858 steps)
        {"name": "tube65536_mixed_o2", "kind": "tube", "n": 65536, "order": 2, "limiter": 0, "prec": "mixed_f64"},
        # a first-order tube of odd size in the compensated FP32 state format (16012 steps)
        {"name": "tube10007_kahan", "kind": "tube", "n": 10007, "order": 1, "limiter": 0, "prec": "mixed_kahan"},
        # an ensemble of tubes of uneven sizes, each to its own end
        {"name": "tubes512_mixed", "kind": "tubes", "count": 512, "nmin": 256, "nmax": 16384, "prec": "mixed_f64"},
        # the circular diaphragm on the largest grid
        {"name": "circle4096_mixed", "kind": "plane", "ic": "circle", "nx": 4096, "ny": 4096, "order": 1, "limiter": 0,
         "prec": "mixed_f64", "steps": 500},
        # an ensemble of square domains of 128 to 1024 cells a side
        {"name": "planes24_mixed", "kind": "planes", "count": 24, "smin": 128, "smax": 1024, "odd": False,
         "prec": "mixed_f64", "steps": 400},
        # base-omp's quadrant problem: second order, MC limiter, 1024 x 1024
        {"name": "quadrants1024_mixed", "kind": "plane", "ic": "quadrants", "nx": 1024, "ny": 1024, "order": 2,
         "limiter": 1, "prec": "mixed_f64", "steps": 800},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["tube", "tube", "tube", "plane", "plane", "plane", "stages", "tubes", "planes"])
    if kind == "tube":
        prec = rng.choice(["f64", "f64_exact", "f32_exact", "mixed_f64", "mixed_f64", "mixed_kahan"])
        order = rng.choice([1, 2])
        n = log(256, 65536) if prec.startswith("mixed") else log(128, 8192)
        return {"kind": kind, "n": n, "order": order, "limiter": rng.choice([0, 1]) if order == 2 else 0, "prec": prec}
    if kind in ("plane", "stages"):
        mixed = kind == "plane" and rng.random() < 0.6
        prec = rng.choice(["mixed_f64", "mixed_f64", "mixed_kahan"]) if mixed else rng.choice(["f64", "f64_exact", "f32_exact"])
        order = rng.choice([1, 2])
        ic = rng.choice(["box", "circle"] if order == 1 else ["shocks", "quadrants", "quadrants"])
        top = 320 if ic == "shocks" else 3000 if mixed else 700   # (larger four-shock runs can break down)
        nx = log(64, top)
        # (one time step for both directions: DT follows from dx)
        ny = int(nx * (rng.uniform(0.9, 1.1) if ic == "shocks" else rng.uniform(0.5, 1.25)))
        steps = rng.randint(20, 60) if kind == "stages" else rng.randint(100, 400)
        return {"kind": kind, "ic": ic, "nx": nx, "ny": ny, "order": order,
                "limiter": rng.choice([0, 1]) if ic == "quadrants" else 0, "prec": prec, "steps": steps}
    if kind == "tubes":
        return {"kind": kind, "count": log(8, 400), "nmin": 256, "nmax": rng.choice([2048, 4096, 8192, 16384]),
                "prec": rng.choice(["mixed_f64", "mixed_kahan"])}
    return {"kind": kind, "count": rng.randint(4, 32), "smin": rng.choice([64, 128]), "smax": rng.choice([512, 1024]),
            "odd": rng.random() < 0.5, "prec": rng.choice(["mixed_f64", "mixed_kahan"]), "steps": rng.randint(100, 400)}


# ---- the problems of a case ----
def _items(case, seed):
    """The case's problems as dicts (nx, ny, order, limiter, initial-data parameters).  Sizes come from the
    case alone, the initial data from the seed."""
    rng = np.random.default_rng([int(seed), 77])
    size = random.Random(repr(sorted(case.items())))

    def tube(n, order, limiter, strong):
        return {"dim": 1, "nx": n, "ny": 1, "order": order, "limiter": limiter, "ic": "tube", "steps": 0,
                "ratio": rng.uniform(2, 50 if strong else 10), "temp": rng.uniform(0.5, 1.5 if strong else 1.0),
                "x_d": rng.uniform(0.3, 0.7)}

    def plane(nx, ny, order, limiter, ic, steps):
        return {"dim": 2, "nx": nx, "ny": ny, "order": order, "limiter": limiter, "ic": ic, "steps": steps,
                "ratio": rng.uniform(2, 20 if ic == "box" else 50), "temp": rng.uniform(0.5, 2.0),
                "radius": rng.uniform(0.1, 0.35), "vary": 1.0 + 0.01 * rng.uniform(-1, 1, 16)}

    if case["kind"] == "tube":
        return [tube(case["n"], case["order"], case["limiter"], case["order"] == 1 and case["prec"].startswith("mixed"))]
    if case["kind"] in ("plane", "stages"):
        return [plane(case["nx"], case["ny"], case["order"], case["limiter"], case["ic"], case["steps"])]
    if case["kind"] == "tubes":
        got = []
        for t in range(case["count"]):
            n = int(round(math.exp(size.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
            order = 1 if t < case["count"] // 2 else 2
            got.append(tube(n, order, 0, order == 1))
        return got
    sides = []
    for _ in range(case["count"]):
        if case["odd"]:
            n = int(round(math.exp(size.uniform(math.log(case["smin"]), math.log(case["smax"])))))
            sides.append([n, int(n * size.uniform(0.5, 1.25))])
        else:
            sides.append([case["smin"] << size.randint(0, (case["smax"] // case["smin"]).bit_length() - 1)] * 2)
    return [plane(nx, ny, 1, 0, "circle", case["steps"]) for nx, ny in sides]


def _initial(item, dev):
    """(nv, n) FP64 primitives rho, u, [v,] T of an item."""
    f = dict(dtype=torch.float64, device=dev)
    nx, ny = item["nx"], item["ny"]
    if item["dim"] == 1:
        left = torch.arange(nx, **f) < item["x_d"] * nx
        rho = torch.where(left, item["ratio"], 1.0).to(torch.float64)
        T = torch.where(left, item["temp"], 1.0).to(torch.float64)
        return torch.stack([rho, torch.zeros_like(rho), T])
    i, j = torch.arange(nx, **f)[:, None], torch.arange(ny, **f)[None, :]
    w = item["vary"]
    out = torch.zeros(4, nx, ny, **f)
    if item["ic"] == "box":
        inside = (i > 0.2 * nx) & (i < 0.8 * nx) & (j > 0.2 * ny) & (j < 0.8 * ny)
        out[0] = torch.where(inside, 1.0, item["ratio"])
        out[3] = 1.0
    elif item["ic"] == "circle":
        x, y = (i + 0.5) / nx - 0.5, (j + 0.5) / ny - 0.5
        inside = x * x + y * y < item["radius"] ** 2
        out[0] = torch.where(inside, item["ratio"], 1.0)
        out[3] = torch.where(inside, item["temp"], 1.0)
    else:
        h = 0.75 if item["ic"] == "shocks" else 0.5
        if item["ic"] == "shocks":   # rho, u, v, p
            q = [(0.138, 1.206, 1.206, 0.029), (0.5323, 0.0, 1.206, 0.3), (0.5323, 1.206, 0.0, 0.3), (1.5, 0.0, 0.0, 1.5)]
        else:
            q = [(1.0, -0.75, 0.5, 1.0), (3.0, -0.75, -0.5, 1.0), (2.0, 0.75, 0.5, 1.0), (1.0, 0.75, -0.5, 1.0)]
        lo_i, lo_j = i < h * nx, j < h * ny
        for k, where in enumerate([lo_i & lo_j, ~lo_i & lo_j, lo_i & ~lo_j, ~lo_i & ~lo_j]):
            rho, u, v, p = (x * w[4 * k + c] for c, x in enumerate(q[k]))
            for c, x in enumerate((rho, u, v, p / (rho * R))):
                out[c] = torch.where(where, x, out[c])
    return out.reshape(4, nx * ny)


def _steps(item, prec):
    """Steps of the time loop (its clock is a float in the published arithmetic)."""
    if item["steps"]:
        return item["steps"]
    real = np.float32 if prec == "f32_exact" else np.float64
    dt = (real(CFL) / (real(R) + real(1))) * (real(1.0) / real(item["nx"]))
    end, time, steps = real(T_END[item["ic"]]), real(0), 0
    while time < end:
        time = time + dt
        steps += 1
    return steps


def _host(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=t.is_cuda)
    p.copy_(t)
    return p


def _params(api, case, item):
    p = api.params(dim=item["dim"], order=item["order"], nx=item["nx"], ny=item["ny"], precision=case["prec"])
    p.t_end, p.n_steps, p.limiter = T_END[item["ic"]], item["steps"], item["limiter"]
    return p


# ---- what is timed ----
def prepare(case, seed):
    api = _api()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    items = _items(case, seed)
    init = [_initial(it, dev) for it in items]
    s = {"kind": case["kind"], "steps": case.get("steps", 0)}
    if case["kind"] in ("tubes", "planes"):
        params = []
        for it in items:
            p = _params(api, case, it)
            if it["dim"] == 1:
                p.ic.kind, p.ic.x_d, p.ic.rho_l, p.ic.T_l = api.IC_SOD, it["x_d"], it["ratio"], it["temp"]
            else:
                p.ic.kind, p.ic.cx, p.ic.cy, p.ic.radius = api.IC_CIRCLE2D, 0.5, 0.5, it["radius"]
                p.ic.rho_l, p.ic.T_l = it["ratio"], it["temp"]
            p.ic.rho_r, p.ic.T_r = 1.0, 1.0
            params.append(p)
        s["in"] = _host(torch.cat([x.reshape(-1) for x in init]))
        s["ctx"] = api.Batch(params)
    else:
        p = _params(api, case, items[0])
        p.ic.kind = api.IC_USER
        s["in"] = _host(init[0])
        s["ctx"] = api.Context(p)
    s["out"] = _host(torch.zeros_like(s["in"], device=dev))
    return s


def run(s):
    ctx, a, out = s["ctx"], s["in"].numpy(), s["out"].numpy()
    if s["kind"] in ("tubes", "planes"):
        ctx.set_all_primitives(a)
        ctx.run()
        return ctx.get_all_primitives(out)
    if len(a) == 4:
        ctx.set_primitives(a[0], a[1], a[3], v=a[2])
    else:
        ctx.set_primitives(a[0], a[1], a[2])
    if s["kind"] == "stages":
        for _ in range(s["steps"]):
            ctx.compute_F_from_P()
            ctx.update_U_from_F()
            ctx.compute_P_from_U()
    else:
        ctx.run()
    return ctx.primitives(out)


def work(case):
    """Initial primitives read and final ones written once; the scheme's arithmetic per cell and step (a divide
    or a square root as one operation): primitives, split fluxes, [slopes,] interface sums and update."""
    cells = flops = 0
    for it in _items(case, 0):
        n = it["nx"] * it["ny"]
        nv = 3 if it["dim"] == 1 else 4
        per = {(1, 1): 56, (1, 2): 98, (2, 1): 134, (2, 2): 246}[it["dim"], it["order"]]
        cells += nv * n
        flops += per * n * _steps(it, case["prec"])
    return {"bytes": 16.0 * cells, "flops": float(flops)}


# ---- the same in 64 bits, in plain torch ----
def _minmod(a, b):
    return torch.where(a * b < 0.0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _sweep(F, U, u, a, normal, order, limiter, dim, first, last):
    """Difference of the interface fluxes, F_{j+1/2} - F_{j-1/2}, along `dim`; first, last: indexes of the wall
    cells along it (several where tubes lie end to end)."""
    M = u / a
    Z2 = 0.5 * a * (1.0 - M * M)
    p = F * (0.5 * (M + 1.0)) + U * Z2
    m = F - p
    if order == 2:
        def half(f):
            d = torch.diff(f, dim=dim)
            l, r = d.narrow(dim, 0, d.shape[dim] - 1), d.narrow(dim, 1, d.shape[dim] - 1)
            s = torch.zeros_like(f)
            s.narrow(dim, 1, f.shape[dim] - 2).copy_(_minmod(0.5 * (l + r), MC_ALPHA * _minmod(l, r)) if limiter else _minmod(l, r))
            s.index_fill_(dim, first, 0.0).index_fill_(dim, last, 0.0)
            return 0.5 * s
        L, Rt = p + half(p), m - half(m)
    else:
        L, Rt = p, m
    n = F.shape[dim]
    face = torch.zeros_like(F)      # face j: between cells j - 1 and j
    face.narrow(dim, 1, n - 1).copy_(L.narrow(dim, 0, n - 1) + Rt.narrow(dim, 1, n - 1))
    right = torch.roll(face, -1, dim)
    pw, mw = p.index_select(dim, last), m.index_select(dim, first)
    if order == 2:
        wl, wr = p.index_select(dim, first) + mw, pw + m.index_select(dim, last)
    else:                           # reflective walls: only the normal momentum's flux is left
        keep = torch.zeros(F.shape[0], *([1] * (F.dim() - 1)), dtype=F.dtype, device=F.device)
        keep[normal] = 2.0
        wl, wr = mw * keep, pw * keep
    return right.index_copy_(dim, last, wr) - face.index_copy_(dim, first, wl)


def _advance(U, dim, order, limiter, lam, steps, first, last):
    for _ in range(steps):
        rho, E = U[0], U[-1]
        u = U[1] / rho
        if dim == 1:
            T = (E / rho - 0.5 * u * u) / CV
        else:
            v = U[2] / rho
            T = (E / rho - 0.5 * (u * u + v * v)) / CV
        a, P = torch.sqrt(GAMMA * R * T), rho * R * T
        F = U * u
        F[1] += P
        F[-1] += u * P
        d = lam[0] * _sweep(F, U, u, a, 1, order, limiter, 1, first[0], last[0])
        if dim == 2:
            F = U * v
            F[2] += P
            F[-1] += v * P
            d += lam[1] * _sweep(F, U, v, a, 2, order, limiter, 2, first[1], last[1])
        U = U - d
    return U


def exact(case, seed):
    items = _items(case, seed)
    steps = [_steps(it, case["prec"]) for it in items]
    per = 60e-6 + 35e-6 * (items[0]["dim"] == 2)
    cells = sum(it["nx"] * it["ny"] * s for it, s in zip(items, steps))
    # (small operations are bound by their launches, large ones by memory and the FP64 rate)
    if max(steps) * per * 8 + cells * 9e-10 * items[0]["dim"] > 18.0:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = [None] * len(items)
    if items[0]["dim"] == 2:
        for t, it in enumerate(items):
            W = _initial(it, dev).reshape(4, it["nx"], it["ny"])
            U = torch.stack([W[0], W[0] * W[1], W[0] * W[2], W[0] * (CV * W[3] + 0.5 * (W[1] ** 2 + W[2] ** 2))])
            lam = (CFL / (R + 1), CFL / (R + 1) * it["ny"] / it["nx"])
            ends = [torch.tensor([e], device=dev) for e in (0, it["nx"] - 1, it["ny"] - 1)]
            U = _advance(U, 2, it["order"], it["limiter"], lam, steps[t], (ends[0], ends[0]), (ends[1], ends[2]))
            u, v = U[1] / U[0], U[2] / U[0]
            out[t] = torch.stack([U[0], u, v, (U[3] / U[0] - 0.5 * (u * u + v * v)) / CV]).reshape(4, -1)
    else:
        for order in (1, 2):      # tubes end to end, the finished ones taken out as the steps go
            live = sorted((t for t, it in enumerate(items) if it["order"] == order), key=lambda t: steps[t])
            W = {t: _initial(items[t], dev) for t in live}
            U = {t: torch.stack([w[0], w[0] * w[1], w[0] * (CV * w[2] + 0.5 * w[1] ** 2)]) for t, w in W.items()}
            done = 0
            while live:
                flat = torch.cat([U[t] for t in live], 1)
                n = torch.tensor([items[t]["nx"] for t in live])
                last = torch.cumsum(n, 0) - 1
                first = last - n + 1
                flat = _advance(flat, 1, order, items[live[0]]["limiter"], (CFL / (R + 1),), steps[live[0]] - done,
                                (first.to(dev),), (last.to(dev),))
                done = steps[live[0]]
                for t, x in zip(live, torch.split(flat, n.tolist(), 1)):
                    U[t] = x
                live = [t for t in live if steps[t] > done]
            for t, x in U.items():
                u = x[1] / x[0]
                out[t] = torch.stack([x[0], u, (x[2] / x[0] - 0.5 * u * u) / CV])
    out = [x.cpu() for x in out]
    if case["kind"] in ("tubes", "planes"):
        return torch.cat([x.reshape(-1) for x in out]).numpy()
    return out[0].numpy()
