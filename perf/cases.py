"""Workloads of a vortex-blob program, through pfblob's public entry points.

Each case is one call, or one short chain of calls, that a blob or blob + panel
simulation makes every step (or every time a body moves): induced velocity by
FMM and by direct summation, induced vorticity, the M4' remesh with and without
diffusion and population control, panel velocity, the panel system, one stage
of the coupled step, many small simulations per launch, and the step on host
arrays.  Blob sets have the core size sigma = h / 0.8 of their spacing h, as
pHyFlow's overlap ratio gives it, so the number of near-field partners of a
blob is the same at every size.

``exact`` restates every result in FP64 with plain torch operations.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "phyflow2.0_b200"))
import pfblob  # noqa: E402
from pfblob.batch import Batch  # noqa: E402

OVERLAP = 0.8
K = 2.0
EPS = 1e-12  # softening of the Gaussian kernel's r^2
PAIRS_EXACT = 1.2e11  # pairs a plain FP64 sum goes through in a few seconds
DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
def listed():
    return [
        # the first steps of a small study, or a probe of a few thousand blobs:
        # every kernel is short, so launches and host work are what it costs
        {"name": "velocity_few_blobs", "kind": "velocity", "layout": "uniform", "method": "fmm",
         "n": 3001, "tol": 1e-6},
        # pHyFlow's Lamb-Oseen example: 100 x 100 blobs, direct summation
        {"name": "velocity_direct_lattice", "kind": "velocity", "layout": "lattice",
         "method": "direct", "n": 10000, "tol": 1e-6},
        # the throughput configuration: a million blobs in the unit square
        {"name": "velocity_million", "kind": "velocity", "layout": "uniform", "method": "fmm",
         "n": 1 << 20, "tol": 1e-6},
        # a shear layer around a body: an annulus, most of the tree is empty
        {"name": "velocity_near_wall", "kind": "velocity", "layout": "wall", "method": "fmm",
         "n": 1803001, "tol": 1e-6},
        # vorticity of a remeshed set at its own blobs (diagnostics, restart of
        # a field from blobs)
        {"name": "vorticity_lattice", "kind": "vorticity", "n": 40401},
        # redistribution of blobs that have lost their lattice order
        {"name": "regrid_million", "kind": "regrid", "layout": "uniform", "n": 1 << 20, "c": 0.0,
         "control": False},
        # the end of a viscous step: diffusion in the remesh weights and
        # population control, on a lattice that one convection step has moved
        {"name": "remesh_diffuse_control", "kind": "regrid", "layout": "patch", "n": 700569,
         "c": 0.3, "control": True},
        # panels of a body acting on the blobs of the layer around it
        {"name": "panels_near_wall", "kind": "panels", "m": 512, "n": 1500007},
        # a body has moved: influence matrix, factorisation, strengths
        {"name": "panel_system", "kind": "system", "m": 512},
        # one stage of the coupled step: blob velocity at the collocation
        # points, panel strengths, velocity of blobs, panels and free stream
        {"name": "coupled_stage", "kind": "coupled", "m": 200, "n": 60007},
        # a sweep of independent simulations of uneven sizes in one launch
        {"name": "batch_sweep", "kind": "batch", "sets": 12, "lo": 2048, "hi": 131072},
        # a step of a program that keeps its blobs in numpy, as pHyFlow's do
        {"name": "step_from_host", "kind": "host", "n": 200003},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["velocity", "velocity", "velocity", "direct", "vorticity", "regrid",
                       "regrid", "control", "panels", "system", "coupled", "batch", "host"])
    tol = rng.choice([1e-6, 1e-6, 1e-8])
    if kind == "velocity":
        layout = rng.choice(["uniform", "wall", "lattice"])
        return {"kind": "velocity", "layout": layout, "method": "fmm", "tol": tol,
                "n": log(2048, 1 << 20)}
    if kind == "direct":
        return {"kind": "velocity", "layout": rng.choice(["uniform", "lattice", "lattice"]),
                "method": "direct", "tol": 1e-6, "n": log(500, 65536)}
    if kind == "vorticity":
        return {"kind": "vorticity", "n": log(1000, 90000)}
    if kind == "regrid":
        return {"kind": "regrid", "layout": rng.choice(["uniform", "uniform", "lattice"]),
                "n": log(3000, 1 << 20), "c": rng.choice([0.0, 0.0, 0.4]), "control": False}
    if kind == "control":
        return {"kind": "regrid", "layout": "patch", "n": log(3000, 1 << 20),
                "c": rng.choice([0.0, 0.3, 0.5]), "control": True}
    if kind == "panels":
        return {"kind": "panels", "m": log(60, 800), "n": log(2000, 1500000)}
    if kind == "system":
        return {"kind": "system", "m": log(60, 900)}
    if kind == "coupled":
        return {"kind": "coupled", "m": log(60, 400), "n": log(5000, 250000)}
    if kind == "batch":
        return {"kind": "batch", "sets": rng.randint(4, 12), "lo": 2048,
                "hi": log(20000, 131072)}
    return {"kind": "host", "n": log(3000, 400000)}


# ---------------------------------------------------------------------------
# inputs (torch only, from the seed)
def _gen(seed, device=DEV):
    return torch.Generator(device=device).manual_seed(1009 * int(seed) + 17)


def _rand(n, gen):
    return torch.rand(n, dtype=torch.float64, device=gen.device, generator=gen)


def _blobs(layout, n, seed, device=DEV):
    """(x, y, g, h) of n blobs ('lattice', 'patch': the square number up to n)."""
    gen = _gen(seed, device)
    if layout == "uniform":  # positions without order, circulations of both signs
        h = 1.64 / math.sqrt(n)
        # a few of them hold the border of the unit square, so that the remesh
        # touches the same nodes whatever the others' positions are
        t = torch.linspace(1e-3 * h, 1.0 - 1e-3 * h, int(1.0 / h) + 2, dtype=torch.float64,
                           device=device)
        a, b = torch.full_like(t, float(t[0])), torch.full_like(t, float(t[-1]))
        m = n - 4 * t.numel()
        x = torch.cat([_rand(m, gen), t, t, a, b])
        y = torch.cat([_rand(m, gen), a, b, t, t])
        order = torch.argsort(_rand(n, gen))
        g = torch.randn(n, dtype=torch.float64, device=device, generator=gen) / n
        return x[order].contiguous(), y[order].contiguous(), g, h
    if layout in ("lattice", "patch"):
        # blobs of a remeshed set after one convection step: moved by a tenth
        # to four tenths of a cell
        s = math.isqrt(n)
        h = 2.0 / s
        c = -1.0 + (torch.arange(s, dtype=torch.float64, device=device) + 0.5) * h
        x, y = c.repeat_interleave(s), c.repeat(s)
        r2 = x * x + y * y
        u = _rand(3, gen).tolist()
        if layout == "lattice":  # a Lamb-Oseen vortex
            rc = 0.2 + 0.02 * u[0]
            g = torch.exp(-r2 / rc**2) / (math.pi * rc**2) * (h * h)
        else:  # a strong vortex patch; outside, the rounding left by earlier remeshes
            g = torch.where(r2 < 0.49, (1.0 + u[0]) * 1e4 * (1.2 - r2) * (h * h),
                            1e-19 * torch.randn(s * s, dtype=torch.float64, device=device,
                                                generator=gen))
        turn = 0.1 * h * torch.exp(-r2)
        x = x - turn * y + (0.2 + 0.1 * u[1]) * h
        y = y + turn * x + (0.2 + 0.1 * u[2]) * h
        return x, y, g, h
    # 'wall': shear layer around the unit circle, jittered lattice cut to 1 <= r <= 1.5
    area = math.pi * (1.5**2 - 1.0)
    h = math.sqrt(area / n)
    hl = 0.993 * h
    m = int(math.ceil(1.5 / hl)) + 1
    c = torch.arange(-m, m + 1, dtype=torch.float64, device=device) * hl
    x, y = c.repeat_interleave(2 * m + 1), c.repeat(2 * m + 1)
    x = x + (_rand(x.numel(), gen) - 0.5) * (0.5 * h)
    y = y + (_rand(y.numel(), gen) - 0.5) * (0.5 * h)
    r = torch.sqrt(x * x + y * y)
    keep = torch.nonzero((r >= 1.0) & (r <= 1.5)).ravel()
    if keep.numel() > n:  # n of them, in lattice order
        pick = torch.argsort(_rand(keep.numel(), gen))[:n]
        keep = keep[torch.sort(pick).values]
    x, y, r = x[keep].contiguous(), y[keep].contiguous(), r[keep]
    g = -(2.0 / 0.02) * torch.exp(-(r - 1.0) / 0.02) * (h * h)
    return x, y, g, h


def _body(m, seed):
    """End points of m panels on an ellipse, its free stream and strengths."""
    gen = _gen(seed, "cpu")
    a, b = 1.0, 0.6 + 0.4 * float(_rand(1, gen))
    th = torch.linspace(math.pi, -math.pi, m + 1, dtype=torch.float64)
    d = float(th[1] - th[0])
    px = a / math.cos(d / 2) * torch.cos(th - d / 2)
    py = b / math.cos(d / 2) * torch.sin(th - d / 2)
    px[-1], py[-1] = px[0], py[0]
    s = torch.randn(m, dtype=torch.float64, generator=gen)
    return px, py, s


def _panel_frame(px, py):
    xs, ys, xe, ye = px[:-1], py[:-1], px[1:], py[1:]
    lx, ly = xe - xs, ye - ys
    ln = torch.sqrt(lx * lx + ly * ly)
    c, s = lx / ln, ly / ln
    xc = 0.5 * (xs + xe) + s * ln * 0.1
    yc = 0.5 * (ys + ye) - c * ln * 0.1
    return [t.contiguous().to(DEV) for t in (xs, ys, xe, ye, c, s, xc, yc)]


def _layer_points(n, seed):
    """Points in the layer around the body of _body (between 1 and 1.5 radii)."""
    gen = _gen(seed + 500)
    r, a = 1.0 + 0.5 * _rand(n, gen), 2.0 * math.pi * _rand(n, gen)
    return r * torch.cos(a), r * torch.sin(a)


def _set_sizes(case, seed):
    gen = _gen(1, "cpu")  # the sizes are the case's, not the seed's
    u = _rand(case["sets"], gen).tolist()
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [int(math.exp(lo + v * (hi - lo))) for v in u]


def _batch_blobs(case, seed):
    return [_blobs("lattice" if i % 3 == 2 else "uniform", n, 100 * seed + i)
            for i, n in enumerate(_set_sizes(case, seed))]


VINF = (1.0, 0.1)
CONTROL = (1e-8, 1e-8)  # pHyFlow's default thresholds


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "velocity":
        x, y, g, h = _blobs(case["layout"], case["n"], seed)
        return {"kind": kind, "a": (x, y, g), "sigma": h / OVERLAP, "tol": case["tol"],
                "method": pfblob.DIRECT_METHOD if case["method"] == "direct"
                else pfblob.FMM_METHOD}
    if kind == "vorticity":
        x, y, g, h = _blobs("lattice", case["n"], seed)
        return {"kind": kind, "a": (x, y, g), "sigma": h / OVERLAP}
    if kind == "regrid":
        x, y, g, h = _blobs(case["layout"], case["n"], seed)
        return {"kind": kind, "a": (x, y, g), "h": h, "c": case["c"], "control": case["control"]}
    if kind == "panels":
        px, py, s = _body(case["m"], seed)
        xs, ys, xe, ye, c, sn, _, _ = _panel_frame(px, py)
        return {"kind": kind, "a": (s.to(DEV), xs, ys, xe, ye, c, sn,
                                    *_layer_points(case["n"], seed))}
    if kind == "system":
        px, py, s = _body(case["m"], seed)
        xs, ys, xe, ye, c, sn, xc, yc = _panel_frame(px, py)
        return {"kind": kind, "a": (xc, yc, xs, ys, xe, ye, c, sn),
                "rhs": -(VINF[0] * c + VINF[1] * sn)}
    if kind == "coupled":
        px, py, _ = _body(case["m"], seed)
        x, y, g, h = _blobs("wall", case["n"], seed)
        panels = pfblob.Panels({"body": {"xPanel": px.numpy(), "yPanel": py.numpy(),
                                         "cmGlobal": np.zeros(2), "thetaLocal": 0.0,
                                         "dPanel": 0.01}}, problemType="fixed")
        blobs = pfblob.Blobs((x.cpu().numpy(), y.cpu().numpy(), g.cpu().numpy()),
                             vInf=list(VINF), nu=0.0, deltaTc=1e-3, h=h, overlap=OVERLAP,
                             blobControlParams={"stepRedistribution": 0,
                                                "stepPopulationControl": 0,
                                                "gThresholdLocal": 1e-8,
                                                "gThresholdGlobal": 1e-8})
        xc, yc = (torch.from_numpy(np.ascontiguousarray(v)).to(DEV)
                  for v in panels.xyCPGlobalCat)
        return {"kind": kind, "solver": pfblob.LagrangianSolver(blobs, panels), "cp": (xc, yc),
                "at": (x, y)}
    if kind == "batch":
        sims = [{"x": x, "y": y, "g": g, "sigma": h / OVERLAP, "overlap": OVERLAP}
                for x, y, g, h in _batch_blobs(case, seed)]
        return {"kind": kind, "batch": Batch(sims)}
    x, y, g, h = _blobs("uniform", case["n"], seed, "cpu")
    return {"kind": "host", "a": (x.numpy(), y.numpy(), g.numpy()), "sigma": h / OVERLAP,
            "bounds": np.array([-1.5 * h, 1.5 * h])}


def run(state):
    kind = state["kind"]
    if kind == "velocity":
        return pfblob.velocity(*state["a"], state["sigma"], k=K, method=state["method"],
                               tol=state["tol"])
    if kind == "vorticity":
        return pfblob.vorticity(*state["a"], state["sigma"], k=K)
    if kind == "regrid":
        h = state["h"]
        out = pfblob.remesh_device(*state["a"], h, -1.5 * h, -1.5 * h, c=state["c"],
                                   population_control=CONTROL if state["control"] else None)
        return out[:3]
    if kind == "panels":
        return pfblob.inducedVelocity(*state["a"])
    if kind == "system":
        A = pfblob.influenceMatrix(*state["a"])
        lu, piv = pfblob.lu_factor(A)
        return A, lu, piv, pfblob.lu_solve((lu, piv), state["rhs"])
    if kind == "coupled":
        solver = state["solver"]
        vx, vy = solver.blobs.evaluateVelocity(*state["cp"])
        solver.panels.solve(vx + VINF[0], vy + VINF[1])
        return solver.evaluateVelocity(*state["at"])
    if kind == "batch":
        state["batch"].run()
        return [[r[k] for k in ("vx", "vy", "x", "y", "g")] for r in state["batch"].results()]
    return pfblob.velocity_and_regrid(*state["a"], state["sigma"], OVERLAP, state["bounds"],
                                      state["bounds"], k=K)


# ---------------------------------------------------------------------------
# the least work of one pass
def _near(n):
    """Partners of a blob inside the Gaussian core's reach (sqrt(ks ln 1e8) = 7.6 h)."""
    return min(n, 180)


def _velocity_work(ns, nt, direct):
    pairs = ns * nt if direct else nt * _near(ns)
    far = 0 if direct else 16 * 8 * (ns + nt) + 20 * (ns + nt)  # P2M and L2P, 16 terms
    return {"bytes": 8.0 * (3 * ns + 4 * nt), "flops": 16.0 * pairs + far}


def _remesh_work(n):
    return {"bytes": 8.0 * 6 * n, "flops": 80.0 * n}


def work(case):
    kind = case["kind"]
    if kind == "velocity":
        return _velocity_work(case["n"], case["n"], case["method"] == "direct")
    if kind == "vorticity":
        return {"bytes": 32.0 * case["n"], "flops": 10.0 * case["n"] * _near(case["n"])}
    if kind == "regrid":
        return _remesh_work(case["n"])
    if kind == "panels":
        return {"bytes": 8.0 * 4 * case["n"] + 56 * case["m"], "flops": 8.0 * 40 * case["n"]}
    if kind == "system":
        m = case["m"]
        return {"bytes": 8.0 * 3 * m * m, "flops": 2.0 / 3 * m**3 + 60.0 * m * m + 2.0 * m * m}
    if kind == "coupled":
        m, n = case["m"], case["n"]
        parts = [_velocity_work(n, m, False), _velocity_work(n, n, False),
                 {"bytes": 8.0 * m * m, "flops": 2.0 * m * m + 8.0 * 40 * n}]
    elif kind == "batch":
        sizes = _set_sizes(case, 0)
        parts = [_velocity_work(n, n, False) for n in sizes] + [_remesh_work(n) for n in sizes]
    else:
        parts = [_velocity_work(case["n"], case["n"], False), _remesh_work(case["n"])]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


# ---------------------------------------------------------------------------
# the results in FP64
def _velocity_exact(x, y, g, ks, xt, yt):
    vx, vy = torch.zeros_like(xt), torch.zeros_like(xt)
    rows = max(1, (1 << 22) // max(1, x.numel()))
    for i in range(0, xt.numel(), rows):
        dx, dy = xt[i:i + rows, None] - x, yt[i:i + rows, None] - y
        r2 = dx * dx + dy * dy + EPS
        s = -torch.expm1(r2 / -ks) / r2
        vx[i:i + rows] = -((dy * s) @ g) / (2 * math.pi)
        vy[i:i + rows] = ((dx * s) @ g) / (2 * math.pi)
    return vx, vy


def _vorticity_exact(x, y, g, ks, xt, yt):
    w = torch.zeros_like(xt)
    rows = max(1, (1 << 22) // max(1, x.numel()))
    for i in range(0, xt.numel(), rows):
        dx, dy = xt[i:i + rows, None] - x, yt[i:i + rows, None] - y
        w[i:i + rows] = torch.exp((dx * dx + dy * dy + EPS) / -ks) @ g
    return w / (math.pi * ks)


def _m4(u, c2):
    a = torch.abs(u)
    outer = 0.5 * (2 - a) ** 2 * (1 - a) - c2 * (2 - a) ** 2 * (1 - 2 * a)
    inner = 1 - 2.5 * a * a + 1.5 * a**3 - c2 * (2 - 9 * a * a + 6 * a**3)
    return torch.where(a < 1, inner, torch.where((a > 1) & (a < 2), outer, torch.zeros_like(a)))


def _remesh_exact(x, y, g, h, b0, c, control=None):
    """M4' (with Wee's c) of pHyFlow's Regrid on the lattice i h + h/2 + b0, the
    touched nodes in (ix, iy) order, then its PopulationControl."""
    il = (torch.ceil((((x - b0) - 2.0 * h) + 0.5 * h) / h) - 1).long()
    jl = (torch.ceil((((y - b0) - 2.0 * h) + 0.5 * h) / h) - 1).long()
    off = b0 / h
    i0, j0 = int(il.min()), int(jl.min())
    width = int(jl.max()) - j0 + 4
    ids, val = [], []
    for a in range(4):
        wx = _m4(((il + a).double() + 0.5 + off) - x / h, c * c)
        for b in range(4):
            wy = _m4(((jl + b).double() + 0.5 + off) - y / h, c * c)
            ids.append((il + a - i0) * width + (jl + b - j0))
            val.append(wx * wy * g)
    cells, inv = torch.unique(torch.cat(ids), sorted=True, return_inverse=True)
    gn = torch.zeros(cells.numel(), dtype=torch.float64, device=x.device)
    gn.index_add_(0, inv, torch.cat(val))
    xn = (cells // width + i0).double() * h + 0.5 * h + b0
    yn = (cells % width + j0).double() * h + 0.5 * h + b0
    if control is not None:
        thr = control[0]
        while not float(torch.abs(gn)[torch.abs(gn) < thr].sum()) < control[1]:
            thr /= 10.0
        keep = ~(torch.abs(gn) < thr)
        xn, yn, gn = xn[keep], yn[keep], gn[keep]
    return xn, yn, gn


def _panel_pairs(xs, ys, xe, ye, c, s, xt, yt):
    """Velocity of each panel at unit strength at the points: two (points, panels) arrays."""
    x2 = c * (xe - xs) + s * (ye - ys)
    dx, dy = xt[:, None] - xs, yt[:, None] - ys
    xp, yp = c * dx + s * dy, c * dy - s * dx
    th = (torch.atan2(yp, xp - x2) - torch.atan2(yp, xp)) / (2 * math.pi)
    lg = torch.log((xp * xp + yp * yp) / ((xp - x2) ** 2 + yp * yp)) / (4 * math.pi)
    return c * th + s * lg, s * th - c * lg


def _panel_exact(strength, xs, ys, xe, ye, c, s, xt, yt):
    vx, vy = torch.zeros_like(xt), torch.zeros_like(xt)
    rows = max(1, (1 << 22) // max(1, xs.numel()))
    for i in range(0, xt.numel(), rows):
        u, v = _panel_pairs(xs, ys, xe, ye, c, s, xt[i:i + rows], yt[i:i + rows])
        vx[i:i + rows], vy[i:i + rows] = u @ strength, v @ strength
    return vx, vy


def exact(case, seed):
    kind = case["kind"]
    if kind in ("velocity", "vorticity"):
        x, y, g, h = _blobs(case.get("layout", "lattice"), case["n"], seed)
        if float(x.numel()) ** 2 > PAIRS_EXACT:
            return None
        f = _velocity_exact if kind == "velocity" else _vorticity_exact
        return f(x, y, g, K * (h / OVERLAP) ** 2, x, y)
    if kind == "regrid":
        x, y, g, h = _blobs(case["layout"], case["n"], seed)
        return _remesh_exact(x, y, g, h, -1.5 * h, case["c"],
                             CONTROL if case["control"] else None)
    if kind == "panels":
        px, py, s = _body(case["m"], seed)
        xs, ys, xe, ye, c, sn, _, _ = _panel_frame(px, py)
        return _panel_exact(s.to(DEV), xs, ys, xe, ye, c, sn, *_layer_points(case["n"], seed))
    if kind == "system":
        px, py, s = _body(case["m"], seed)
        xs, ys, xe, ye, c, sn, xc, yc = _panel_frame(px, py)
        u, v = _panel_pairs(xs, ys, xe, ye, c, sn, xc, yc)
        A = u * c[:, None] + v * sn[:, None]
        return A, None, None, torch.linalg.solve(A, -(VINF[0] * c + VINF[1] * sn))
    if kind == "coupled":
        px, py, _ = _body(case["m"], seed)
        xs, ys, xe, ye, c, sn, xc, yc = _panel_frame(px, py)
        x, y, g, h = _blobs("wall", case["n"], seed)
        if float(x.numel()) ** 2 > PAIRS_EXACT:
            return None
        ks = K * (h / OVERLAP) ** 2
        vx, vy = _velocity_exact(x, y, g, ks, xc, yc)
        u, v = _panel_pairs(xs, ys, xe, ye, c, sn, xc, yc)
        s = torch.linalg.solve(u * c[:, None] + v * sn[:, None],
                               -((vx + VINF[0]) * c + (vy + VINF[1]) * sn))
        bx, by = _velocity_exact(x, y, g, ks, x, y)
        wx, wy = _panel_exact(s, xs, ys, xe, ye, c, sn, x, y)
        return bx + wx + VINF[0], by + wy + VINF[1]
    if kind == "batch":
        return [[*_velocity_exact(x, y, g, K * (h / OVERLAP) ** 2, x, y),
                 *_remesh_exact(x, y, g, h / OVERLAP * OVERLAP, -1.5 * (h / OVERLAP * OVERLAP),
                                0.0)]
                for x, y, g, h in _batch_blobs(case, seed)]
    x, y, g, h = (v.to(DEV) if isinstance(v, torch.Tensor) else v
                  for v in _blobs("uniform", case["n"], seed, "cpu"))
    if float(x.numel()) ** 2 > PAIRS_EXACT:
        return None
    hs = h / OVERLAP * OVERLAP
    return (*_velocity_exact(x, y, g, K * (h / OVERLAP) ** 2, x, y),
            *_remesh_exact(x, y, g, hs, -1.5 * h, 0.0))
