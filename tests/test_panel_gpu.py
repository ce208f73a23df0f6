"""Vortex-panel velocity on the GPU vs the reference Cython kernel (golden)
and the oracle.  Gate: normwise relative error <= 1e-6."""
import numpy as np
import pytest
import torch

import oracle
from conftest import normwise_err

pytestmark = pytest.mark.gpu
TOL = 1e-6


def test_cylinder_vs_reference_golden(golden):
    import pfblob
    p = golden("panel_cyl")
    vx, vy = pfblob.inducedVelocity(p["gamma"], p["xs"], p["ys"], p["xe"], p["ye"], p["cosa"],
                                    p["sina"], p["xv"], p["yv"])
    # the point 1e-6 from the panel (index 3) has a large, well-defined value
    assert normwise_err(vx[4:], vy[4:], p["vx"][4:], p["vy"][4:]) <= TOL
    assert abs(vx[3] - p["vx"][3]) <= 1e-5 * abs(p["vx"][3]) + 1e-6
    # on the line extension of a panel: finite and equal to the reference
    assert np.allclose(vx[:3], p["vx"][:3], rtol=1e-5, atol=1e-7)


def test_512_panels_shear_layer_points():
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(512)
    rng = np.random.default_rng(2)
    r = rng.uniform(1.0, 1.5, 20000)
    t = rng.uniform(-np.pi, np.pi, 20000)
    xv, yv = r * np.cos(t), r * np.sin(t)
    rx, ry = oracle.panel_velocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    vx, vy = pfblob.inducedVelocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    assert normwise_err(vx, vy, rx, ry) <= TOL


def test_accumulate_onto_blob_velocity():
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(64)
    dev = torch.device("cuda", 0)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    xv = T(np.linspace(-2, 2, 1000))
    yv = T(np.full(1000, 1.7))
    vx = torch.full((1000,), 0.25, dtype=torch.float64, device=dev)
    vy = torch.full((1000,), -0.5, dtype=torch.float64, device=dev)
    pfblob.panel_velocity_device(T(ps.gamma), T(ps.xs), T(ps.ys), T(ps.xe), T(ps.ye), T(ps.cosa),
                                 T(ps.sina), xv, yv, vx, vy, accumulate=True)
    rx, ry = oracle.panel_velocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina,
                                   xv.cpu().numpy(), yv.cpu().numpy())
    assert normwise_err(vx.cpu().numpy() - 0.25, vy.cpu().numpy() + 0.5, rx, ry) <= TOL


def test_far_points_series_to_1e10():
    """Points well away from the body take the groups' series only: they match
    the FP64 pair formula to 1e-10 (the series' stated remainder), far inside
    the 1e-6 gate that the FP32 transcendentals of the near field set."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(512)
    rng = np.random.default_rng(4)
    r = rng.uniform(2.0, 6.0, 20000)
    t = rng.uniform(-np.pi, np.pi, 20000)
    xv, yv = r * np.cos(t), r * np.sin(t)
    rx, ry = oracle.panel_velocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    vx, vy = pfblob.inducedVelocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    assert normwise_err(vx, vy, rx, ry) <= 1e-10


def test_shuffled_panels_and_many_groups():
    """The grouping never changes the sum: panels in random order (every group
    spans the body, so every point is near) and a body of 1000 panels (a
    partial last group, several shared-memory tiles) both meet the gate."""
    import pfblob
    from pfblob import workloads as wl
    rng = np.random.default_rng(6)
    r = rng.uniform(1.0, 3.0, 8000)
    t = rng.uniform(-np.pi, np.pi, 8000)
    xv, yv = r * np.cos(t), r * np.sin(t)
    for m, shuffle in ((512, True), (1000, False), (1000, True)):
        ps = wl.cylinder_panels(m)
        arrs = [ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina]
        if shuffle:
            perm = rng.permutation(m)
            arrs = [a[perm] for a in arrs]
        rx, ry = oracle.panel_velocity(*arrs, xv, yv)
        vx, vy = pfblob.inducedVelocity(*arrs, xv, yv)
        assert normwise_err(vx, vy, rx, ry) <= TOL, (m, shuffle)


def test_source_panels_vs_reference_golden(golden):
    """Constant-source panels (panelKernel=0): velocity against the
    reference's Cython kernel (gate 1e-6; the point 1e-6 from panel 0 and the
    points on its line extension as for vortex panels) and the influence
    matrix against its assemble_influenceMatrix (1e-12)."""
    import pfblob
    d = golden("source_panel")
    args = [d[k] for k in ("sigma", "xs", "ys", "xe", "ye", "cosa", "sina")]
    vx, vy = pfblob.inducedVelocity(*args, d["xv"], d["yv"], panelKernel=0)
    assert normwise_err(vx[4:], vy[4:], d["vx"][4:], d["vy"][4:]) <= TOL
    e3 = np.hypot(vx[3] - d["vx"][3], vy[3] - d["vy"][3])
    assert e3 <= 1e-5 * np.hypot(d["vx"][3], d["vy"][3]) + 1e-6
    assert np.allclose(vx[:3], d["vx"][:3], rtol=1e-5, atol=1e-7)
    assert np.allclose(vy[:3], d["vy"][:3], rtol=1e-5, atol=1e-7)
    A = pfblob.influenceMatrix(d["xcp"], d["ycp"], *args[1:], panelKernel=0)
    assert np.abs(A - d["A"]).max() <= 1e-12 * np.abs(d["A"]).max()


def test_source_panels_far_field_and_panels_class():
    """Far points take the groups' series only (1e-10 against the FP64
    oracle); a 'css' Panels body solves the no-through-flow condition
    (RHS = -v.n) with the source influence matrix."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(512)
    rng = np.random.default_rng(8)
    r = rng.uniform(2.0, 6.0, 8000)
    t = rng.uniform(-np.pi, np.pi, 8000)
    xv, yv = r * np.cos(t), r * np.sin(t)
    args = (ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina)
    rx, ry = oracle.source_panel_velocity(*args, xv, yv)
    vx, vy = pfblob.inducedVelocity(*args, xv, yv, panelKernel=0)
    assert normwise_err(vx, vy, rx, ry) <= 1e-10
    m = 64
    th = np.linspace(0.0, 2.0 * np.pi, m + 1)
    th[-1] = 0.0
    geo = {"b": {"xPanel": 0.5 * np.cos(th), "yPanel": 0.5 * np.sin(th),
                 "cmGlobal": np.array([0.1, 0.2]), "thetaLocal": 0.3, "dPanel": 0.01}}
    panels = pfblob.Panels(geo, panelKernel='css', problemType='fixed')
    vxe, vye = rng.standard_normal(m), rng.standard_normal(m)
    panels.solve(vxe, vye)
    n = panels.normCat
    rhs = (-vxe) * n[0] + (-vye) * n[1]
    s_ref = np.linalg.solve(panels.A, rhs)
    assert np.abs(panels.sPanel - s_ref).max() <= 1e-10 * np.abs(s_ref).max()
    assert np.all(np.asarray(panels.gTotal) == 0.0)


def _annulus(n, r0, r1, seed):
    rng = np.random.default_rng(seed)
    r = rng.uniform(r0, r1, n)
    t = rng.uniform(-np.pi, np.pi, n)
    return r * np.cos(t), r * np.sin(t)


def test_box_grid_path_near_wall_vs_oracle():
    """2^16 points (the box-grid path: far groups through each box's local
    expansion, near groups per point) in the near-wall annulus: the gate."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(512)
    xv, yv = _annulus(1 << 16, 1.0, 1.5, 8)
    rx, ry = oracle.panel_velocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    vx, vy = pfblob.inducedVelocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    assert normwise_err(vx, vy, rx, ry) <= TOL


def test_box_grid_path_far_points_to_1e10():
    """Far points on the box-grid path carry every group through the local
    expansions: still within 1e-10 of the FP64 pair formula."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(512)
    xv, yv = _annulus(1 << 16, 2.0, 6.0, 9)
    rx, ry = oracle.panel_velocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    vx, vy = pfblob.inducedVelocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina, xv, yv)
    assert normwise_err(vx, vy, rx, ry) <= 1e-10


@pytest.mark.parametrize("m,shuffle", [(512, False), (2048, False), (512, True)])
def test_box_grid_path_as_accurate_as_per_point_path(m, shuffle):
    """The same points through both paths (40,000 at once: box grid; 10,000
    at a time: every group per point) against the FP64 oracle: the box grid
    meets the gate with the per-point path's accuracy (both are set by the
    FP32 transcendentals of the pair formula at the points nearest the body;
    the box grid takes the FP64 series of sub-groups for more of its near
    panels); also with shuffled panels, whose groups span the body."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(m)
    arrs = [ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina]
    if shuffle:
        perm = np.random.default_rng(10).permutation(m)
        arrs = [a[perm] for a in arrs]
    xv, yv = _annulus(40000, 1.0, 3.0, 11)
    vx, vy = pfblob.inducedVelocity(*arrs, xv, yv)
    px, py = [], []
    for k in range(0, 40000, 10000):
        a, b = pfblob.inducedVelocity(*arrs, xv[k:k + 10000], yv[k:k + 10000])
        px.append(a)
        py.append(b)
    px, py = np.concatenate(px), np.concatenate(py)
    rx, ry = oracle.panel_velocity(*arrs, xv, yv)
    e_box, e_pt = normwise_err(vx, vy, rx, ry), normwise_err(px, py, rx, ry)
    assert e_box <= TOL and e_box <= 1.5 * e_pt + 1e-10, (e_box, e_pt)


@pytest.mark.parametrize("n,m", [(32768, 128), (32769, 130), (50001, 200), (200003, 512)])
def test_box_order_gives_the_input_orders_values(n, m):
    """Points in an order that stays in a box for long are evaluated in place,
    unordered ones in box order: the same points sorted into grid cells and
    shuffled give bitwise the same velocities (a point's arithmetic does not
    depend on the order), and
    so does accumulation onto given velocities."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(m)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    arrs = [dev(a) for a in (ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina)]
    xv, yv = _annulus(n, 1.0, 1.5, n)
    cell = np.floor((xv + 1.5) / 3.0 * 64) * 64 + np.floor((yv + 1.5) / 3.0 * 64)
    order = np.argsort(cell, kind="stable")
    xs, ys = dev(xv[order]), dev(yv[order])
    ax, ay = pfblob.inducedVelocity(*arrs, xs, ys)
    shuf = torch.randperm(n, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    bx, by = pfblob.inducedVelocity(*arrs, xs[shuf].contiguous(), ys[shuf].contiguous())
    assert torch.equal(ax[shuf], bx) and torch.equal(ay[shuf], by)
    cx, cy = torch.ones_like(bx), torch.full_like(by, -2.0)
    pfblob.panel_velocity_device(*arrs, xs[shuf].contiguous(), ys[shuf].contiguous(), cx, cy,
                                 accumulate=True)
    assert torch.equal(cx, bx + 1.0) and torch.equal(cy, by - 2.0)
    rx, ry = oracle.panel_velocity(ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina,
                                   xv[:2000].copy(), yv[:2000].copy())
    inv = np.argsort(order)[:2000]
    assert normwise_err(ax.cpu().numpy()[inv], ay.cpu().numpy()[inv], rx, ry) <= TOL


def _ring_points(n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = 1.0 + 0.5 * torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    a = 6.283185307179586 * torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    return r * torch.cos(a), r * torch.sin(a)


def test_more_points_than_one_part():
    """Above 2^24 points the set is taken in parts: bitwise the parts' own calls,
    also accumulated."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(128)
    arrs = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in (ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina)]
    part = 1 << 24
    x, y = _ring_points(part + 40001, 24)
    vx, vy = torch.ones_like(x), torch.full_like(y, -2.0)
    pfblob.panel_velocity_device(*arrs, x, y, vx, vy, accumulate=True)
    for k in (slice(0, part), slice(part, None)):
        ax, ay = pfblob.inducedVelocity(*arrs, x[k], y[k])
        assert torch.equal(vx[k], ax + 1.0) and torch.equal(vy[k], ay - 2.0)


def test_points_in_parts_where_memory_is_short():
    """4 million points need 117 MB of scratch; with 48 MB free they are taken in
    smaller parts, to the same values within the gate, and no error is left."""
    import threading
    import pfblob
    from pfblob import _lib
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(128)
    arrs = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in (ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina)]
    x, y = _ring_points(1 << 22, 22)
    rx, ry = pfblob.inducedVelocity(*arrs, x, y)
    vx, vy = torch.zeros_like(x), torch.zeros_like(y)
    out = {}

    def run():  # a thread's context has a scratch arena of its own
        try:
            pfblob.panel_velocity_device(*arrs, x[:40000], y[:40000], vx[:40000], vy[:40000])
            torch.cuda.synchronize()
            _lib.check(_lib.lib.pf_trim(_lib.context(0)))
            torch.cuda.empty_cache()
            fill = torch.empty(torch.cuda.mem_get_info()[0] - (48 << 20), dtype=torch.uint8,
                               device="cuda")
            pfblob.panel_velocity_device(*arrs, x, y, vx, vy)
            torch.cuda.synchronize()
            out["error"] = _lib.lib.pf_last_error()
            del fill
        except Exception as e:  # noqa: BLE001 (shown by the assertion below)
            out["raised"] = e

    t = threading.Thread(target=run)
    t.start()
    t.join()
    torch.cuda.empty_cache()
    assert out == {"error": b""}, out
    assert normwise_err(vx.cpu().numpy(), vy.cpu().numpy(), rx.cpu().numpy(),
                        ry.cpu().numpy()) <= TOL


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_points_that_are_not_finite_leave_the_others_alone(bad):
    """In a large set too, a point that is not finite changes no other point's
    velocity (bitwise), and its own is not finite."""
    import pfblob
    from pfblob import workloads as wl
    ps = wl.cylinder_panels(128)
    arrs = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in (ps.gamma, ps.xs, ps.ys, ps.xe, ps.ye, ps.cosa, ps.sina)]
    x, y = _ring_points(40000, 40)
    x[0], y[0], x[1], y[1] = -1.5, -1.5, 1.5, 1.5  # the others' box
    vx, vy = pfblob.inducedVelocity(*arrs, x, y)
    idx = [7, 20000, 39999]
    rest = torch.ones(40000, dtype=torch.bool, device="cuda")
    rest[idx] = False
    x[idx[0]] = bad
    y[idx[1]] = bad
    x[idx[2]] = y[idx[2]] = bad
    wx, wy = pfblob.inducedVelocity(*arrs, x, y)
    assert torch.equal(vx[rest], wx[rest]) and torch.equal(vy[rest], wy[rest])
    assert not torch.isfinite(wx[~rest] + wy[~rest]).any()
