"""Induced vorticity of Gaussian blobs on the GPU (pf_vorticity_direct) vs the
reference's own ww2parGauss loop (golden) and the FP64 oracle.

Tolerance: max_i |w_i - w_ref_i| / max_i |w_ref_i| <= 1e-6."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-6


def err(w, r):
    return float(np.abs(np.asarray(w) - r).max() / np.abs(r).max())


def test_c1_vs_reference_golden(golden):
    import pfblob
    d = golden("vort_c1")
    w = pfblob.vorticity(d["x"], d["y"], d["g"], float(d["sigma"]))
    assert err(w, d["w"]) <= TOL


def test_edge_cases_and_separate_targets_vs_reference_golden(golden):
    import pfblob
    d = golden("vort_rand")
    w = pfblob.vorticity(d["x"], d["y"], d["g"], float(d["sigma"]), xEval=d["xt"], yEval=d["yt"])
    assert np.all(np.isfinite(w))
    assert err(w, d["w"]) <= TOL


@pytest.mark.parametrize("n", [1, 300, 5000, 70000])
def test_sizes_vs_oracle_and_repeatable(n):
    """Covers the source-segment path (small sets) and the plain path."""
    import pfblob
    rng = np.random.default_rng(n)
    x, y = rng.random(n), rng.random(n)
    g = rng.standard_normal(n) / n
    sigma = 0.005
    a = pfblob.vorticity(x, y, g, sigma)
    b = pfblob.vorticity(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(),
                         torch.from_numpy(g).cuda(), sigma)
    assert np.array_equal(a, b.cpu().numpy())
    sub = rng.choice(n, min(n, 2000), replace=False)
    r = oracle.vorticity_direct(x, y, g, 2 * sigma * sigma, x[sub].copy(), y[sub].copy())
    assert err(a[sub], r) <= TOL


def test_empty_and_options():
    import pfblob
    x = np.zeros(0)
    assert pfblob.vorticity(x, x, x, 0.01).shape == (0,)
    w = pfblob.vorticity(x, x, x, 0.01, xEval=np.ones(3), yEval=np.ones(3))
    assert np.array_equal(w, np.zeros(3))
    with pytest.raises(Exception):
        pfblob.vorticity(np.ones(3), np.ones(3), np.ones(3), 0.01, method=0)


@pytest.mark.parametrize("n,order", [(33, "lattice"), (257, "lattice"), (5000, "lattice"),
                                     (20164, "lattice"), (5000, "random"), (5000, "clusters")])
def test_sources_beyond_reach_add_nothing(n, order):
    """Sources out of the exponential's FP32 range are skipped: lattice order
    (most chunks skipped), random order (none), two clusters far apart (all of
    the other one) against the FP64 oracle, 1e-6 as above; and a source that
    is not finite still reaches every target."""
    import pfblob
    rng = np.random.default_rng(n)
    s = int(np.sqrt(n))
    h = 2.0 / max(s, 2)
    if order == "lattice":
        c = -1.0 + (np.arange(s) + 0.5) * h
        x, y = (a.ravel().copy() for a in np.meshgrid(c, c, indexing="ij"))
    else:
        x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        if order == "clusters":
            x[n // 2:] += 50.0
            x[: n // 2] *= 0.1
    g = rng.standard_normal(x.size) / x.size
    sigma = h / 0.8
    w = pfblob.vorticity(x, y, g, sigma)
    assert err(w, oracle.vorticity_direct(x, y, g, 2 * sigma * sigma, x, y)) <= TOL
    for bad in (np.nan, np.inf):
        gb = g.copy()
        gb[x.size // 3] = bad
        assert np.isnan(pfblob.vorticity(x, y, gb, sigma, xEval=np.array([900.0]),
                                         yEval=np.array([-900.0]))).all()


@pytest.mark.parametrize("ns,nt,order", [(9216, 9216, "lattice"), (9409, 9409, "lattice"),
                                         (12100, 12100, "lattice"), (18225, 18225, "lattice"),
                                         (9500, 9500, "random"), (13000, 13001, "clusters"),
                                         (150001, 700, "random"), (33, 3000001, "lattice")])
def test_tested_and_untested_sets(ns, nt, order):
    """Around the number of pairs from which sources are tested (8.5e7), one wave of
    CTAs and several, many sources for few targets and the reverse: against the
    FP64 oracle, 1e-6 as above; the strengths of sources beyond every target's
    reach change no bit; a source that is not finite still reaches all."""
    import pfblob
    rng = np.random.default_rng(ns + nt)

    def points(n):
        if order == "lattice":
            s = int(np.ceil(np.sqrt(n)))
            c = -1.0 + (np.arange(s) + 0.5) * (2.0 / s)
            return [a.ravel()[:n].copy() for a in np.meshgrid(c, c, indexing="ij")]
        x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        if order == "clusters":
            x[n // 2:] += 50.0
        return [x, y]

    x, y = points(ns)
    xt, yt = (x, y) if nt == ns else points(nt)
    g = rng.standard_normal(ns) / ns
    sigma = 2.5 / np.sqrt(max(ns, nt))
    far = rng.choice(ns, ns // 10, replace=False)
    y[far] = 200.0
    if nt == ns:
        yt = np.where(np.isin(np.arange(ns), far), 0.5, y)
    w = pfblob.vorticity(x, y, g, sigma, xEval=xt, yEval=yt)
    sub = rng.choice(nt, min(nt, 2000), replace=False)
    r = oracle.vorticity_direct(x, y, g, 2 * sigma * sigma, xt[sub].copy(), yt[sub].copy())
    assert err(w[sub], r) <= TOL
    g2 = g.copy()
    g2[far] *= 1e6
    assert np.array_equal(w, pfblob.vorticity(x, y, g2, sigma, xEval=xt, yEval=yt))
    g2[far[0]] = np.inf
    assert np.isnan(pfblob.vorticity(x, y, g2, sigma, xEval=xt, yEval=yt)).all()
