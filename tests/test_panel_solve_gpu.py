"""Panel influence matrix (vs the reference Cython assemble_influenceMatrix)
and the on-device LU factor / solve of the panel system (vs numpy's solve)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_influence_matrix_vs_reference_golden(golden):
    import pfblob
    d = golden("panel_influence")
    A = pfblob.influenceMatrix(d["xcp"], d["ycp"], d["xs"], d["ys"], d["xe"], d["ye"], d["cosa"],
                               d["sina"])
    assert A.shape == d["A"].shape
    assert np.abs(A - d["A"]).max() <= 1e-12 * np.abs(d["A"]).max()


@pytest.mark.parametrize("n", [1, 31, 96, 700])
def test_lu_solve_matches_numpy(golden, n):
    import pfblob
    rng = np.random.default_rng(n)
    if n == 96:
        A = golden("panel_influence")["A"]
    else:
        A = rng.standard_normal((n, n)) + n * np.eye(n) * 0.1
    b = rng.standard_normal(n)
    lu, piv = pfblob.lu_factor(A)
    x = pfblob.lu_solve((lu, piv), b)
    ref = np.linalg.solve(A, b)
    assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()
    assert np.abs(A @ x - b).max() <= 1e-12 * np.abs(A).max() * np.abs(x).max() * n
    # device tensors in, device tensors out, same numbers
    At = torch.from_numpy(A).cuda()
    lt, pt = pfblob.lu_factor(At)
    xt = pfblob.lu_solve((lt, pt), torch.from_numpy(b).cuda())
    assert np.array_equal(xt.cpu().numpy(), x)
    assert torch.equal(At, torch.from_numpy(A).cuda())  # input not overwritten


def test_partial_pivoting_and_singular_warning():
    import pfblob
    A = np.array([[0.0, 2.0, 1.0], [1.0, 1.0, 0.0], [3.0, 0.0, 1.0]])
    b = np.array([1.0, 2.0, 3.0])
    lu, piv = pfblob.lu_factor(A)
    assert piv[0] == 2  # largest |a_i0| is row 2
    assert np.allclose(pfblob.lu_solve((lu, piv), b), np.linalg.solve(A, b), rtol=1e-14)
    S = np.array([[1.0, 2.0], [2.0, 4.0]])
    with pytest.warns(RuntimeWarning):
        pfblob.lu_factor(S)


@pytest.mark.parametrize("n", [2, 8, 32, 33, 64, 255, 257, 511, 513, 900, 1023, 1025, 2047, 2049])
def test_lu_at_panel_edges_within_the_rounding_bound(n):
    """P A = L U to the a priori bound of Gaussian elimination,
    |PA - LU| <= 2 n u |L||U| elementwise (u = 2^-53, any order of the sums),
    with |L| <= 1 (partial pivoting), at the sizes where the panel kernels
    change; the same bound for the two substitutions' residual."""
    import pfblob
    rng = np.random.default_rng(1000 + n)
    A = rng.standard_normal((n, n))
    A[:, rng.permutation(n)[: n // 3]] *= 1e-3
    b = rng.standard_normal(n)
    lu, piv = pfblob.lu_factor(A)
    P = np.arange(n)
    for k in range(n):
        assert k <= piv[k] < n
        P[[k, piv[k]]] = P[[piv[k], k]]
    L, U = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert np.abs(L).max() <= 1.0
    u = 2.0 ** -53
    LU = np.abs(L) @ np.abs(U)
    assert (np.abs(A[P] - L @ U) <= 4 * n * u * LU).all()  # 2 n u, and as much for numpy's product
    x = pfblob.lu_solve((lu, piv), b)
    r = np.abs(A @ x - b)[P]
    assert (r <= 8 * n * u * (LU @ np.abs(x)) + 4 * n * u * np.abs(b)[P]).all()


def _substitution_residual(lu, piv, b, x):
    """|P b - L U x| and |L| |U| |x| in extended precision, row by row."""
    n = b.shape[0]
    e = np.longdouble
    p = b.astype(e)
    for k in range(n):
        p[[k, piv[k]]] = p[[piv[k], k]]
    L, U = np.tril(lu, -1).astype(e) + np.eye(n, dtype=e), np.triu(lu).astype(e)
    return np.abs(L @ (U @ x.astype(e)) - p), np.abs(L) @ (np.abs(U) @ np.abs(x.astype(e)))


@pytest.mark.parametrize("n,at", [(24, 0), (24, 11), (24, 23), (33, 0), (33, 31), (33, 32),
                                  (512, 5), (512, 250), (512, 511)])
@pytest.mark.parametrize("what,s", [("column", 1e-101), ("column", 1e-150), ("column", 1e150),
                                    ("diagonal", 1e-101), ("diagonal", 1e-150),
                                    ("diagonal", 1e150), ("diagonal", 1e-305),
                                    ("diagonal", 1e305)])
def test_lu_solve_with_one_extreme_diagonal(n, at, what, s):
    """Given factors, one column of U or only its diagonal of an extreme
    magnitude (at 1e-305 and 1e305 the quotients U / d leave the normal range):
    the residual bound of the two substitutions, |P b - L U x| <= 2 n u |L||U||x|
    with u = 2^-53, one more rounding per quotient, and a factor 2."""
    import pfblob
    rng = np.random.default_rng(7 * n + at)
    lu = rng.uniform(0.5, 1.0, (n, n)) * np.where(rng.random((n, n)) < 0.5, -1.0, 1.0)
    lu = np.tril(lu, -1) / n + np.triu(lu, 1) / n + np.diag(lu.diagonal())
    if what == "column":
        lu[: at + 1, at] *= s
    else:
        lu[at, at] = s
    piv = np.array([rng.integers(k, n) for k in range(n)], dtype=np.int32)
    e = np.longdouble
    xt = (rng.uniform(0.5, 1.0, n) / np.where(np.arange(n) == at, s, 1.0)
          if what == "column" else rng.uniform(0.5, 1.0, n))
    b = (np.tril(lu, -1).astype(e) + np.eye(n, dtype=e)) @ (np.triu(lu).astype(e) @ xt.astype(e))
    for k in reversed(range(n)):
        b[[k, piv[k]]] = b[[piv[k], k]]
    b = b.astype(np.float64)
    x = pfblob.lu_solve((lu, piv), b)
    assert np.isfinite(x).all()
    r, size = _substitution_residual(lu, piv, b, x)
    assert (r <= 4 * (n + 2) * 2.0 ** -53 * size).all()


def test_lu_solve_at_the_ends_of_the_range():
    """Small systems whose solution is exact: a right-hand side that overflows
    when it is divided by the diagonal before the others' share is taken off,
    a zero diagonal (the unknowns below it are right, it and those above are not
    finite)."""
    import pfblob
    piv = np.arange(3, dtype=np.int32)

    def solve(u, b):
        n = len(b)
        return pfblob.lu_solve((np.array(u), piv[:n]), np.array(b))

    assert solve([[2.0, 1.0], [0.0, 1e-120]], [3.0, 1e-120]).tolist() == [1.0, 1.0]
    assert solve([[2.0, 3.0, 0.0], [0.0, 1e-120, 0.0], [0.0, 0.0, 1.0]],
                 [8.0, 2e-120, 1.0]).tolist() == [1.0, 2.0, 1.0]
    assert solve([[1e-99, 1.0], [0.0, 1.0]], [1e250, 1e250]).tolist() == [0.0, 1e250]
    x = solve([[2.0, 1.0, 4.0], [0.0, 0.0, 2.0], [0.0, 0.0, 8.0]], [1.0, 1.0, 16.0])
    assert x[2] == 2.0 and x[1] == -np.inf and not np.isfinite(x[0])


def test_lu_factor_wide_stripes():
    """m > 4096, where a stripe has 32 columns: the bound of
    test_lu_at_panel_edges_within_the_rounding_bound, in FP64 on the device."""
    import pfblob
    n, u = 4100, 2.0 ** -53
    gen = torch.Generator(device="cuda").manual_seed(4100)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen)
    lu, piv = pfblob.lu_factor(A)
    P, pv = np.arange(n), piv.cpu().numpy()
    for k in range(n):
        assert k <= pv[k] < n
        P[[k, pv[k]]] = P[[pv[k], k]]
    L = torch.tril(lu, -1) + torch.eye(n, dtype=torch.float64, device="cuda")
    U = torch.triu(lu)
    assert float(L.abs().max()) <= 1.0
    err = (A[torch.from_numpy(P).cuda()] - L @ U).abs()
    assert bool((err <= 4 * n * u * (L.abs() @ U.abs())).all())


def test_lu_solve_right_hand_side_in_global_memory():
    """More unknowns than shared memory holds (8192), factors given."""
    import pfblob
    n, u = 8200, 2.0 ** -53
    gen = torch.Generator(device="cuda").manual_seed(8200)
    lu = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen) / n
    lu.diagonal().add_(1.0)
    lu[:, 8000] *= 1e-120
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    rng = np.random.default_rng(8200)
    pv = np.array([rng.integers(k, n) for k in range(n)], dtype=np.int32)
    x = pfblob.lu_solve((lu, torch.from_numpy(pv).cuda()), b)
    P = np.arange(n)
    for k in range(n):
        P[[k, pv[k]]] = P[[pv[k], k]]
    L = torch.tril(lu, -1) + torch.eye(n, dtype=torch.float64, device="cuda")
    U = torch.triu(lu)
    r = (L @ (U @ x) - b[torch.from_numpy(P).cuda()]).abs()
    size = L.abs() @ (U.abs() @ x.abs())
    assert bool((r <= 8 * n * u * size).all())
