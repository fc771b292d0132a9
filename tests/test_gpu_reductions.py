"""The reductions of the JD iteration where their launch shape changes: one
CTA (n <= 2048), two CTAs, the wide grid from 4096 rows on, a partial last
stride, and more columns than one column group (8) holds."""
import numpy as np
import pytest
import scipy.linalg as sl

from jadamilu_gb300 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,neig", [(33, 2), (2048, 9), (2049, 1), (4095, 3), (4096, 9), (4097, 1), (8193, 9),
                                    (17000, 2)])
def test_solve_at_reduction_edges(gpu, n, neig):
    """A residual of TOL bounds the distance to an eigenvalue by TOL; the
    rest is the rounding of ||A|| ~ n in the two solvers."""
    ia, ja, a = M.tridiag(n)
    r = gpu.dpjd((a, ja, ia), neig, isearch=2, sigma=0.0, madspace=20, maxit=5000, tol=1e-10, droptol=1e-3,
                 icntl=(0, 1, 0, 0, 0))
    assert r["info"] == 0 and r["neig"] == neig
    w = sl.eigh_tridiagonal(np.arange(n, dtype=np.float64), np.full(n - 1, 5.0), eigvals_only=True, select="i",
                            select_range=(0, min(n, 60) - 1))
    bound = 1e-10 + 64 * np.finfo(float).eps * n
    for lam in r["eigs"]:
        assert np.min(np.abs(w - lam)) <= bound
    assert len(set(np.round(r["eigs"], 6))) == neig
    A = M.to_scipy_full(ia, ja, a)
    for k in range(neig):
        v = r["x"][:, k]
        assert np.linalg.norm(A @ v - r["eigs"][k] * v) <= 2 * bound * np.linalg.norm(v)
