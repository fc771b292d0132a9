"""The inner iteration in one launch against the same iteration as separate
kernels (option fuse_inner = 0: the caller's-matvec sequence), bit for bit, on
both sides of every size at which the launch shape changes: 512 rows (one
thread block), 4096 (two rows per thread), 8192 (one cluster), 77824 (one
block per SM), 311296 (four of the reduction's blocks in each)."""
import numpy as np
import pytest

from jadamilu_gb300 import matrices as M

pytestmark = pytest.mark.gpu


def _problem(kind, n):
    ia, ja, a = M.tridiag(n)
    b = np.where(ja == np.repeat(np.arange(1, n + 1), np.diff(ia)), 4.0, 1.0)
    if kind.startswith("complex"):
        a = a * np.where(b == 1.0, np.exp(0.7j), 1.0)
        b = b * np.where(b == 1.0, np.exp(-0.4j), 1.0)
    return (a, ja, ia), ((b, ja.copy(), ia) if kind.endswith("generalized") else None)


@pytest.mark.parametrize("n", [512, 513, 4095, 4096, 8192, 8193, 77824, 77825, 311296, 311297])
@pytest.mark.parametrize("kind,isearch", [("real", 2), ("complex", 0), ("generalized", 0), ("complex generalized", 2)])
def test_one_launch_equals_separate_kernels(gpu, n, kind, isearch):
    """Nine pairs: one to nine columns in the projections."""
    A, B = _problem(kind, n)
    got = []
    for fuse in (1, 0):
        gpu.set_option("fuse_inner", fuse)
        try:
            kw = dict(isearch=isearch, sigma=0.0, madspace=20, maxit=4000, tol=1e-9, droptol=1e-3, icntl=(0, 1, 0, 0, 0))
            if B is not None:
                r = (gpu.zpjd_gep if kind.startswith("c") else gpu.dpjd_gep)(A, B, 9, **kw)
            else:
                r = (gpu.zpjd if kind.startswith("c") else gpu.dpjd)(A, 9, **kw)
        finally:
            gpu.set_option("fuse_inner", 1)
        assert r["info"] == 0 and r["neig"] == 9
        got.append(r)
    assert got[0]["iter"] == got[1]["iter"]
    for key in ("eigs", "res", "x"):
        np.testing.assert_array_equal(got[0][key], got[1][key])


def test_batch_of_problems_with_grid_barriers(gpu):
    """Problems of 13,824 to 21,952 rows, whose inner iterations are launches
    with a grid barrier, from eight worker streams at once: every one gets its
    closed-form eigenvalues (a residual of TOL bounds their distance)."""
    tol = 1e-9
    problems, exact = [], []
    for k in range(16):
        m = 24 + k % 5
        ia, ja, a = M.laplace3d(m)
        s = 1.0 + 0.1 * k
        problems.append((s * a, ja, ia))
        exact.append(s * M.laplace3d_eigenvalues(m, 4))
    for r, w in zip(gpu.dpjd_batch(problems, 4, workers=8, isearch=0, tol=tol, icntl=(0, 0, 0, 0, 0)), exact):
        assert r["info"] == 0 and r["neig"] == 4
        assert np.max(np.abs(np.sort(r["eigs"]) - w)) <= tol + 64 * np.finfo(float).eps * 12 * 2.5


@pytest.mark.parametrize("n", [4096, 8193, 77825])
@pytest.mark.parametrize("kind,isearch", [("real", 2), ("complex generalized", 2)])
def test_most_columns(gpu, n, kind, isearch):
    """32 pairs, the most that the drivers sort: up to 32 columns in a projection."""
    A, B = _problem(kind, n)
    got = []
    for fuse in (1, 0):
        gpu.set_option("fuse_inner", fuse)
        try:
            kw = dict(isearch=isearch, sigma=0.0, madspace=20, maxit=20000, tol=1e-9, droptol=1e-3,
                      icntl=(0, 1, 0, 0, 0))
            r = gpu.dpjd(A, 32, **kw) if B is None else gpu.zpjd_gep(A, B, 32, **kw)
        finally:
            gpu.set_option("fuse_inner", 1)
        assert r["info"] == 0 and r["neig"] == 32
        got.append(r)
    assert got[0]["iter"] == got[1]["iter"]
    for key in ("eigs", "res", "x"):
        np.testing.assert_array_equal(got[0][key], got[1][key])
