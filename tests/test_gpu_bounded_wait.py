"""The bounded grid barrier of the inner iteration: when its polls run out the
kernel returns, the solve ends with INFO = -54330, and nothing of that stays."""
import numpy as np
import pytest

from jadamilu_gb300 import matrices as M

pytestmark = pytest.mark.gpu

KW = dict(isearch=0, madspace=20, maxit=2000, tol=1e-9, droptol=1e-3, icntl=(0, 1, 0, 0, 0))


def _laplace(m, cplx):
    ia, ja, a = M.laplace3d(m)
    return (a.astype(complex) if cplx else a), ja, ia


# one CTA per SM up to 77,824 rows, four of the reduction's CTAs in each beyond
@pytest.mark.parametrize("m", [22, 43])
@pytest.mark.parametrize("cplx", [False, True])
def test_polls_run_out(gpu, m, cplx):
    A = _laplace(m, cplx)
    solve = gpu.zpjd if cplx else gpu.dpjd
    good = solve(A, 2, **KW)
    assert good["info"] == 0
    for _ in range(2):
        try:
            gpu.set_option("barrier_polls", 0)
            assert solve(A, 2, **KW)["info"] == -54330
        finally:
            gpu.set_option("barrier_polls", 1 << 22)
        r = solve(A, 2, **KW)
        assert r["info"] == 0
        np.testing.assert_array_equal(r["eigs"], good["eigs"])
        np.testing.assert_array_equal(r["x"], good["x"])


def test_other_arithmetic_is_not_blamed(gpu):
    """A complex solve after a real one whose polls ran out."""
    A, Az = _laplace(22, False), _laplace(22, True)
    try:
        gpu.set_option("barrier_polls", 0)
        assert gpu.dpjd(A, 2, **KW)["info"] == -54330
    finally:
        gpu.set_option("barrier_polls", 1 << 22)
    assert gpu.zpjd(Az, 2, **KW)["info"] == 0
