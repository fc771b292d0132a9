"""Generalized problems handed over one after another: the products with B
must read the B of their own call.  Bilinear elements on the unit square give
a B with nine entries per row and eigenvalues in closed form; the GPU is kept
busy by another stream, so that the host runs ahead of the solver's kernels."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

M1 = 140  # unknowns per side: n = 19600
NEIG = 4
TOL = 1e-10


def _pencil(cx, cy, cb, phase):
    """(A, B) = (cx K x M + cy M x K, cb M x M) of the 1-D stiffness K and mass
    M, both turned by a diagonal unitary with `phase`, as upper triangles; and
    the smallest eigenvalues (cx l_i + cy l_j) / cb."""
    e = np.ones(M1)
    K = sp.diags([-e[1:], 2 * e, -e[1:]], [-1, 0, 1])
    Mm = sp.diags([e[1:] / 6, 4 * e / 6, e[1:] / 6], [-1, 0, 1])
    out = []
    for S in (cx * sp.kron(K, Mm) + cy * sp.kron(Mm, K), cb * sp.kron(Mm, Mm)):
        S = sp.csr_matrix(S)
        if phase:
            d = sp.diags(np.exp(1j * phase * np.arange(M1 * M1)))
            S = sp.csr_matrix(d @ S @ d.conj())
            S.setdiag(S.diagonal().real)
        U = sp.csr_matrix(sp.triu(S))
        U.sort_indices()
        out.append((U.data, U.indices.astype(np.int32) + 1, U.indptr.astype(np.int32) + 1))
    t = np.arange(1, M1 + 1) * np.pi / (M1 + 1)
    lam = 6 * (2 - 2 * np.cos(t)) / (4 + 2 * np.cos(t))
    w = np.sort(((cx * lam[:, None] + cy * lam[None, :]) / cb).ravel())[:NEIG]
    return out[0], out[1], w


@pytest.mark.parametrize("cplx", [False, True])
def test_solves_in_turn(gpu, cplx):
    """The residual is at most TOL |B u|, so an eigenvalue is within TOL
    sqrt(cond B) = 3 TOL (M's eigenvalues lie in [1/3, 1]) of one of the
    pencil, and the rounding of both sides is bounded by 64 eps |A| |B^-1|."""
    torch = pytest.importorskip("torch")
    phase = 0.3 if cplx else 0.0
    problems = [_pencil(1.0, 1.3, 1.0, phase), _pencil(1.7, 0.9, 3.0, phase)]
    solve = gpu.zpjd_gep if cplx else gpu.dpjd_gep
    kw = dict(isearch=0, madspace=20, maxit=4000, tol=TOL, droptol=1e-3)
    A, B, _ = problems[0]
    first = solve(A, B, NEIG, icntl=(0, 1, 0, 0, 0), **kw)
    assert first["info"] == 0
    side = torch.cuda.Stream()
    busy = torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    seen = {}
    for k in range(8):
        A, B, w = problems[k % 2]
        with torch.cuda.stream(side):
            for _ in range(4):
                torch.mm(busy, busy)
        r = solve(A, B, NEIG, icntl=(0, -1, 0, 0, 0), **kw)
        assert r["info"] == 0 and r["neig"] == NEIG
        norm = 8.0 * 9.0 / (3.0 if k % 2 else 1.0) * 1.3
        assert np.max(np.abs(np.sort(r["eigs"]) - w)) <= 3 * TOL + 64 * np.finfo(float).eps * norm
        if k % 2 in seen:
            np.testing.assert_array_equal(r["eigs"], seen[k % 2]["eigs"])
            np.testing.assert_array_equal(r["x"], seen[k % 2]["x"])
        else:
            seen[k % 2] = r
    torch.cuda.synchronize()
