"""Eigenvalue gradients where the kernels change shape: column counts around
the 8 a thread carries and the 8 / 16 / 64 held in registers, eigenvectors
stored by column, by row and non-contiguously, with and without B."""
import numpy as np
import pytest

from jadamilu_gb300 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 64])
@pytest.mark.parametrize("layout", ["columns", "rows", "strided"])
@pytest.mark.parametrize("with_b", [False, True])
def test_layouts_and_column_counts(gpu, k, layout, with_b):
    K, Mm = M.fem_p1(20, seed=3)
    ia, ja, a = K
    n = len(ia) - 1
    rng = np.random.default_rng(k)
    X = rng.standard_normal((n, k))
    w = rng.uniform(0.5, 1.5, k)
    md = Mm[2] if with_b else np.ones(n)
    rows, cols = np.repeat(np.arange(n), np.diff(ia)), np.asarray(ja) - 1
    c = w / np.einsum("nk,n,nk->k", X, md, X)
    terms = c * X[rows] * X[cols]
    scale = np.where(rows == cols, 1.0, 2.0)
    given = {"columns": np.asfortranarray(X), "rows": X, "strided": np.repeat(X, 2, axis=1)[:, ::2]}[layout]
    g = gpu.eig_grad((a, ja, ia), given, w=w, bdiag=md if with_b else None)
    # the norms are sums of n positive terms (n eps relative each), then k products of three factors are added
    bound = (2 * n + k + 8) * np.finfo(float).eps * np.abs(terms).sum(1) * scale
    assert np.all(np.abs(g - terms.sum(1) * scale) <= bound)
