"""The full matrix around the size from which it is built on the device (4096
stored entries; the host pass below), with full slices, a remainder of one and
of 31 rows, either triangle or a mixture, unsorted rows, and a row of more
transposed entries than the device takes.  A product against scipy."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _triangle(n, nnz, kind, hub, cplx):
    """Hermitian A and its stored half, `nnz` entries: the diagonal, with `hub` the pairs of unknown 0, and random pairs,
    each stored once in the row that `kind` says, rows in random order."""
    rng = np.random.default_rng(n + nnz)
    i = np.arange(1, n if hub else 1)
    pairs = set(zip(np.zeros_like(i).tolist(), i.tolist()))
    while len(pairs) < nnz - n:
        p, q = sorted(rng.integers(0, n, 2).tolist())
        if p < q:
            pairs.add((p, q))
    p, q = np.array(sorted(pairs)).T
    low = np.full(len(p), kind == "lower") if kind != "mixed" else rng.random(len(p)) < 0.5
    row = np.concatenate([np.arange(n), np.where(low, q, p)])
    col = np.concatenate([np.arange(n), np.where(low, p, q)])
    v = rng.standard_normal(nnz) + (1j * rng.standard_normal(nnz) * (row != col) if cplx else 0)
    S = sp.coo_matrix((v, (row, col)), shape=(n, n)).tocsr()
    A = S + S.conj().T - sp.diags(S.diagonal())
    order = np.lexsort((rng.random(nnz), row))
    ia = np.searchsorted(row[order], np.arange(n + 1)) + 1
    return A, (v[order], (col[order] + 1).astype(np.int32), ia.astype(np.int32))


@pytest.mark.parametrize("n,nnz", [(1344, 4095), (1344, 4096), (1344, 4097), (2047, 8000), (2048, 8000), (2049, 8000),
                                   (3000, 4097)])
@pytest.mark.parametrize("kind", ["upper", "lower", "mixed"])
@pytest.mark.parametrize("hub", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
def test_product(gpu, n, nnz, kind, hub, cplx):
    if hub and nnz < 2 * n:
        pytest.skip("fewer entries than the hub row has")
    A, stored = _triangle(n, nnz, kind, hub, cplx)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)
    # each row sum has at most n + 4 terms: (n + 4) eps times the sum of their sizes, twice for complex products
    bound = 2 * (n + 4) * np.finfo(float).eps * (abs(A) @ np.abs(x))
    assert np.all(np.abs(gpu.spmv(stored, x) - A @ x) <= bound + 1e-300)


@pytest.mark.parametrize("n", [100, 3000])
@pytest.mark.parametrize("where", ["pointer beyond", "pointer decreasing", "column 0", "column n + 1"])
def test_same_refusals_on_both_sides(gpu, n, where):
    A, (a, ja, ia) = _triangle(n, 3 * n, "upper", False, False)
    if where.startswith("pointer"):
        ia[n // 2] = ia[n] + 5 if where.endswith("beyond") else ia[n // 2 - 1] - 1
    else:
        ja[-1] = 0 if where.endswith("0") else n + 1
    with pytest.raises(RuntimeError):
        gpu.spmv((a, ja, ia), np.ones(n))
