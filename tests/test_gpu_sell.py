"""The full matrix built on the device from the caller's triangle, where it
can go wrong: slices of one row, full slices and a remainder, either triangle
or a mixture, unsorted rows, and rows with more transposed entries (64) than
the device build takes (the host pass).  A product against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _triangle(n, kind, hub, cplx, seed):
    """Random Hermitian A and its stored half: each pair (i, j) once, in row i
    or j as `kind` says, the entries of a row in random order."""
    rng = np.random.default_rng(seed)
    pairs = {(i, i) for i in range(n)}
    for i in range(n):
        for j in rng.integers(0, n, 3):
            pairs.add((min(i, j), max(i, j)))
        if hub:
            pairs.add((0, i))
    A = np.zeros((n, n), complex if cplx else float)
    rows = [[] for _ in range(n)]
    for i, j in sorted(pairs):
        v = rng.standard_normal() + (1j * rng.standard_normal() if cplx and i != j else 0)
        A[i, j], A[j, i] = v, np.conj(v)
        low = kind == "lower" or (kind == "mixed" and rng.random() < 0.5)
        rows[j if low else i].append((i if low else j))
    ia, ja, a = [1], [], []
    for i, r in enumerate(rows):
        rng.shuffle(r)
        ja += [j + 1 for j in r]
        a += [A[i, j] for j in r]
        ia.append(len(ja) + 1)
    return A, (np.array(a), np.array(ja, np.int32), np.array(ia, np.int32))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 200])
@pytest.mark.parametrize("kind", ["upper", "lower", "mixed"])
@pytest.mark.parametrize("hub", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
def test_product_with_any_triangle(gpu, n, kind, hub, cplx):
    A, stored = _triangle(n, kind, hub, cplx, n)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)
    # each row sum has at most n + 4 terms: (n + 4) eps times the sum of their sizes, twice for complex products
    bound = 2 * (n + 4) * np.finfo(float).eps * (np.abs(A) @ np.abs(x))
    assert np.all(np.abs(gpu.spmv(stored, x) - A @ x) <= bound + 1e-300)


def test_out_of_range_column_is_refused(gpu):
    a, ja, ia = np.ones(3), np.array([1, 7, 2], np.int32), np.array([1, 3, 4], np.int32)
    with pytest.raises(RuntimeError):
        gpu.spmv((a, ja, ia), np.ones(2))
