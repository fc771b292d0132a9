"""Hand-over of matrices with one row at and beyond the 4096 stored entries
that the device build takes (the host pass beyond): a product against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stored", [4095, 4096, 4097, 5000])
@pytest.mark.parametrize("row", ["first", "last"])
@pytest.mark.parametrize("cplx", [False, True])
def test_row_of_many_stored_entries(gpu, stored, row, cplx):
    n = 6000
    rng = np.random.default_rng(stored)
    hub = 0 if row == "first" else n - 1
    cols = np.sort(rng.choice(np.setdiff1d(np.arange(n), [hub]), stored - 1, replace=False))
    ja = [[i] for i in range(n)]
    ja[hub] = [hub, *cols]
    ia = np.cumsum([1] + [len(r) for r in ja]).astype(np.int32)
    ja = (np.concatenate(ja) + 1).astype(np.int32)
    a = rng.standard_normal(len(ja)) + (1j * rng.standard_normal(len(ja)) if cplx else 0)
    own = ja - 1 == np.repeat(np.arange(n), np.diff(ia))
    a[own] = a[own].real
    x = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)
    off = a[~own]
    y = a[own] * x
    size = np.abs(y)
    y[hub] += off @ x[cols]
    size[hub] += np.abs(off) @ np.abs(x[cols])
    y[cols] += np.conj(off) * x[hub]
    size[cols] += np.abs(off) * np.abs(x[hub])
    # a row has at most `stored` terms: that many times eps, twice for complex products and for the two sums
    assert np.all(np.abs(gpu.spmv((a, ja, ia), x) - y) <= 4 * (stored + 4) * np.finfo(float).eps * size + 1e-300)


@pytest.mark.parametrize("bad", [0, -5, 6001, 1 << 30])
@pytest.mark.parametrize("at", [1, 4999])
def test_bad_column_in_a_long_row_is_refused(gpu, bad, at):
    n, stored = 6000, 5000
    ja = np.concatenate([np.arange(1, stored + 1), np.arange(2, n + 1)]).astype(np.int32)
    ja[at] = bad
    ia = np.concatenate([[1], np.arange(stored + 1, stored + n + 1)]).astype(np.int32)
    with pytest.raises(RuntimeError):
        gpu.spmv((np.ones(len(ja)), ja, ia), np.ones(n))
