"""A matrix prepared on the device for several solves: what becomes of it when
a later one is refused."""
import ctypes as C

import numpy as np
import pytest

from jadamilu_gb300 import matrices as M

pytestmark = pytest.mark.gpu

KW = dict(isearch=0, madspace=20, maxit=2000, tol=1e-10, droptol=1e-3, icntl=(0, 1, 0, 0, 0))


def _rows_held(gpu):
    out = np.zeros(3, np.int64)
    gpu.load().jdgpu_dmatrix_info(out.ctypes.data_as(C.c_void_p))
    return int(out[2])


@pytest.mark.parametrize("bad", [0, 1 << 30])
def test_refused_matrix_is_not_used(gpu, bad):
    """A refused matrix (a column out of range) of another row structure must
    not leave its slice pointers to solves with the one prepared before."""
    ia, ja, a = M.laplace3d(12)
    plain = gpu.dpjd((a.copy(), ja.copy(), ia), 3, **KW)
    assert plain["info"] == 0
    n = len(ia) - 1
    ib = np.arange(1, 40 * n + 2, 40, dtype=np.int32)  # 40 entries per row
    jb = (np.arange(40 * n) % n + 1).astype(np.int32)
    jb[-1] = bad
    try:
        gpu.prepare_matrix((a, ja, ia))
        assert _rows_held(gpu) == n
        with pytest.raises(RuntimeError):
            gpu.prepare_matrix((np.ones(40 * n), jb, ib))
        assert _rows_held(gpu) == 0
        r = gpu.dpjd((a.copy(), ja.copy(), ia), 3, **KW)
    finally:
        gpu.release_matrix()
    assert r["info"] == 0 and r["x"].shape == (n, 3)
    np.testing.assert_array_equal(r["eigs"], plain["eigs"])
    np.testing.assert_array_equal(r["x"], plain["x"])


def test_stream_replaced_between_prepare_and_solve(gpu):
    """The stream changes after the hand-over, after a solve and after one that
    ends by an error (more basis vectors than a restart takes), each time with
    work just done on the stream that goes; a kept factor leaves little host work
    in between."""
    torch = pytest.importorskip("torch")
    ia, ja, a = M.laplace3d(24)
    kept = dict(KW, icntl=(0, -1, 0, 0, 0))
    plain = gpu.dpjd((a.copy(), ja.copy(), ia), 3, **KW)
    assert plain["info"] == 0
    streams = [torch.cuda.Stream() for _ in range(2)]
    try:
        for k in range(6):
            gpu.release_matrix()
            r = gpu.dpjd((a.copy(), ja.copy(), ia), 3, **dict(kept, madspace=40))
            assert r["info"] == -54330
            gpu.set_stream(streams[k % 2].cuda_stream)
            gpu.prepare_matrix((a, ja, ia))
            gpu.set_stream(streams[(k + 1) % 2].cuda_stream if k % 3 else 0)
            r = gpu.dpjd((a.copy(), ja.copy(), ia), 3, **kept)
            assert r["info"] == 0
            np.testing.assert_array_equal(r["eigs"], plain["eigs"])
    finally:
        gpu.set_stream(0)
        gpu.release_matrix()


def test_generalized_solves_with_a_prepared_matrix(gpu):
    """Only A is prepared: every generalized solve hands its own B over, after
    one of a smaller size and after one with another B."""
    def pencil(m, seed):
        K, B = M.fem_p1(m, seed=seed)
        return (K[2], K[1], K[0]), (B[2], B[1], B[0])

    small = pencil(20, 3)
    A, B = pencil(100, 3)
    B2 = (2.0 * B[0], B[1], B[2])
    plain = [gpu.dpjd_gep(A, Bk, 3, **KW)["eigs"] for Bk in (B, B2)]
    assert gpu.dpjd_gep(*small, 3, **KW)["info"] == 0
    try:
        gpu.prepare_matrix(A)
        for Bk, w in zip((B, B2), plain):
            r = gpu.dpjd_gep(A, Bk, 3, **KW)
            assert r["info"] == 0
            np.testing.assert_array_equal(r["eigs"], w)
    finally:
        gpu.release_matrix()


def test_solve_of_another_size_is_refused(gpu):
    ia, ja, a = M.laplace3d(12)
    try:
        gpu.prepare_matrix((a, ja, ia))
        for m in (10, 14):
            ib, jb, b = M.laplace3d(m)
            assert gpu.dpjd((b, jb, ib), 3, **KW)["info"] == -54330
        assert gpu.dpjd((a, ja, ia), 3, **KW)["info"] == 0
    finally:
        gpu.release_matrix()
