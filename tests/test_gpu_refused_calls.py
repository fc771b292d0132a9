"""A refused matrix (a column out of range in its last entry) costs no device
memory, however often it is handed over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1000000  # slice pointers of 250 KB
CALLS = 64


def _bad(n, dtype):
    ia = np.arange(1, n + 2, dtype=np.int32)
    ja = np.arange(1, n + 1, dtype=np.int32)
    ja[-1] = n + 1
    return np.ones(n, dtype), ja, ia


@pytest.mark.parametrize("entry", ["dspmv", "zspmv", "eigvec_grad"])
def test_memory_after_refusals(gpu, entry):
    torch = pytest.importorskip("torch")
    A = _bad(N, np.complex128 if entry == "zspmv" else np.float64)
    x = np.ones(N, A[0].dtype)

    def call():
        with pytest.raises(RuntimeError):
            if entry == "eigvec_grad":
                gpu.eigvec_grad(A, 1.0, x, x)
            else:
                gpu.spmv(A, x)

    call()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(CALLS):
        call()
    assert before - torch.cuda.mem_get_info()[0] < 8 << 20  # kept, the slice pointers alone are 16 MB
