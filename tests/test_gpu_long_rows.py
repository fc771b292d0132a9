"""Preconditioner rows longer than one batch of the kernel that runs narrow
levels: an arrow matrix, whose last row of L holds every other unknown and is a
level of its own.  The factor is exact, and the numbers are chosen so that
nothing in the sums rounds, so one entry left out of thousands shows in every
storage precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# relative rounding of a stored factor entry: float64, float32, bfloat16
STORE = {0: 2.0 ** -52, 1: 2.0 ** -23, 2: 2.0 ** -8}


@pytest.mark.parametrize("hub", [1023, 1024, 1025, 4095, 4096, 4097, 9999, 16384])
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("graph", [0, 1])
def test_arrow_matrix(gpu, hub, precision, graph):
    """A = [4 I, e/2; e^T/2, d]: L's last row is e^T/8, D = diag(4, d - hub/16).
    With integer b and b_last = 1 + sum(b)/8 the forward sweep gives exactly 1
    in the last place, the backward sweep x_last = 1/(d - hub/16) and
    x_i = b_i/4 - x_last/8: each is a few products of stored entries."""
    n, d = hub + 1, 20000.0
    ia = np.append(np.arange(hub + 1) * 2 + 1, 2 * hub + 2).astype(np.int32)
    ja = np.empty(2 * hub + 1, np.int32)
    a = np.empty(2 * hub + 1)
    ja[0:-1:2], ja[1:-1:2], ja[-1] = np.arange(1, n), n, n
    a[0:-1:2], a[1:-1:2], a[-1] = 4.0, 0.5, d
    b = np.random.default_rng(hub).integers(-3, 4, n).astype(float)
    b[-1] = 1 + b[:-1].sum() / 8
    last = 1 / (d - hub / 16)
    exact = np.append(b[:-1] / 4 - last / 8, last)
    try:
        gpu.set_option("coupled_min_n", 1 << 30)  # the plain form at every size
        gpu.set_option("apply_graph", graph)
        x, info = gpu.ildl_apply((a, ja, ia), b, shift=0.0, droptol=1e-3, spd=False, precision=precision)
    finally:
        gpu.set_option("coupled_min_n", 4096)
        gpu.set_option("apply_graph", 0)
    assert info["nnz_l"] == hub and info["fwd_depth"] == 2
    # D^-1 and L are stored with one rounding each, and at most six more follow in products and sums
    assert np.all(np.abs(x - exact) <= 8 * STORE[precision] * (np.abs(b) / 4 * (np.arange(n) < hub) + last))
