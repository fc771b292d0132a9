"""Device memory that stays with the solver after a large matrix, in a process
of its own (the workspaces of earlier solves would hide it)."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
sys.path[:0] = sys.argv[1:]
import torch
import jadamilu_gb300 as J
from jadamilu_gb300 import matrices as M

def held():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

def prepare(n):
    ia, ja, a = M.tridiag(n)
    J.prepare_matrix((a, ja, ia))

N = 3000000
prepare(1000)
start = held()
prepare(N)
# the workspace: one vector and 32 columns of scratch; the matrix: three slots of 12 bytes per row, slice pointers
work, matrix = N * 8 * 33, N * 36 + N // 4
mid = held()
print(start - mid - work - matrix)
prepare(1000)
print(start - held() - work)
J.dpjdcleanup()
J.release_matrix()
print(start - held() - work)
"""


def test_memory_kept_is_bounded(gpu):
    """At most 32 MB beyond the matrix itself (the triangle alone is 108 MB here), none after the clean-up call; 8
    MB more for the allocator's granularity and the reductions' partial sums."""
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CHILD, *sys.path[:2]], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    large, small, cleaned = (int(v) for v in r.stdout.split())
    assert large <= (32 + 8) << 20 and small <= (2 * 32 + 8) << 20 and cleaned <= 8 << 20
