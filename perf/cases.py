"""The eigensolver's workloads as timed cases, through its public Python entry points.

Kinds of case:

* ``solve``: one complete DPJD / ZPJD / DPJD_GEP call on host arrays with a kept preconditioner
  (ICNTL(2) = -1), the way a sweep over slowly changing matrices runs: the program factors a base matrix
  once and solves each perturbed matrix of the sweep with that factor.  The factor is the program's handle;
  the library keeps one per arithmetic and process, and so does this file (``_keep``).
* ``whole``: DPJD from scratch, factorisation included (ICNTL(2) = 1), on a matrix small enough for that.
* ``revcom``: DPJDREVCOM in device mode, the matvec served by the caller's own GPU operator.
* ``spmv``: one product with a matrix handed over by the caller.
* ``eig_grad`` / ``eigvec_grad``: the two backward entry points.

The batched entry point is not listed: its refactorisation decisions follow the wall clock, so two runs of the
same batch differ.  Its problems (Anderson lattices of edge 16 to 40) are here as single solves.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import jadamilu_gb300 as J
from jadamilu_gb300 import matrices as M

# Solver settings of each matrix family: those of bench.py's workloads.
SETTINGS = {
    "anderson": dict(isearch=2, sigma=0.0, madspace=25, droptol=1e-3, mem=20.0),
    "laplace": dict(isearch=0, sigma=0.0, madspace=20, droptol=1e-3, mem=20.0),
    "tight_binding": dict(isearch=0, sigma=0.0, madspace=20, droptol=1e-3, mem=20.0),
    "fem": dict(isearch=0, sigma=0.0, madspace=20, droptol=1e-3, mem=20.0),
    "tridiag": dict(isearch=2, sigma=0.0, madspace=20, droptol=1e-3, mem=20.0),
}
# Measured averages behind work(): MATVECs per eigenpair at the first size and their growth with n, entries of L
# per row.
EFFORT = {
    "anderson": (20.0, 4096, 0.19, 65.0),
    "laplace": (27.0, 8000, 0.2, 25.0),
    "tight_binding": (120.0, 262144, 0.2, 12.0),
    "fem": (89.0, 260100, 0.2, 12.0),
    "tridiag": (15.0, 1000, 0.0, 2.0),
}


def listed():
    return [
        # The user guide's first sample: a latency-bound call on 1000 unknowns, the factorisation included.
        dict(name="tridiag_1000", kind="whole", family="tridiag", size=1000, neig=5, precision=0),
        # The Laplacian configuration: ten smallest, plain float64, positive definite preconditioner.
        dict(name="laplace_20", kind="solve", family="laplace", size=20, neig=10, precision=0),
        # The smallest problem of the batched configuration (five interior pairs, single-precision factor).
        dict(name="anderson_16", kind="solve", family="anderson", size=16, neig=5, precision=1),
        # An odd lattice in the middle of that range, with the bfloat16 factor.
        dict(name="anderson_25_bf16", kind="solve", family="anderson", size=25, neig=5, precision=2),
        # The largest problem of the batched configuration.
        dict(name="anderson_40", kind="solve", family="anderson", size=40, neig=5, precision=1),
        # The headline: 10 interior pairs at n = 1e6.
        dict(name="anderson_100", kind="solve", family="anderson", size=100, neig=10, precision=1),
        # The complex Hermitian configuration, complex64 factor.
        dict(name="tight_binding_64", kind="solve", family="tight_binding", size=64, neig=8, precision=1),
        # The generalized configuration, float64 throughout.
        dict(name="fem_512", kind="solve", family="fem", size=512, neig=6, precision=0),
        # A matrix-free user operator on the GPU behind device-pointer reverse communication.
        dict(name="revcom_24", kind="revcom", family="anderson", size=24, neig=5, precision=1),
        # A caller's own product with the built-in matvec: hand-over of the matrix and one product.
        dict(name="spmv_50", kind="spmv", family="anderson", size=50),
        # The differentiation configuration: gradient of the sum of the 6 smallest eigenvalues.
        dict(name="eig_grad_512", kind="eig_grad", family="fem", size=512, neig=6),
        # Gradient of an eigenvector loss: factorisation and adjoint solve.
        dict(name="eigvec_grad_48", kind="eigvec_grad", family="fem", size=48, neig=3),
    ]


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["whole", "laplace", "anderson", "anderson", "tight_binding", "fem", "revcom", "spmv",
                       "eig_grad", "eigvec_grad"])
    if what == "whole":
        return dict(kind="whole", family="tridiag", size=edge(300, 3000), neig=rng.randint(1, 8),
                    precision=rng.choice([0, 0, 1]))
    if what == "laplace":
        return dict(kind="solve", family="laplace", size=edge(10, 32), neig=rng.randint(1, 10),
                    precision=rng.choice([0, 0, 1]))
    if what == "anderson":
        return dict(kind="solve", family="anderson", size=edge(12, 100), neig=rng.randint(1, 10),
                    precision=rng.choice([0, 1, 1, 2]))
    if what == "tight_binding":
        return dict(kind="solve", family="tight_binding", size=edge(12, 64), neig=rng.randint(1, 8),
                    precision=rng.choice([0, 1]))
    if what == "fem":
        return dict(kind="solve", family="fem", size=edge(32, 512), neig=rng.randint(1, 6),
                    precision=rng.choice([0, 0, 1]))
    if what == "revcom":
        return dict(kind="revcom", family="anderson", size=edge(12, 40), neig=rng.randint(1, 5), precision=1)
    if what == "spmv":
        return dict(kind="spmv", family=rng.choice(["anderson", "tight_binding", "fem"]), size=edge(12, 100))
    if what == "eig_grad":
        return dict(kind="eig_grad", family="fem", size=edge(16, 512), neig=rng.randint(1, 12))
    return dict(kind="eigvec_grad", family="fem", size=edge(16, 60), neig=rng.randint(1, 4))


# ------------------------------------------------------------------ matrices
_base = {}  # the last base matrix: generating one takes longer than perturbing it


def _matrix(family, size):
    """(A, B) as (a, ja, ia) triples; B is None but for the FEM pencil."""
    key = (family, size)
    if key not in _base:
        _base.clear()
        B = None
        if family == "fem":
            A, B = M.fem_p1(size, sigma=0.5, seed=3)
        elif family == "tight_binding":
            A = M.tight_binding3d(size, phi=1.0 / 17.0, disorder=4.0, seed=1)
        elif family == "anderson":
            A = M.anderson3d(size, disorder=16.5, seed=0)
        elif family == "laplace":
            A = M.laplace3d(size)
        else:
            A = M.tridiag(size)
        _base[key] = (A, B)
    A, B = _base[key]
    turn = lambda t: None if t is None else (t[2], t[1], t[0])
    return turn(A), turn(B)


def _perturbed(A, seed, step):
    """A with its diagonal moved by up to `step` of the mean absolute diagonal (the diagonal leads each row)."""
    a, ja, ia = A
    at = np.asarray(ia[:-1], np.int64) - 1
    rng = np.random.default_rng(seed)
    a = a.copy()
    a[at] += step * np.abs(a[at]).mean() * rng.uniform(-1.0, 1.0, len(at))
    return a, ja.copy(), ia.copy()


# ------------------------------------------------------------- kept factors
_kept = {}  # arithmetic -> the case whose factor the library holds


def _key(case):
    return (case["family"], case["size"], case["precision"])


def _keep(case, A, B):
    """Factors the base matrix (one MATVEC of budget: the call ends once the factor is there)."""
    arith = "z" if case["family"] == "tight_binding" else "d"
    if _kept.get(arith) != _key(case):
        _kept[arith] = None
        A = (A[0].copy(), A[1].copy(), A[2].copy())
        _call(case, A, B, dict(SETTINGS[case["family"]], maxit=1, tol=1e-10, icntl=(0, 0, 0, 0, case["precision"])))
        _kept[arith] = _key(case)


def _call(case, A, B, kw):
    if B is not None:
        return J.dpjd_gep(A, B, case["neig"], **kw)
    return (J.zpjd if case["family"] == "tight_binding" else J.dpjd)(A, case["neig"], **kw)


# --------------------------------------------------------------- revcom operator
class _DeviceVector:
    def __init__(self, address, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(address, False), version=3)


class _Lattice:
    """The periodic Anderson Hamiltonian as a gather over the six neighbours and the site itself."""

    def __init__(self, m, diag):
        i = np.arange(m ** 3)
        x, y, z = i % m, (i // m) % m, i // (m * m)
        nb = [i]
        for s in (1, m - 1):
            nb += [(x + s) % m + m * y + m * m * z, x + m * ((y + s) % m) + m * m * z,
                   x + m * y + m * m * ((z + s) % m)]
        self.col = torch.tensor(np.stack(nb, 1), device="cuda")
        val = np.full((m ** 3, 7), -1.0)
        val[:, 0] = diag
        self.val = torch.tensor(val, device="cuda")
        self.streams = {}

    def __call__(self, x, y, n, stream):
        if stream not in self.streams:
            self.streams[stream] = torch.cuda.ExternalStream(stream)
        with torch.cuda.stream(self.streams[stream]):
            xv, yv = (torch.as_tensor(_DeviceVector(p, n), device="cuda") for p in (x, y))
            torch.sum(self.val * xv[self.col], 1, out=yv)


# ------------------------------------------------------------------ the cases
def _pencil_pair(A, B, index):
    """Eigenpair `index` of a small FEM pencil (dense, in 64 bits)."""
    K, md = _dense(A), torch.tensor(B[0], device="cuda")
    s = 1.0 / torch.sqrt(md)
    w, V = torch.linalg.eigh(s[:, None] * K * s[None, :])
    x = s * V[:, index]
    return float(w[index]), x * torch.sign(x[torch.argmax(torch.abs(x))])


def _dense(A):
    a, ja, ia = A
    n = len(ia) - 1
    r = torch.tensor(np.repeat(np.arange(n), np.diff(ia)), device="cuda")
    c = torch.tensor(np.asarray(ja, np.int64) - 1, device="cuda")
    v = torch.tensor(a, device="cuda")
    D = torch.zeros((n, n), dtype=v.dtype, device="cuda")
    D[c, r] = v.conj()
    D[r, c] = v
    return D


def prepare(case, seed):
    kind, family = case["kind"], case["family"]
    A, B = _matrix(family, case["size"])
    s = dict(case=case)
    rng = np.random.default_rng(seed + 1)
    n = len(A[2]) - 1
    if kind in ("solve", "revcom"):
        _keep(case, A, B)
        s["A"], s["B"] = _perturbed(A, seed, 1e-5), B
        s["kw"] = dict(SETTINGS[family], maxit=100000, tol=1e-10, icntl=(0, -1, 0, 0, case["precision"]))
        if kind == "revcom":
            s["op"] = _Lattice(case["size"], s["A"][0][np.asarray(s["A"][2][:-1]) - 1])
    elif kind == "whole":
        _kept["d"] = None
        s["A"], s["B"] = _perturbed(A, seed, 1e-3), B
        s["kw"] = dict(SETTINGS[family], maxit=100000, tol=1e-10, icntl=(0, 1, 0, 0, case["precision"]))
    elif kind == "spmv":
        s["A"] = _perturbed(A, seed, 1e-2)
        s["x"] = rng.standard_normal(n)
        if family == "tight_binding":
            s["x"] = s["x"] + 1j * rng.standard_normal(n)
    elif kind == "eig_grad":
        # the modes of the unit square with noise: shaped like eigenvectors, and the formula holds for any X
        m = case["size"] - 2
        t = np.pi * np.arange(1, m + 1) / (m + 1)
        modes = sorted(((i * i + j * j, i, j) for i in range(1, 6) for j in range(1, 6)))[:case["neig"]]
        s["A"], s["B"] = _perturbed(A, seed, 1e-3), B
        s["X"] = np.stack([np.outer(np.sin(i * t), np.sin(j * t)).ravel() for _, i, j in modes], 1)
        s["X"] += 0.1 * rng.standard_normal(s["X"].shape)
        s["w"] = rng.uniform(0.5, 1.5, case["neig"])
    else:
        s["A"], s["B"] = _perturbed(A, seed, 1e-3), B
        lam, x = _pencil_pair(s["A"], B, case["neig"] - 1)
        s["lam"], s["x"], s["g"] = lam, x.cpu().numpy(), rng.standard_normal(n)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("solve", "whole"):
        if kind == "solve" and _kept.get("z" if case["family"] == "tight_binding" else "d") != _key(case):
            raise RuntimeError("another case's factor is kept")
        r = _call(case, s["A"], s["B"], s["kw"])
        return {"eigs": r["eigs"], "x": r["x"], "neig": r["neig"], "info": r["info"]}
    if kind == "revcom":
        r = J.dpjdrevcom(s["A"], case["neig"], s["op"], device=True, **s["kw"])
        return {"eigs": r["eigs"], "x": r["x"], "neig": r["neig"], "info": r["info"]}
    if kind == "spmv":
        return J.spmv(s["A"], s["x"])
    if kind == "eig_grad":
        return J.eig_grad(s["A"], s["X"], w=s["w"], bdiag=s["B"][0])
    # the iteration count and residual that come with it are diagnostics
    return J.eigvec_grad(s["A"], s["lam"], s["x"], s["g"], bdiag=s["B"][0])[0]


def _sizes(case):
    """(unknowns, stored entries of one triangle)."""
    m, family = case["size"], case["family"]
    if family == "fem":
        return (m - 2) ** 2, (m - 2) ** 2 + 3 * (m - 2) * (m - 3) - (m - 3)
    if family == "tridiag":
        return m, 2 * m - 1
    return m ** 3, m ** 3 + 3 * m * m * (m if family == "anderson" else m - 1)


def work(case):
    kind, family = case["kind"], case["family"]
    n, nnz = _sizes(case)
    val = 16 if family == "tight_binding" else 8
    if kind == "spmv":
        return {"bytes": nnz * (val + 4) + 4 * n + 2 * n * val, "flops": 4 * nnz * (4 if val == 16 else 1)}
    if kind == "eig_grad":
        k = case["neig"]
        return {"bytes": nnz * 12 + 4 * n + n * (k + 1) * 8, "flops": 2 * nnz * k + 4 * n * k}
    neig = 1 if kind == "eigvec_grad" else case["neig"]
    per, n0, power, fill = EFFORT[family]
    store = {0: val, 1: val // 2, 2: val // 4}[case.get("precision", 0)]
    full = 2 * nnz - n
    matvecs = neig * per * (n / n0) ** power
    # per MATVEC: the matrix once, the factor once in each sweep, and the vectors of the inner iteration (search
    # direction, its product, residual, preconditioned residual, two solutions: read and written once)
    one = full * (val + 4) + 2 * n * fill * (store + 4) + 12 * n * val
    return {"bytes": matvecs * one, "flops": matvecs * (2 * full + 4 * n * fill + 20 * n) * (4 if val == 16 else 1)}


def exact(case, seed):
    kind, family = case["kind"], case["family"]
    n, _ = _sizes(case)
    if kind in ("solve", "whole", "revcom"):
        # eigenvalues by a dense eigensolver; an eigenvector's sign, and its direction in a cluster, are free
        if n > 9000:
            return None
        A, B = _matrix(family, case["size"])
        D = _dense(_perturbed(A, seed, 1e-3 if kind == "whole" else 1e-5))
        if B is not None:
            d = 1.0 / torch.sqrt(torch.tensor(B[0], device="cuda"))
            D = d[:, None] * D * d[None, :]
        w = torch.linalg.eigvalsh(D)
        if SETTINGS[family]["isearch"] == 2:
            w = w[torch.argsort(torch.abs(w))]
        return {"eigs": torch.sort(w[:case["neig"]])[0].cpu().numpy(), "x": None, "neig": None, "info": None}
    s = prepare(case, seed)
    a, ja, ia = s["A"]
    rows, cols = np.repeat(np.arange(n), np.diff(ia)), np.asarray(ja, np.int64) - 1
    off = rows != cols
    if kind == "spmv":
        y = np.zeros(n, s["x"].dtype)
        for part in (np.real, np.imag) if np.iscomplexobj(y) else (np.real,):
            unit = 1j if part is np.imag else 1.0
            y += unit * np.bincount(rows, part(a * s["x"][cols]), n)
            y += unit * np.bincount(cols[off], part(np.conj(a[off]) * s["x"][rows[off]]), n)
        return y
    md = s["B"][0]
    if kind == "eig_grad":
        X = s["X"]
        c = s["w"] / np.einsum("nk,n,nk->k", X, md, X)
        return np.einsum("k,qk,qk->q", c, X[rows], X[cols]) * np.where(off, 2.0, 1.0)
    # mu of P^T (A - lam B) P mu = P^T g with x^T B mu = 0, as one bordered system
    x, b = torch.tensor(s["x"], device="cuda"), torch.tensor(md, device="cuda")
    g = torch.tensor(s["g"], device="cuda")
    x = x / torch.sqrt(x @ (b * x))
    K = torch.zeros((n + 1, n + 1), dtype=torch.float64, device="cuda")
    K[:n, :n] = _dense(s["A"]) - s["lam"] * torch.diag(b)
    K[n, :n] = K[:n, n] = b * x
    rhs = torch.cat([g - b * x * (x @ g), torch.zeros(1, dtype=torch.float64, device="cuda")])
    mu = torch.linalg.solve(K, rhs)[:n].cpu().numpy()
    x = x.cpu().numpy()
    return np.where(off, -(mu[rows] * x[cols] + mu[cols] * x[rows]), -mu[rows] * x[rows])
