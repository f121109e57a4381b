"""The solver's kernels called one by one, and its path for rows too long for shared memory.

A wait of the persistent kernels that runs out: the kernel ends with an error word, the
context stays usable, and the caller of an enqueued apply learns of it from sync() or the next
factorisation or solve, once.  The waits run out because the rows that they wait for are not in
the kernel's list.

Arnoldi passes around a tile of columns (96) and the staged coefficients (512), against numpy: a
sum of n products has an error below n 1.1e-16 of the sum of their magnitudes.

Factorisation by levels (a node with more neighbours than a block row in shared memory may have):
the same entries as elimination in plain numpy, bit for bit, in FP64 and FP32.
"""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from cases import gm, syn

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def kernels_lib(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not found")
    so = tmp_path_factory.mktemp("solver") / "solver_kernels.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-diag-suppress", "128", "-o", str(so),
                    str(ROOT / "tests" / "host" / "solver_kernels.cu")], check=True)
    return C.CDLL(str(so))


@pytest.mark.gpu
def test_reported_once(cuda_lib, kernels_lib):
    out = (C.c_int * 6)()
    assert kernels_lib.solver_reports(out) == 0
    t = gm.abi.ERR_TIMEOUT
    assert list(out) == [t, 0, t, 0, t, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_wait_runs_out(kernel, cuda_lib, kernels_lib):
    assert kernels_lib.solver_wait_runs_out(kernel) == gm.abi.ERR_TIMEOUT
    out = (C.c_int * 6)()
    assert kernels_lib.solver_reports(out) == 0   # the device goes on


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [1, 95, 96, 97, 511, 512, 513, 530])
def test_arnoldi_passes(nv, cuda_lib, kernels_lib):
    n = 1317   # six tiles of rows, the last with 37
    rng = np.random.default_rng(nv)
    V, w0 = np.asfortranarray(rng.standard_normal((n, nv))) / np.sqrt(n), rng.standard_normal(n)
    w, h, h1, h2, w1, hn = w0.copy(), np.zeros(nv), np.zeros(nv), np.zeros(nv), np.zeros(n), np.zeros(1)
    d = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    assert kernels_lib.solver_arnoldi(d(V), C.c_int64(n), nv, d(w), d(h), d(h1), d(h2), d(w1), d(hn)) == 0
    eps, A = 2.0 ** -53, np.abs(V)
    assert np.all(np.abs(h - V.T @ w0) <= 2 * n * eps * (A.T @ np.abs(w0)))
    # each pass from the vectors that the one before left
    assert np.all(np.abs(w1 - (w0 - V @ h)) <= 2 * (nv + 1) * eps * (np.abs(w0) + A @ np.abs(h)))
    assert np.all(np.abs(h2 - V.T @ w1) <= 2 * n * eps * (A.T @ np.abs(w1)))
    assert np.array_equal(h1, h + h2)
    assert np.all(np.abs(w - (w1 - V @ h2)) <= 2 * (nv + 1) * eps * (np.abs(w1) + A @ np.abs(h2)))
    assert abs(hn[0] - np.linalg.norm(w)) <= 2 * n * eps * np.linalg.norm(w)


def _eliminate(rows, F, nd):
    """ILU(0) of node blocks F[i][j], row by row with the entries' subtractions in scalar ikj order."""
    for i in rows:
        R = F[i]
        for k in sorted(j for j in R if j < i):
            B, U = R[k], F[k][k]
            for c in range(nd):
                for c2 in range(c):
                    B[:, c] -= B[:, c2] * U[c2, c]
                B[:, c] /= U[c, c]
            for j, Uj in F[k].items():
                if j > k and j in R:
                    for m in range(nd):
                        R[j] -= np.outer(B[:, m], Uj[m])
        D = R[i]
        for c2 in range(nd - 1):
            D[c2 + 1:, c2] /= D[c2, c2]
            D[c2 + 1:, c2 + 1:] -= np.outer(D[c2 + 1:, c2], D[c2, c2 + 1:])
            for j in R:
                if j > i:
                    R[j][c2 + 1:] -= np.outer(D[c2 + 1:, c2], R[j][c2])


@pytest.mark.gpu
@pytest.mark.parametrize("n, precond, dtype", [(660, gm.PRECOND_ILU, np.float64), (1300, gm.PRECOND_ILU_FP32, np.float32)])
def test_factorisation_by_levels(n, precond, dtype, cuda_lib):
    # a fan of n triangles around node 0, whose block row passes an SM's shared memory
    a = 2.0 * np.pi * np.arange(n) / n
    coords = np.vstack([[0.0, 0.0], np.stack([np.cos(a), np.sin(a)], axis=1)])
    i = np.arange(n)
    conn = np.stack([0 * i, 1 + i, 1 + (i + 1) % n], axis=1).astype(np.int32)
    mesh = gm.Mesh(coords, conn, np.zeros(n + 1, dtype=np.int32), np.zeros(n, dtype=np.uint8), np.zeros((0, 3), dtype=np.int32))
    fa = gm.FluidAssembly(mesh, syn.material_for(1, 0), syn.setup_for(2, 1))
    nd, (rp, col) = fa.nd, fa.node_graph()[:2]
    rng = np.random.default_rng(0)
    F, vals = [], []
    for r in range(n + 1):
        cols = col[rp[r]:rp[r + 1]]
        blocks = [rng.standard_normal((nd, nd)) + (4.0 * len(cols) if c == r else 0.0) * np.eye(nd) for c in cols]
        vals.append(np.hstack(blocks).ravel())
        F.append({int(c): b.astype(dtype) for c, b in zip(cols, blocks)})
    sol = fa.linear_solver(gm.SolverParams(fill=0, precond=precond))
    n0 = sol.launch_count()
    sol.factorize(np.concatenate(vals))
    assert sol.launch_count() - n0 >= sol.levels()[0]   # a launch per level
    f_rp, f_col, blocks = sol.factor()
    _eliminate(range(n + 1), F, nd)
    for r in range(n + 1):
        for p in range(f_rp[r], f_rp[r + 1]):
            assert np.array_equal(blocks[p].astype(dtype), F[r][int(f_col[p])]), (r, f_col[p])
