"""The substitutions on both sides of the rule that takes a system of few unknowns to one cluster
or to all multiprocessors: much work per level (node rows, or bytes of the factor), little.  M^-1
against triangular solves of the same factor, with the tolerances of the other substitution tests:
1e-12 with an FP64 factor; with FP32 the backward error of a row's products and additions.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from cases import gm, syn
from test_gpu_solver_edges import F32, F64, _assembled


@pytest.mark.gpu
@pytest.mark.parametrize("kind, nc, fill, precond", [
    ("tet", 3, 0, F64), ("tet", 3, 1, F64), ("tet", 3, 0, F32), ("tet", 3, 1, F32), ("hex", 4, 1, F32), ("hex", 4, 0, F32)])
def test_substitutions_by_work_per_level(kind, nc, fill, precond, cuda_lib):
    import torch
    mesh = syn.box_tet_delaunay(14, seed=1) if kind == "tet" else syn.box_hex(9, 9, 62, jitter=0.1, seed=1)
    fa, lp = _assembled(mesh, nc)
    assert fa.n_rows * (8 if precond == F64 else 4) <= 200 * 1024
    sol = fa.linear_solver(gm.SolverParams(fill=fill, precond=precond))
    sol.factorize(lp.vals)
    f_rp, f_col, blocks = sol.factor()
    F = sp.bsr_matrix((np.asarray(blocks, dtype=np.float64), f_col, f_rp)).tocsr()
    n = fa.n_rows
    L, U = (sp.tril(F, -1) + sp.eye(n)).tocsr(), sp.triu(F).tocsr()
    v = np.random.default_rng(2).standard_normal(n)
    z = torch.zeros(n, dtype=torch.float64, device="cuda:0")
    sol.apply(torch.tensor(v, device="cuda:0"), z)
    z = z.cpu().numpy()
    if precond == F64:
        ref = sla.spsolve_triangular(U, sla.spsolve_triangular(L, v, lower=True), lower=False)
        assert np.linalg.norm(z - ref) <= 1e-12 * np.linalg.norm(ref)
        return
    m = max(np.diff(L.indptr).max(), np.diff(U.indptr).max()) + 2
    bound = 2.0 * m * 2.0 ** -24 * (abs(L) @ (abs(U) @ np.abs(z)))
    assert np.all(np.abs(L @ (U @ z) - v) <= 2.0 * bound + 2.0 ** -23 * np.abs(v))
