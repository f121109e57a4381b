"""The linear solver's kernels where their paths change: the sweeps of one cluster up to the
longest result vector that a CTA holds (200 KiB) and through L2 beyond, rows of more blocks than a
warp holds at once, a single element; Arnoldi passes over more columns than a tile (96) and than
the staged Hessenberg part (512), with a vector length that no tile divides.

Tolerances.  M^-1 with an FP64 factor against triangular solves of the same factor: 1e-12 as for
the small systems.  With an FP32 factor the solution's error grows with the condition of the
triangles (the kernel's and any other order's alike), so its backward error is bounded: each
substitution satisfies its equations to the rounding of a row's m products and its m additions,
2 m 6e-8 of their absolute values.  Krylov: the reported residual is that of the returned x.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

import cases
from cases import gm, syn

F64, F32 = gm.PRECOND_ILU, gm.PRECOND_ILU_FP32


def _assembled(mesh, nc):
    import torch
    fa = gm.FluidAssembly(mesh, syn.material_for(nc, 1), syn.setup_for(mesh.dim, nc))
    lp = fa.linear_system("cuda:0")
    I, P = (torch.tensor(x, device="cuda:0") for x in syn.state_for(mesh, nc, 1))
    fa.execute(I, P, 1e-3, lp, form=gm.FORM_FP64)
    return fa, lp


@pytest.mark.gpu
@pytest.mark.parametrize("mesh, nc, fill, precond", [
    (("quad", 1, 1), 1, 1, F64), (("quad", 79, 79), 1, 1, F64), (("quad", 80, 79), 1, 1, F64),
    (("quad", 127, 79), 2, 1, F32), (("quad", 128, 79), 2, 1, F32), (("hex", 5, 4, 4), 4, 2, F64),
    (("hex", 5, 4, 4), 4, 2, F32), (("hex", 17, 16, 14), 2, 1, F64), (("hex", 4, 4, 3), 3, 3, F64)])
def test_substitutions(mesh, nc, fill, precond, cuda_lib):
    import torch
    m = syn.channel_quad(*mesh[1:], jitter=0.2, seed=1) if mesh[0] == "quad" else syn.box_hex(*mesh[1:], jitter=0.1, seed=1)
    fa, lp = _assembled(m, nc)
    sol = fa.linear_solver(gm.SolverParams(fill=fill, precond=precond))
    sol.factorize(lp.vals)
    f_rp, f_col, blocks = sol.factor()
    F = sp.bsr_matrix((np.asarray(blocks, dtype=np.float64), f_col, f_rp)).tocsr()
    n = fa.n_rows
    v = np.random.default_rng(2).standard_normal(n)
    z = torch.zeros(n, dtype=torch.float64, device="cuda:0")
    sol.apply(torch.tensor(v, device="cuda:0"), z)
    y = sla.spsolve_triangular((sp.tril(F, -1) + sp.eye(n)).tocsr(), v, lower=True)
    ref = sla.spsolve_triangular(sp.triu(F).tocsr(), y, lower=False)
    z = z.cpu().numpy()
    if precond == F64:
        assert np.linalg.norm(z - ref) <= 1e-12 * np.linalg.norm(ref)
        return
    L, U = (sp.tril(F, -1) + sp.eye(n)).tocsr(), sp.triu(F).tocsr()
    m = max(np.diff(L.indptr).max(), np.diff(U.indptr).max()) + 2
    bound = 2.0 * m * 2.0 ** -24 * (abs(L) @ (abs(U) @ np.abs(z)))
    assert np.all(np.abs(L @ (U @ z) - v) <= 2.0 * bound + 2.0 ** -23 * np.abs(v))


@pytest.mark.gpu
@pytest.mark.parametrize("iters", [96, 97, 512, 513, 530])
def test_many_krylov_columns(iters, cuda_lib):
    import torch
    fa, lp = _assembled(syn.channel_tri(16, 8), 3)
    assert fa.n_rows % 256 != 0 and fa.n_rows > 530
    sol = fa.linear_solver(gm.SolverParams(precond=gm.PRECOND_NONE, maxsubspace=540, maxiters=iters, rel_res_tol=0.0))
    x = torch.zeros(fa.n_rows, dtype=torch.float64, device="cuda:0")
    sol.solve(lp.vals, lp.rhs, x)
    assert sol.num_it == iters
    A = sp.csr_matrix((lp.vals.cpu().numpy(), lp.col, lp.row_ptr), shape=(fa.n_rows,) * 2)
    b = lp.rhs.cpu().numpy()
    assert np.linalg.norm(b - A @ x.cpu().numpy()) == pytest.approx(sol.ARE, rel=1e-4, abs=1e-10 * np.linalg.norm(b))
    # the least-squares residual never grows with the space
    few = fa.linear_solver(gm.SolverParams(precond=gm.PRECOND_NONE, maxsubspace=540, maxiters=90, rel_res_tol=0.0))
    y = torch.zeros_like(x)
    few.solve(lp.vals, lp.rhs, y)
    assert sol.ARE <= few.ARE * (1.0 + 1e-9)
