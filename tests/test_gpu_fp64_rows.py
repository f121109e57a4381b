"""The FP64 interior pass at the edges of its blocks of elements (32 simplices, 4 others).

Meshes of one element, a block less one, one block and one more element, a partial last block
and several chunks, with blocked rows in every element (the trace comes from another kernel), through the
atomic and the coloured scatter, the element blocks and the frozen adjoint, against the
oracle.  Tolerance: the FP64 parity bound 1e-12 of the assembled matrix and rhs (a row sums
some hundred products, each rounded to 1.1e-16 relative, and entries of one row are of one
size up to the cancellation of a few neighbours).
"""
import numpy as np
import pytest

from cases import gm, syn, rel


def _first(mesh, n):
    """The first n elements of a mesh (their boundary sides kept)."""
    conn = mesh.conn[:n]
    used, inv = np.unique(conn, return_inverse=True)
    bd = mesh.bd_sides[mesh.bd_sides[:, 0] < n]
    return gm.Mesh(mesh.coords[used], inv.reshape(conn.shape).astype(np.int32), mesh.node_flag[used],
                   mesh.el_on_boundary[:n], bd)


def _case(kind, nc, n, everywhere, tau):
    mesh = {"tri": lambda: syn.channel_tri(16, 8), "tet": lambda: syn.box_tet_delaunay(6, seed=3),
            "quad": lambda: syn.channel_quad(9, 6, jitter=0.2, seed=3),
            "hex": lambda: syn.box_hex(3, 4, 3, jitter=0.1, seed=3)}[kind]()
    mesh = _first(mesh, n)
    setup = syn.setup_for(mesh.dim, nc, dirichlet_T_everywhere=everywhere, tau=tau)
    mat = syn.material_for(nc, 2)
    I, P = syn.state_for(mesh, nc, 2)
    return mesh, mat, setup, I, P, 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nc,n,everywhere,tau", [
    ("tet", 3, 1, True, gm.TAU_2019), ("tet", 3, 31, True, gm.TAU_2014), ("tet", 1, 32, False, gm.TAU_2007),
    ("tet", 4, 33, True, gm.TAU_2001), ("tet", 2, 130, False, gm.TAU_2019), ("tri", 2, 33, True, gm.TAU_2019),
    ("tri", 4, 95, False, gm.TAU_2014), ("tri", 1, 64, True, gm.TAU_2019),
    ("quad", 2, 1, True, gm.TAU_2019), ("quad", 4, 37, False, gm.TAU_2014), ("quad", 1, 54, True, gm.TAU_2007),
    ("hex", 4, 5, True, gm.TAU_2019), ("hex", 1, 36, False, gm.TAU_2001), ("hex", 3, 7, True, gm.TAU_2014),
    ("hex", 2, 4, False, gm.TAU_2019)])
def test_block_edges_match_the_oracle(kind, nc, n, everywhere, tau, cuda_lib):
    import oracle
    mesh, mat, setup, I, P, dt = _case(kind, nc, n, everywhere, tau)
    fa = gm.FluidAssembly(mesh, mat, setup)
    lp = fa.linear_system()
    vals, rhs, s, _ = oracle.assemble(mesh, mat, setup, I, P, dt, lp.row_ptr, lp.col)
    assert s == 0
    for chunk in (0, 36):          # one chunk; chunks that end inside a block of records
        fa.set_chunk(chunk)
        for mode in (gm.SCATTER_ATOMIC, gm.SCATTER_COLOURED):
            fa.set_scatter(mode)
            fa.execute(I, P, dt, lp, form=gm.FORM_FP64)
            assert rel(lp.vals, vals) <= 1e-12 and rel(lp.rhs, rhs) <= 1e-12
    b = np.zeros(fa.n_rows)
    fa.residual(I, P, dt, b, form=gm.FORM_FP64)
    assert rel(b, rhs) <= 1e-12
    lam = np.random.default_rng(1).normal(size=fa.n_rows)
    g = np.zeros(fa.n_rows)
    fa.vjp(I, P, dt, lam, gm.VJP_FROZEN, g)
    lp.vals[:] = vals
    assert rel(g, lp.matrix_scipy().T @ lam) <= 1e-12
