"""The mixed interior pass at the edges of its blocks of 32 elements.

One element, a block less one, one block, one more element, a partial last block and chunks that
end inside a block, with blocked rows in every element (the trace comes from another kernel),
through the atomic and the coloured scatter, the residual and the element blocks, against the
oracle.  Tolerance: 1e-6 relative, the mixed form's bound: a row is a sum of some hundred FP32
products, each rounded to 6e-8, whose errors add like a random walk (about ten times 6e-8).
"""
import numpy as np
import pytest

from cases import gm, rel
from test_gpu_fp64_rows import _case

TOL = 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nc,n,everywhere,tau", [
    ("tet", 3, 1, True, gm.TAU_2019), ("tet", 4, 31, True, gm.TAU_2014), ("tet", 1, 32, False, gm.TAU_2007),
    ("tet", 4, 33, True, gm.TAU_2001), ("tet", 2, 130, False, gm.TAU_2019), ("tri", 2, 33, True, gm.TAU_2019),
    ("tri", 4, 95, False, gm.TAU_2014), ("tri", 1, 64, True, gm.TAU_2019),
    ("quad", 2, 1, True, gm.TAU_2019), ("quad", 4, 37, False, gm.TAU_2014), ("quad", 3, 54, True, gm.TAU_2007),
    ("hex", 4, 33, True, gm.TAU_2019), ("hex", 1, 36, False, gm.TAU_2001), ("hex", 3, 7, True, gm.TAU_2014),
    ("hex", 2, 32, False, gm.TAU_2019)])
def test_block_edges_match_the_oracle(kind, nc, n, everywhere, tau, cuda_lib):
    import oracle
    mesh, mat, setup, I, P, dt = _case(kind, nc, n, everywhere, tau)
    fa = gm.FluidAssembly(mesh, mat, setup)
    lp = fa.linear_system()
    vals, rhs, s, _ = oracle.assemble(mesh, mat, setup, I, P, dt, lp.row_ptr, lp.col)
    assert s == 0
    for chunk in (0, 36):
        fa.set_chunk(chunk)
        for mode in (gm.SCATTER_ATOMIC, gm.SCATTER_COLOURED):
            fa.set_scatter(mode)
            fa.execute(I, P, dt, lp, form=gm.FORM_MIXED)
            assert rel(lp.vals, vals) <= TOL and rel(lp.rhs, rhs) <= TOL
    b = np.zeros(fa.n_rows)
    fa.residual(I, P, dt, b, form=gm.FORM_MIXED)
    assert rel(b, rhs) <= TOL
    el = np.array([0, n - 1, n // 2], dtype=np.int32)
    m, r = fa.element_blocks(I, P, dt, el, form=gm.FORM_MIXED)
    m64, r64 = fa.element_blocks(I, P, dt, el, form=gm.FORM_FP64)
    assert rel(m, m64) <= TOL and rel(r, r64) <= TOL
