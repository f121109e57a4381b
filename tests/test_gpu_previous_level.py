"""The FP64 matrix and the frozen adjoint do not depend on the previous level P: a P that is no
state at all (zeros, as of a buffer never written, or NaN) leaves them alone, with status 0; only
the rhs is then not a number.  Bound: the FP64 parity bound 1e-12 against the oracle's matrix.
"""
import numpy as np
import pytest

import cases
from cases import gm, rel


def _gases():
    return gm.Material([gm.ideal_gas(0.018), gm.ideal_gas(0.044), gm.ideal_gas(0.028)])


@pytest.mark.gpu
@pytest.mark.parametrize("P_value", [0.0, float("nan")])
@pytest.mark.parametrize("kind,nc,gases", [("tri", 1, False), ("tri", 3, True), ("quad", 2, False), ("tet", 3, False),
                                           ("tet", 3, True), ("hex", 4, False)])
def test_matrix_without_a_previous_level(kind, nc, gases, P_value, cuda_lib):
    import oracle
    mesh, mat, setup, I, P, dt = cases.make(kind, nc)
    if gases:
        mat = _gases()
    fa = gm.FluidAssembly(mesh, mat, setup)
    lp = fa.linear_system()
    vals, rhs, s, _ = oracle.assemble(mesh, mat, setup, I, P, dt, lp.row_ptr, lp.col)
    assert s == 0
    none = np.full_like(P, P_value)
    fa.execute(I, none, dt, lp, form=gm.FORM_FP64)
    assert rel(lp.vals, vals) <= 1e-12
    # zeros are a state of a material without a gas
    assert np.isfinite(lp.rhs).all() == (nc == 1 and P_value == 0.0)
    lam = np.random.default_rng(1).normal(size=fa.n_rows)
    g = np.zeros(fa.n_rows)
    fa.vjp(I, none, dt, lam, gm.VJP_FROZEN, g)
    lp.vals[:] = vals
    assert rel(g, lp.matrix_scipy().T @ lam) <= 1e-12
