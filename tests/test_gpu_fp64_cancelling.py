"""The FP64 form where sums of the interpolation cancel, against the oracle: fields that are
uniform over the mesh (their gradients are what rounding leaves, and they decide the directions
of h and of the discontinuity capturing), a shear flow oblique to the axes (dv v = 0 up to
rounding), nodal velocities whose sum vanishes at points (|v| < DBL_EPSILON decides tau).

Tolerance: the FP64 parity bound 1e-12 of the assembled matrix and rhs, as for other states: the
cancelling sums are formed with the reference's operations, so what they decide is the same.
"""
import numpy as np
import pytest

from cases import gm, syn, rel


def _mesh(kind):
    return {"tri": lambda: syn.channel_tri(16, 8), "quad": lambda: syn.channel_quad(12, 6, jitter=0.2, seed=1),
            "tet": lambda: syn.box_tet_delaunay(6, seed=2), "hex": lambda: syn.box_hex(4, 4, 3, jitter=0.1, seed=3)}[kind]()


def _state(mesh, nc, field):
    I, P = syn.state_for(mesh, nc, 0, no_slip_flag=-1)
    d, nd = mesh.dim, gm.nb_dofs(mesh.dim, nc)
    S = I.reshape(-1, nd)
    along, across = np.array([0.6, 0.8, 0.0])[:d], np.array([-0.8, 0.6, 0.0])[:d]
    if field == "uniform":
        S[:] = S[0]
    if field in ("uniform", "uniform velocity"):
        S[:, 1:1 + d] = np.array([20.0, 7.0, 3.0])[:d]
    elif field == "oblique shear":
        S[:, 1:1 + d] = (20.0 + 10.0 * (mesh.coords @ across))[:, None] * along
    else:  # nodal velocities -40, 0, 40 along one direction
        S[:, 1:1 + d] = 40.0 * np.random.default_rng(0).integers(-1, 2, size=(len(S), 1)) * along
    return S.ravel().copy(), P


@pytest.mark.gpu
@pytest.mark.parametrize("field", ["uniform", "uniform velocity", "oblique shear", "opposite velocities"])
@pytest.mark.parametrize("kind,nc", [("tri", 1), ("tri", 3), ("quad", 3), ("tet", 1), ("tet", 3), ("hex", 1), ("hex", 3)])
def test_cancelling_sums_match_the_oracle(kind, nc, field, cuda_lib):
    import oracle
    mesh = _mesh(kind)
    mat, setup = syn.material_for(nc, 0), syn.setup_for(mesh.dim, nc)
    I, P = _state(mesh, nc, field)
    fa = gm.FluidAssembly(mesh, mat, setup)
    lp = fa.linear_system()
    vals, rhs, s, _ = oracle.assemble(mesh, mat, setup, I, P, 1e-3, lp.row_ptr, lp.col)
    assert s == 0
    fa.execute(I, P, 1e-3, lp, form=gm.FORM_FP64)
    assert rel(lp.vals, vals) <= 1e-12 and rel(lp.rhs, rhs) <= 1e-12
    b = np.zeros(fa.n_rows)
    fa.residual(I, P, 1e-3, b, form=gm.FORM_FP64)
    assert rel(b, rhs) <= 1e-12
