"""Equal time levels.  A time step starts from I = P (the predictor), where U - U_P is zero: the
rhs without stabilisation then does not depend on dt, to the bit.  One rounding of U that U_P does
not share, divided by the small dt of the test, is 1e-8 of the rhs.

Element by element (no sums over elements), both forms, the chemicals' mixture and a mixture of
two magmas.
"""
import importlib

import numpy as np
import pytest

from cases import gm, syn

magma = importlib.import_module("gales-multi-fluid_gb300.magma")


@pytest.mark.gpu
@pytest.mark.parametrize("form", [gm.FORM_FP64, gm.FORM_MIXED])
@pytest.mark.parametrize("material", [1, 2, 3, 4, "magma", "magma with crystals"])
@pytest.mark.parametrize("kind", ["tri", "quad", "tet", "hex"])
def test_equal_levels_have_no_rate_of_change(kind, material, form, cuda_lib):
    mesh = {"tri": lambda: syn.channel_tri(16, 8), "quad": lambda: syn.channel_quad(12, 6, jitter=0.2, seed=1),
            "tet": lambda: syn.box_tet_delaunay(6, seed=2), "hex": lambda: syn.box_hex(4, 4, 3, jitter=0.1, seed=3)}[kind]()
    magmas = isinstance(material, str)
    nc = 2 if magmas else material
    setup = syn.setup_for(mesh.dim, nc, tau=gm.TAU_NONE, dc_2006=False)
    I, _ = syn.state_for(mesh, nc, 0, no_slip_flag=-1)
    fa = gm.FluidAssembly(mesh, syn.material_for(nc, 0), setup)
    if magmas:   # pressures inside the solubility tables
        p = I.reshape(-1, gm.nb_dofs(mesh.dim, nc))[:, 0]
        p[:] = 7.5e7 + 2.0e8 * (p - p.min()) / (p.max() - p.min())
        kw = dict(crystal_on_mu="Einstein_Roscoe", crystal_fraction=0.1) if "crystals" in material else {}
        mg = magma.MagmaMaterial(syn.magma_pair(**kw))
        fa.set_magma(mg)
    els = np.arange(mesh.n_elements, dtype=np.int32)
    _, a = fa.element_blocks(I, I.copy(), 1e-3, els, 0, form, want_matrix=False)
    _, b = fa.element_blocks(I, I.copy(), 1e-9, els, 0, form, want_matrix=False)
    assert np.abs(a).max() > 0.0 and np.array_equal(a, b)
