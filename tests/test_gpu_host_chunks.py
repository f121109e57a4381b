"""Chunks of a host-buffer assembly: as many as there are pieces of the matrix worth a copy of
their own.  A small mesh is one chunk (its launches are those of a device-buffer call and the two
clear kernels), a large one several; both equal the device-buffer assembly up to the order in
which the elements' values are added (sums of some ten values in FP64: 1e-13)."""
import numpy as np
import pytest

from cases import gm, rel, syn


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nc,chunks", [("tri", 2, 1), ("tet", 1, 1), ("quad", 3, 2), ("hex", 4, 4)])
def test_pinned_assembly_in_chunks(kind, nc, chunks, cuda_lib):
    torch = pytest.importorskip("torch")
    mesh = {"tri": lambda: syn.channel_tri(30, 25), "tet": lambda: syn.box_tet_delaunay(6, seed=3),
            "quad": lambda: syn.channel_quad(151, 101, jitter=0.2, seed=1),
            "hex": lambda: syn.box_hex(21, 19, 17, jitter=0.1, seed=1)}[kind]()
    I, P = syn.state_for(mesh, nc, 0)
    fa = gm.FluidAssembly(mesh, syn.material_for(nc, 0), syn.setup_for(mesh.dim, nc))
    dev = torch.device("cuda:0")
    ref = fa.linear_system(device=dev)
    n0 = fa.launch_count()
    fa.execute(torch.tensor(I, device=dev), torch.tensor(P, device=dev), 1e-3, ref, form=gm.FORM_MIXED)
    single = fa.launch_count() - n0
    pin = lambda n: torch.full((n,), float("nan"), dtype=torch.float64).pin_memory()
    lp = gm.LinearSystem(ref.row_ptr, ref.col, pin(len(ref.vals)), pin(len(ref.rhs)))
    for _ in range(2):
        n0 = fa.launch_count()
        fa.execute(torch.from_numpy(I).pin_memory(), torch.from_numpy(P).pin_memory(), 1e-3, lp, form=gm.FORM_MIXED)
        extra = fa.launch_count() - n0 - single - 2
        assert extra == 0 if chunks == 1 else extra >= 2 * (chunks - 1)
        assert rel(lp.vals.numpy(), ref.vals.cpu().numpy()) <= 1e-13
        assert rel(lp.rhs.numpy(), ref.rhs.cpu().numpy()) <= 1e-13
