"""The assembly's form of the magma mixture (gales_magma_fast.cuh) against the property code it
rearranges (gales_magma.cuh), both compiled for the host: gas and crystal models, table kinds,
sub-mixture kinds, points in the tables, outside them and where no real sound speed exists.

Tolerance: some 40 operations of 1.1e-16 each on sums of one sign (cv subtracts a few per cent):
1e-14; the viscosity is a power of ten whose exponent, of order ten, is a quotient with a
difference of like numbers below: 100 times that.
"""
import ctypes as C
import shutil
import subprocess

import numpy as np
import pytest

from test_magma import MODELS, ROOT, _points, gm, magma, syn

FIELDS = ("rho", "mu", "cp", "cv", "kappa", "c", "alpha", "beta")


@pytest.fixture(scope="module")
def fast_lib(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not found")
    so = tmp_path_factory.mktemp("magma") / "magma_fast_host.so"
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-x", "cu", "-shared", "-Xcompiler", "-fPIC", "-Xcompiler",
                    "-ffp-contract=off", "-o", str(so), str(ROOT / "tests" / "host" / "magma_fast_host.cu")],
                   check=True)
    L = C.CDLL(str(so))
    dp = C.POINTER(C.c_double)
    L.magma_fast_host.argtypes = [C.POINTER(gm.abi.MagmaDesc), C.c_int32, dp, dp, dp, dp, C.c_int64, C.c_int, dp, dp,
                                  C.POINTER(C.c_int32)]
    L.magma_fast_host.restype = None
    return L


def _run(L, comps, p, T, Y, shear, which):
    d = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    n, nc = len(p), len(comps)
    out, comp, st = np.zeros((8, n)), np.zeros((nc, 4, n)), np.zeros(n, dtype=np.int32)
    Y = np.ascontiguousarray(Y)
    L.magma_fast_host(magma.descs(comps), nc, d(p), d(T), d(Y), d(shear), n, which, d(out), d(comp),
                      st.ctypes.data_as(C.POINTER(C.c_int32)))
    return out, comp, st


def _check(L, comps, p, T, Y, shear):
    o, c, s = _run(L, comps, p, T, Y, shear, 0)
    o1, c1, s1 = _run(L, comps, p, T, Y, shear, 1)
    assert np.array_equal(s, s1)
    for k, name in enumerate(FIELDS):
        np.testing.assert_allclose(o1[k], o[k], rtol=1e-12 if name == "mu" else 1e-14, atol=0, equal_nan=True,
                                   err_msg=name)
    np.testing.assert_allclose(c1[:, :3], c[:, :3], rtol=1e-14, atol=0, equal_nan=True)
    # the gas volume fraction: of a dissolved volatile's small remainder, to its own rounding
    np.testing.assert_allclose(c1[:, 3], c[:, 3], rtol=1e-14, atol=1e-16, equal_nan=True)
    zero = np.zeros_like(shear)
    r, _, sr = _run(L, comps, p, T, Y, zero, 2)
    o0, _, s0 = _run(L, comps, p, T, Y, zero, 0)
    assert np.array_equal(sr, s0)
    np.testing.assert_allclose(r[[0, 3]], o0[[0, 3]], rtol=1e-14, atol=0, equal_nan=True)


@pytest.mark.parametrize("gas, crystal, cf, n_T", MODELS + [("Pal_2003", "Einstein_Roscoe", 0.1, 7)])
def test_magma_pairs(gas, crystal, cf, n_T, fast_lib):
    _check(fast_lib, syn.magma_pair(gas, crystal, cf, n_T=n_T), *_points())


@pytest.mark.parametrize("n_T", [0, 7])
def test_outside_the_tables_and_without_a_sound_speed(n_T, fast_lib):
    p = np.array([1.0e7, 4.0e8, 1.0e8, 1.0e8, np.nan, 1.0e8, 2.0e9, 1.0e8])
    T = np.array([1200.0, 1300.0, 900.0, 2000.0, 1300.0, np.nan, 1300.0, -300.0])
    Y = np.tile([0.3, 0.7], (len(p), 1))
    _check(fast_lib, syn.magma_pair(n_T=n_T), p, T, Y, np.full(len(p), 2.0))


def test_other_sub_mixtures(fast_lib):
    melt = magma.CustomMix("melt", rho=2400.0, mu=1.0e3, cp=1200.0, kappa=1.5, alpha=3e-5, beta=1e-10)
    rigid = magma.CustomMix("rigid", rho=2600.0, mu=1.0e2, cp=1000.0, kappa=1.0, alpha=0.0, beta=0.0)
    comps = [syn.magma_pair()[0], melt, rigid]
    p, T, Y, shear = _points(nc=3)
    _check(fast_lib, comps, p, T, Y, shear)
