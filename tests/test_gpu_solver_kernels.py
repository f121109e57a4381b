"""A wait of the solver's persistent kernels that runs out: the kernel ends with an error word, the
context stays usable, and the caller of an enqueued apply learns of it from sync() or the next
factorisation or solve, once.  The waits run out because the rows that they wait for are not in
the kernel's list."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

from cases import gm

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
