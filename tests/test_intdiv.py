"""The FP64 division, multiplication and comparisons on the integer pipe (csrc/fgb_intdiv.cuh,
fgb_bits.cuh) give the hardware's results bit for bit: on the host build with
the reciprocal estimate as it is and pushed off by a unit either way, and on the
GPU."""
import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fesom2_tracer_dwarf_gb300", "csrc")
SRC = os.path.join(HERE, "intdiv_check.cu")


@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_divide_host(tmp_path, ulps):
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    exe = str(tmp_path / "intdiv")
    subprocess.run(["g++", "-O2", "-std=c++17", f"-DULPS={ulps}", "-I", CSRC, "-x", "c++", SRC, "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "0"


@pytest.mark.gpu
def test_divide_and_compare_device(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import build as B

    lib = str(tmp_path / "libintdiv_check.so")
    subprocess.run([B._nvcc(), *B.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
                    "-I", CSRC, "-shared", SRC, "-o", lib], check=True)
    f = ctypes.CDLL(lib).check_device
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_int, ctypes.c_int, ctypes.c_ulonglong]
    assert f(152, 800, 20260301) == 0
