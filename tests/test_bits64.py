"""The FP64 kernels' integer comparisons, upwind product, limiter sums and
constant divisors (csrc/fgb_bits.cuh, fgb_kernels.cuh, fgb_intdiv.cuh) give what
the floating-point hardware gives, over normal, extreme and special operands:
the divisors on the host build too, with the reciprocal estimate pushed off by
a unit either way."""
import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "fesom2_tracer_dwarf_gb300", "csrc")
SRC = os.path.join(HERE, "bits64_check.cu")


@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_divisors_host(tmp_path, ulps):
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    exe = str(tmp_path / "bits64")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DULPS={ulps}", "-I", CSRC, "-I", HERE, "-x", "c++", SRC,
                    "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "0"


@pytest.mark.gpu
def test_helpers_device(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import build as B

    lib = str(tmp_path / "libbits64_check.so")
    subprocess.run([B._nvcc(), *B.ARCH, "-O3", "-std=c++17", "-fmad=false", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
                    "-I", CSRC, "-I", HERE, "-I", os.path.join(ROOT, "include"), "-shared", SRC, "-o", lib], check=True)
    f = ctypes.CDLL(lib).check_bits_device
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_int, ctypes.c_int, ctypes.c_ulonglong]
    assert f(152, 900, 20260411) == 0
