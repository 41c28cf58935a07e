"""Spills (ptxas's report for sm_103a, no GPU needed) of FP32 kernels beside
the headline ones of test_kernel_resources: at most what the timed builds had,
so that a change which pushes a variant's values into local memory shows. The
FP64 node and edge kernels: none, at the blocks their launch bounds ask for."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

# kernel -> bytes of spill stores at most
EXPECTED = {
    "kf_hflux<1, true, 4, 1>": 16,
    "kf_hflux<1, true, 4, 2>": 0,
    "kf_hflux<2, true, 4, 1>": 12,
    "kf_hflux<2, true, 4, 2>": 0,
    "kf_hflux<1, true, 2, 1>": 0,
    "kf_hflux_mean<1, true, 4>": 0,
    "kf_hflux_mean<2, true, 2>": 0,
    "kf_lo64<1, 4, true, true, false>": 0,
    "kf_lo64<3, 4, true, true, false>": 0,
    "kf_lo64<1, 2, false, true, false>": 0,
    "kf_ratio64<2, false, true>": 0,
    "kf_ratio64<1, false, true>": 0,
    "kf_update<1, 1, false, true, false>": 0,
    "kf_update<2, 1, false, false, false>": 8,
    "kf_vflux4": 0,
}


# exact FP64 form: kernel -> blocks of 128 threads per SM its launch bound asks for (256 threads: twice)
EXPECTED_F64 = {
    "k_fct_lo<double, 1>": 7,
    "k_fct_lo<double, 3>": 6,
    "k_fct_ratio<double>": 6,
    "k_fct_update<double>": 7,
    "k_nofct_update<double, 3>": 6,
    "k_hflux<double, 1, true, true, true>": 8,
}


def _report(tmp_path, source, *flags):
    """{kernel: (bytes of spill stores, registers)} of a unit."""
    from fesom2_tracer_dwarf_gb300 import build as B

    try:
        nvcc = B._nvcc()
    except RuntimeError:
        pytest.skip("nvcc is not installed")
    if shutil.which("c++filt") is None:
        pytest.skip("c++filt is not installed")
    cmd = [nvcc, *B.ARCH, *B.NVCC_COMMON, *flags, "-Xptxas", "-v", "-c", os.path.join(HERE, source), "-o",
           str(tmp_path / "unit.o")]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    text = subprocess.run(["c++filt"], input=r.stdout + r.stderr, capture_output=True, text=True).stdout
    out, cur = {}, None
    for line in text.splitlines():
        m = re.search(r"Compiling entry function '(?:void )?(?:fgb::(?:fast|exact64)::)?([^(']+)", line)
        if m:
            cur = m.group(1).strip()
            out[cur] = [None, None]
        m = re.search(r"(\d+) bytes spill stores", line)
        if m and cur:
            out[cur][0] = int(m.group(1))
        m = re.search(r"Used (\d+) registers", line)
        if m and cur:
            out[cur][1] = int(m.group(1))
    return out


def test_variants_spill_no_more_than_measured(tmp_path):
    rep = _report(tmp_path, "kernel_variants.cu")
    for name, most in EXPECTED.items():
        assert name in rep, f"{name} not in the report: {sorted(rep)}"
        assert rep[name][0] <= most, f"{name}: {rep[name][0]} bytes of spill stores, {most} when it was measured"


def test_fp64_kernels_fit_their_launch_bounds(tmp_path):
    rep = _report(tmp_path, "kernel_variants_f64.cu", "-fmad=false")
    for name, blocks in EXPECTED_F64.items():
        assert name in rep, f"{name} not in the report: {sorted(rep)}"
        spill, regs = rep[name]
        assert spill == 0, f"{name}: {spill} bytes of spill stores"
        assert regs <= 65536 // (blocks * 128), f"{name}: {regs} registers for {blocks} blocks"
