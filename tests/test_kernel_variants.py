"""Spills (ptxas's report for sm_103a, no GPU needed) of FP32 kernels beside
the headline ones of test_kernel_resources: at most what the timed builds had,
so that a change which pushes a variant's values into local memory shows."""
import os
import re
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


def test_variants_spill_no_more_than_measured(tmp_path):
    import shutil

    from fesom2_tracer_dwarf_gb300 import build as B

    try:
        nvcc = B._nvcc()
    except RuntimeError:
        pytest.skip("nvcc is not installed")
    if shutil.which("c++filt") is None:
        pytest.skip("c++filt is not installed")
    cmd = [nvcc, *B.ARCH, *B.NVCC_COMMON, "-Xptxas", "-v", "-c", os.path.join(HERE, "kernel_variants.cu"), "-o",
           str(tmp_path / "kernel_variants.o")]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    text = subprocess.run(["c++filt"], input=r.stdout + r.stderr, capture_output=True, text=True).stdout
    spill, cur = {}, None
    for line in text.splitlines():
        m = re.search(r"Compiling entry function '(?:void )?(?:fgb::fast::)?([^(']+)", line)
        if m:
            cur = m.group(1).strip()
        m = re.search(r"(\d+) bytes spill stores", line)
        if m and cur:
            spill[cur] = int(m.group(1))
    for name, most in EXPECTED.items():
        assert name in spill, f"{name} not in the report: {sorted(spill)}"
        assert spill[name] <= most, f"{name}: {spill[name]} bytes of spill stores, {most} when it was measured"
