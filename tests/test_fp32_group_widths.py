"""The compensated low-order sums of the FP32 form do not depend on the width of
a tracer group: groups of two and four tracers (packed arithmetic) give the
increments of groups of one (scalar arithmetic, each product and sum rounded by
itself) bit for bit, for every vertical scheme and kernel variant. A product
fused into a compensated sum's addition would differ."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("wmode", ["shared", "apart", "wsplit"])
@pytest.mark.parametrize("frozen", [False, True])
@pytest.mark.parametrize("ver", ["UPW1", "QR4C", "CDIFF", "PPM"])
def test_compensated_low_order_increments(ver, frozen, wmode):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import _lib, engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    nx, ny, nz, K = 13, 11, 37, 4
    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(5)
    en = rng.integers(3, nz + 2, size=2 * (nx - 1) * (ny - 1)).astype(np.int32)
    en[0] = nz + 1
    m = Mesh(nx, ny, nz + 1, Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb,
             elem_nlev=en)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=2e-3)
    we = np.clip(w, -5e-4, 5e-4)
    T = synthetic.random_field(m, rng, K)
    for variant in (3, 2, 1):  # the whole-column kernel, two layers and one layer per lane
        lo = []
        for V in (1, 2, 4):
            e = engine.TracerAdvection(m, K, "fp32", "MUSCL", ver, "FCT", copy_ab=not frozen, tracer_vec=V, plain_sums=6)
            e.set_launch([0] * 4 + [variant])
            e.set_tracers(T, T * 1.001 if frozen else None)
            e.set_velocity(vel, w, {"shared": None, "apart": w.copy(), "wsplit": we}[wmode],
                           w - we if wmode == "wsplit" else None)
            e.step(100.0, 1, _lib.STAGE_VFLUX | _lib.STAGE_HFLUX | _lib.STAGE_LO)
            off = (ctypes.c_longlong * 7)()
            assert _lib.load().fgb_workspace_offsets(m.handle, _lib.FP32, K, off) == 0
            a = e.workspace.cpu().numpy().view(np.float32)[off[3] // 4 :][: K * m.N * m.LZ]
            lo.append(a.reshape(K // V, m.N, m.LZ, V).transpose(0, 3, 1, 2).reshape(K, m.N, m.LZ))
        if variant == 1 and wmode == "wsplit":
            continue  # the solver's own arithmetic follows in the same array
        assert np.array_equal(lo[0], lo[1]) and np.array_equal(lo[0], lo[2]), variant
