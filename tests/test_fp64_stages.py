"""FP64 forms: a whole step (volume fluxes formed in the edge-flux kernel,
element gradients formed once) gives the bits of the same step called stage by
stage (separate volume fluxes, gradients formed per edge), on ragged meshes
whose layer counts cross the warp's width and whose edges do not fill the last
block."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
@pytest.mark.parametrize("hor,lim", [("UPW1", "FCT"), ("MUSCL", "FCT"), ("MFCT", "FCT"), ("MUSCL", "NONE")])
@pytest.mark.parametrize("nx,ny,nz,K,ph", [(2, 2, 2, 1, 1.0), (7, 6, 3, 3, 0.75), (13, 9, 31, 2, 1.0), (11, 12, 32, 4, 1.0),
                                           (12, 7, 33, 5, 0.75), (9, 8, 65, 2, 1.0)])
def test_whole_step_equals_stages(nx, ny, nz, K, ph, hor, lim, precision):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import _lib, engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(nx * 100 + nz)
    en = rng.integers(min(3, nz + 1), nz + 2, size=2 * (nx - 1) * (ny - 1)).astype(np.int32)  # 2..nz layers
    en[0] = nz + 1
    m = Mesh(nx, ny, nz + 1, Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb,
             elem_nlev=en)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=1e-3)
    T = synthetic.random_field(m, rng, K)
    out = []
    for masks in ([_lib.STAGE_ALL], [1, 2, 4, 8, 16]):
        e = engine.TracerAdvection(m, K, precision, hor, "PPM", lim, ph=ph, copy_ab=lim == "FCT")
        e.set_tracers(T)
        e.set_velocity(vel, w)
        for _ in range(2):
            for mask in masks:
                e.step(100.0, 1, mask)
        out.append(e.values())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
