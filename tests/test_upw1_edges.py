"""FP32 upwind edge fluxes on both sides of the sizes at which the default moves
from the tiled to the per-edge kernel (groups of two and four tracers): the
same bits as with either kernel asked for, and within the FP32 bar of FP64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,K,V,lim,frozen", [
    (31, 29, 64, 4, 4, "FCT", True),    # 57,536 node-layers: tiled
    (97, 91, 61, 4, 4, "FCT", True),    # 564,928: per-edge for one group with a T_AB of its own
    (97, 91, 61, 8, 4, "FCT", True),    # tiled for two groups
    (129, 130, 63, 2, 2, "FCT", True),  # 1,073,280: per-edge for one group of two
    (181, 182, 64, 4, 4, "NONE", False),  # 2,108,288: per-edge without a limiter
    (181, 182, 64, 2, 2, "NONE", False)])
def test_upwind_edge_kernels_agree(nx, ny, nz, K, V, lim, frozen):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(K + nx)
    en = np.full(2 * (nx - 1) * (ny - 1), nz + 1, dtype=np.int32)
    en[: 4 * nx] = rng.integers(3, nz + 2, size=4 * nx)
    m = Mesh(nx, ny, nz + 1, Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb,
             elem_nlev=en)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=1e-4)
    T = synthetic.random_field(m, rng, K)
    TA = T + rng.normal(0, 0.05, size=T.shape) if frozen else None
    wet = np.arange(nz)[None, :] < (m.get("nlevels_nod2D") - 1)[:, None]

    def step(precision, cfg):
        kw = dict(tracer_vec=V) if precision == "fp32" else {}
        e = engine.TracerAdvection(m, K, precision, "UPW1", "PPM", lim, copy_ab=not frozen, **kw)
        e.set_launch(cfg)
        e.set_tracers(T, TA)
        e.set_velocity(vel, w)
        e.step(100.0)
        return e.values()[:, wet]

    default, tiled, per_edge = (step("fp32", c) for c in ([], [0] * 9 + [1], [8]))
    assert np.array_equal(default, tiled) and np.array_equal(default, per_edge)
    exact = step("fp64", [])
    assert np.abs(default - exact).max() <= 1e-5 * np.abs(exact).max()
