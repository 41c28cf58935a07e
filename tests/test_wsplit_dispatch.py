"""Which kernels an FP32 step under w_split launches: the whole-column LO kernel
with the implicit step on its own, or the LO kernel that solves it in the same
pass, by columns, scheme, group width and cfg[4]; counted by launches, which
the values alone do not show."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

# volume, edge and mean-gradient fluxes, LO, limiting factors, update; the implicit step apart is one more
SAME_PASS, APART = 6, 7


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,K,V,ver,cfg4,launches", [
    (11, 9, 4, 4, "PPM", 0, SAME_PASS), (11, 9, 4, 4, "PPM", 3, APART), (11, 9, 3, 1, "CDIFF", 0, SAME_PASS),
    (67, 66, 1, 1, "PPM", 0, APART), (67, 66, 2, 2, "PPM", 0, APART), (67, 66, 8, 4, "PPM", 0, APART),
    (67, 66, 2, 2, "PPM", 2, SAME_PASS), (67, 66, 1, 1, "QR4C", 0, APART), (67, 66, 2, 2, "QR4C", 0, SAME_PASS),
    (67, 66, 4, 4, "QR4C", 0, SAME_PASS), (67, 66, 4, 4, "QR4C", 3, APART), (67, 66, 8, 4, "QR4C", 0, APART),
    (67, 66, 3, 1, "UPW1", 0, APART), (67, 66, 6, 2, "CDIFF", 0, APART), (67, 66, 2, 2, "CDIFF", 0, SAME_PASS),
    (67, 66, 8, 4, "UPW1", 0, SAME_PASS)])
def test_launches_under_wsplit(nx, ny, K, V, ver, cfg4, launches):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    nz = 13
    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(7)
    en = rng.integers(3, nz + 2, size=2 * (nx - 1) * (ny - 1)).astype(np.int32)
    en[0] = nz + 1
    m = Mesh(nx, ny, nz + 1, Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb,
             elem_nlev=en)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=2e-3)
    we = np.clip(w, -5e-4, 5e-4)
    T = synthetic.random_field(m, rng, K)
    out = []
    for cfg in ([0] * 4 + [cfg4], [0] * 4 + [2]):
        e = engine.TracerAdvection(m, K, "fp32", "MUSCL", ver, "FCT", copy_ab=True, tracer_vec=V)
        e.set_launch(cfg)
        e.set_tracers(T)
        e.set_velocity(vel, w, we, w - we)
        e.step(100.0)
        out.append((e.launches, e.values()))
    assert out[0][0] == launches and out[1][0] == SAME_PASS
    wet = np.arange(nz)[None, :] < (m.get("nlevels_nod2D") - 1)[:, None]
    # two roundings of the same FP32 result
    assert np.abs(out[0][1] - out[1][1])[:, wet].max() <= 1e-5 * np.abs(out[1][1][:, wet]).max()
