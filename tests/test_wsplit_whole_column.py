"""FP32 w_split through the whole-column LO kernel and the separate implicit
step: asked for on a small ragged mesh (every vertical scheme and group width,
T_AB shared or separate) and taken by default on a mesh of more than a wave of
columns, against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

REL_TOL = 1e-5  # the FP32 form's bar against FP64 (relative max-norm)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,K,V,ver,frozen", [
    (11, 9, 2, 1, 1, "UPW1", False), (11, 9, 31, 4, 4, "QR4C", True), (11, 9, 32, 2, 2, "CDIFF", False),
    (11, 9, 33, 3, 1, "PPM", True), (11, 9, 63, 4, 4, "PPM", False), (11, 9, 64, 8, 4, "QR4C", False),
    (67, 66, 9, 2, 2, "PPM", False), (67, 66, 12, 4, 4, "QR4C", False)])
def test_wsplit_whole_column(oracle_mod, nx, ny, nz, K, V, ver, frozen):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    O = oracle_mod
    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(13 * nz + K)
    en = rng.integers(3, nz + 2, size=2 * (nx - 1) * (ny - 1)).astype(np.int32)
    en[0] = nz + 1
    kw = dict(Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb, elem_nlev=en)
    m, om = Mesh(nx, ny, nz + 1, **kw), O.Mesh(nx, ny, nz + 1, **kw)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=2e-3)
    we = np.clip(w, -5e-4, 5e-4)
    T = synthetic.random_field(m, rng, K)
    TA = T + rng.normal(0, 0.05, size=T.shape) if frozen else T
    vals, vab = np.ascontiguousarray(T.copy()), np.ascontiguousarray(TA.copy())
    sch = ("MUSCL", ver, "FCT", 0.8, 0.7)
    W = O.Work(om)
    for _ in range(2):
        O.analytic_step(om, W, 100.0, vel, w, vals, vab, [sch] * K, copy_ab=not frozen, wi=w - we, we=we)
    e = engine.TracerAdvection(m, K, "fp32", *sch[:3], ph=0.8, pv=0.7, copy_ab=not frozen, tracer_vec=V)
    if m.N <= 152 * 28:
        e.set_launch([0] * 4 + [3])
    e.set_tracers(T, TA if frozen else None)
    e.set_velocity(vel, w, we, w - we)
    before = e.launches
    e.step(100.0)
    # volume, edge (and mean-gradient) fluxes, LO, the implicit step on its own, ratio, update
    assert e.launches - before >= 6
    e.step(100.0)
    wet = np.arange(nz)[None, :] < (m.get("nlevels_nod2D") - 1)[:, None]
    assert np.abs(e.values() - vals)[:, wet].max() <= REL_TOL * np.abs(vals).max()
