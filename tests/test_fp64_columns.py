"""FP64 node kernels against the oracle where their dealing of (tracer, layer)
pairs to lanes can go wrong: layer counts around the warp's width, ragged
columns, tracer counts that fill no chunk, every vertical scheme, the AB levels
and the implicit vertical step. The exact form bit for bit, the fast form to
1e-12 (fused multiply-add and reciprocals, relative to the largest value)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("ver,lim", [("UPW1", "FCT"), ("QR4C", "FCT"), ("CDIFF", "FCT"), ("PPM", "FCT"), ("QR4C", "NONE"),
                                     ("PPM", "NONE")])
@pytest.mark.parametrize("nz,K,wsplit", [(2, 1, False), (3, 5, True), (9, 3, False), (31, 6, True), (32, 2, False),
                                         (33, 3, True), (64, 7, False), (65, 1, True), (97, 3, False)])
def test_columns(oracle_mod, nz, K, wsplit, ver, lim):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    O = oracle_mod
    wsplit = wsplit and lim == "FCT"
    nx, ny = 9, 8
    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(100 * nz + K)
    en = rng.integers(3, nz + 2, size=2 * (nx - 1) * (ny - 1)).astype(np.int32)  # 2..nz layers
    en[0] = nz + 1
    kw = dict(Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb, elem_nlev=en)
    m, om = Mesh(nx, ny, nz + 1, **kw), O.Mesh(nx, ny, nz + 1, **kw)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=1e-3)
    T = synthetic.random_field(m, rng, K)
    dt = 100.0
    eps = 0.1 if K % 2 else None
    we = np.clip(w, -3e-4, 3e-4) if wsplit else None
    wi = w - we if wsplit else None
    vals, vab = np.ascontiguousarray(T.copy()), np.ascontiguousarray(T.copy())
    W = O.Work(om)
    sch = ("MUSCL", ver, lim, 0.8, 0.7)
    for _ in range(2):
        O.analytic_step(om, W, dt, vel, w, vals, vab, [sch] * K, copy_ab=eps is None, ab2_eps=eps, wi=wi, we=we)
    wet = np.arange(nz)[None, :] < (m.get("nlevels_nod2D") - 1)[:, None]
    for precision in ("fp64", "fp64fast"):
        e = engine.TracerAdvection(m, K, precision, "MUSCL", ver, lim, ph=0.8, pv=0.7, copy_ab=eps is None, ab2_eps=eps)
        e.set_tracers(T)
        e.set_velocity(vel, w, we, wi)
        e.step(dt, 2)
        err = np.abs(e.values() - vals)[:, wet].max()
        assert err <= (0.0 if precision == "fp64" else 1e-12 * np.abs(vals).max()), (precision, err)
