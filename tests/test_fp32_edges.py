"""FP32 edge stages against the oracle where their splits can go wrong: layer
counts whose last pass of 32 leaves 4, 8, 12, 16 or 20 layers (several edges
per warp), ragged columns and coasts (layers with mean gradients in a kernel of
their own, runs of up to eight), every group width, T_AB separate or not, and
velocities on an address that 16-byte loads cannot take."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

REL_TOL = 1e-5  # the FP32 form's bar against FP64 (relative max-norm)


@pytest.mark.gpu
@pytest.mark.parametrize("hor,lim", [("UPW1", "FCT"), ("MUSCL", "FCT"), ("MFCT", "FCT"), ("MUSCL", "NONE")])
@pytest.mark.parametrize("nz,K,V,frozen,shift", [(2, 1, 1, False, 0), (4, 4, 4, True, 0), (9, 4, 4, False, 2),
                                                 (33, 3, 1, False, 0), (40, 2, 2, True, 2), (44, 4, 4, False, 0),
                                                 (47, 6, 2, False, 0), (52, 4, 4, True, 0), (64, 8, 4, False, 0),
                                                 (70, 4, 4, False, 0)])
def test_edge_stages(oracle_mod, nz, K, V, frozen, shift, hor, lim):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    O = oracle_mod
    nx, ny = 11, 9
    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(7 * nz + K)
    en = rng.integers(3, nz + 2, size=2 * (nx - 1) * (ny - 1)).astype(np.int32)  # 2..nz layers
    en[0] = nz + 1
    kw = dict(Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb, elem_nlev=en)
    m, om = Mesh(nx, ny, nz + 1, **kw), O.Mesh(nx, ny, nz + 1, **kw)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=1e-3)
    T = synthetic.random_field(m, rng, K)
    TA = T + rng.normal(0, 0.05, size=T.shape) if frozen else T
    vals, vab = np.ascontiguousarray(T.copy()), np.ascontiguousarray(TA.copy())
    O.analytic_step(om, O.Work(om), 100.0, vel, w, vals, vab, [(hor, "UPW1", lim, 0.7, 1.0)] * K, copy_ab=not frozen)
    e = engine.TracerAdvection(m, K, "fp32", hor, "UPW1", lim, ph=0.7, copy_ab=not frozen, tracer_vec=V)
    if shift:  # 8-byte aligned velocities
        pad = torch.zeros(e.vel.numel() + 4, dtype=e.dtype, device=e.device)
        e.vel = pad[shift:shift + e.vel.numel()].view(e.vel.shape)
        assert e.vel.data_ptr() % 16 == 8
    e.set_tracers(T, TA if frozen else None)
    e.set_velocity(vel, w)
    e.step(100.0)
    wet = np.arange(nz)[None, :] < (m.get("nlevels_nod2D") - 1)[:, None]
    assert np.abs(e.values() - vals)[:, wet].max() <= REL_TOL * np.abs(vals).max()
