"""Values below a column's bottom do not enter the fluxes: with the padded
arrays of T (and T_AB) filled with NaN or infinity there, as a land mask may
be, the wet values are the same bits as with zeros. Closed ragged basins, whose
coasts and bottom steps take mean gradients over elements of different depths.
FP64 with and without the limiter, FP32 without it (its low-order stage weights
the layers below an edge's bottom with a volume flux of zero)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


FORMS = [("fp64", 1, []), ("fp64fast", 1, []), ("fp32", 4, []), ("fp32", 2, []), ("fp32", 1, []),
         ("fp32", 4, [8, 0, 0, 0, 0, 0, 0, 1]), ("fp32", 2, [4, 0, 0, 0, 0, 0, 0, 2])]
SCHEMES = [("MUSCL", "PPM", "FCT", False), ("MFCT", "QR4C", "FCT", True), ("MUSCL", "CDIFF", "NONE", True),
           ("MFCT", "PPM", "NONE", False), ("UPW1", "UPW1", "NONE", False)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision,V,cfg,hor,ver,lim,frozen",
                         [f + s for f in FORMS for s in SCHEMES if f[0] != "fp32" or s[2] == "NONE"])
def test_fill_below_the_bottom_is_not_read(precision, V, cfg, hor, ver, lim, frozen):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    nx, ny, nz, K = 11, 9, 37, 4
    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(29)
    en = rng.integers(3, nz + 2, size=2 * (nx - 1) * (ny - 1)).astype(np.int32)
    en[0] = nz + 1
    m = Mesh(nx, ny, nz + 1, Lx=nx * 1e3, Ly=ny * 1e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb,
             elem_nlev=en)
    vel, w = synthetic.random_flow(m, rng, umax=0.3, wmax=1e-3)
    T = synthetic.random_field(m, rng, K)
    kw = dict(tracer_vec=V) if precision == "fp32" else {}
    dry = torch.arange(m.LZ)[None, :] >= torch.as_tensor(m.get("nlevels_nod2D")).long()[:, None] - 1
    out = []
    for fill in (0.0, float("nan"), float("inf")):
        e = engine.TracerAdvection(m, K, precision, hor, ver, lim, ph=0.8, pv=0.7, copy_ab=not frozen, **kw)
        e.set_launch(cfg)
        e.set_tracers(T)
        e.set_velocity(vel, w)
        for t in (e.T, e.TA):
            if t is not None:
                t[(slice(None), dry.to(t.device))] = fill
        e.step(100.0)
        out.append(e.values()[:, ~dry[:, :nz].numpy()])
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[1], out[0]) and np.array_equal(out[2], out[0])
