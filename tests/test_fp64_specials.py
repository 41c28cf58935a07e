"""The bit-exact FP64 step against the oracle where its integer-pipe shortcuts
end: infinities, NaNs, signed zeros, products and doubles that overflow or fall
into the subnormal range, in the tracers, the velocities and the vertical
velocity. Same bits (NaN where the oracle has NaN) in every wet cell.

Left out: a NaN tracer value under the limiter, whose bounds compare in
another order than the reference's element loop (max and min of NaNs depend
on the order)."""
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

INF, NAN = np.inf, np.nan
# name -> factors of T, vel, w; values planted in T (tracer, node, layer), vel (element, layer, component) and w
SPECIALS = {
    "tracer_inf": dict(T=[((1, 17, 2), INF), ((2, 60, 0), INF)]),
    "tracer_-inf": dict(T=[((1, 17, 2), -INF), ((2, 50, 1), INF)]),
    "tracer_nan": dict(T=[((1, 17, 2), NAN)]),
    "velocity_nan": dict(vel=[((31, 1, 0), NAN)]),
    "velocity_inf": dict(vel=[((31, 1, 0), INF), ((60, 0, 1), -INF)]),
    "w_nan": dict(w=[((17, 1), NAN), ((40, 2), NAN), ((23, 3), NAN), ((50, 0), NAN)]),
    "w_inf": dict(w=[((17, 1), INF), ((44, 2), INF)]),
    "w_-inf": dict(w=[((17, 1), -INF), ((44, 2), -INF)]),
    "signed_zeros": dict(T=[((0,), 0.0), ((1,), -0.0)], w=[((slice(None, None, 2),), -0.0)],
                         vel=[((slice(None, None, 3),), 0.0)]),
    "subnormal_products": dict(scale=(1e-310, 1.0, 1e-5)),
    "huge_w": dict(scale=(1.0, 1.0, 1e300)),
    "huge_tracers": dict(scale=(2e306, 1.0, 1.0)),
    "huge_velocity": dict(scale=(1.0, 1e306, 1.0)),
    "large_products": dict(scale=(1e150, 1e10, 1e10)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("closed", [True, False])
@pytest.mark.parametrize("hor,ver,lim", list(itertools.product(["UPW1", "MUSCL", "MFCT"], ["UPW1", "QR4C", "CDIFF", "PPM"],
                                                                ["NONE", "FCT"])))
def test_step_on_special_values(oracle_mod, closed, hor, ver, lim):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    O, nz, K = oracle_mod, 12, 3
    zb = synthetic.stretched_zbar(nz)
    kw = dict(nx=11, ny=9, nl=nz + 1, Lx=11e3, Ly=9e3, depth=-zb[-1], periodic=not closed, orient_left=True, zbar=zb)
    if closed:
        en = np.random.default_rng(3).integers(3, nz + 2, size=2 * 10 * 8).astype(np.int32)
        en[0] = nz + 1
        kw["elem_nlev"] = en
    m, om = Mesh(**kw), O.Mesh(**kw)
    wet = np.arange(nz)[None, :] < (m.get("nlevels_nod2D") - 1)[:, None]
    rng = np.random.default_rng(77)
    vel0, w0 = synthetic.random_flow(m, rng)
    T0 = synthetic.random_field(m, rng, K)
    for name, frozen, ph in itertools.product(SPECIALS, (False, True), (1.0, 0.7)):
        if name == "tracer_nan" and lim == "FCT":
            continue
        s = SPECIALS[name]
        f = s.get("scale", (1.0, 1.0, 1.0))
        T, vel, w = T0 * f[0], vel0 * f[1], w0 * f[2]
        for a, key in ((T, "T"), (vel, "vel"), (w, "w")):
            for at, v in s.get(key, ()):
                a[at] = v
        vals, vab = np.ascontiguousarray(T.copy()), np.ascontiguousarray(T * (1.001 if frozen else 1.0))
        e = engine.TracerAdvection(m, K, "fp64", hor, ver, lim, ph=ph, pv=ph, copy_ab=not frozen)
        e.set_tracers(T, vab if frozen else None)
        e.set_velocity(vel, w)
        e.step(300.0)
        with np.errstate(all="ignore"):
            O.analytic_step(om, O.Work(om), 300.0, vel, w, vals, vab, [(hor, ver, lim, ph, ph)] * K, copy_ab=not frozen)
        got = e.values()
        assert np.array_equal(got[:, wet], vals[:, wet], equal_nan=True), (name, frozen, ph)
