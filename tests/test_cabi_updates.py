"""The C interface uploads only the fields that changed: a velocity handed over
between steps, alone or with the tracer's own values again, gives the oracle's
steps, in both precisions, for layer counts that pad to 4 and that do not."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("nl", [5, 6, 33])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("values_too", [False, True])
def test_velocity_between_steps(oracle_mod, nl, precision, values_too):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import synthetic
    from fesom2_tracer_dwarf_gb300.demo_tracer import FESOMTracerAdvection
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    O = oracle_mod
    nx, ny, nz, dt = 9, 8, nl - 1, 200.0
    om, m = O.Mesh(nx, ny, nl), Mesh(nx, ny, nl, upload=False)
    rng = np.random.default_rng(nl)
    flows = [synthetic.random_flow(m, rng) for _ in range(3)]
    T = synthetic.random_field(m, rng, 1)[0]
    vals, vab = np.ascontiguousarray(T.copy()), np.ascontiguousarray(T.copy())
    dl = np.zeros_like(vals)
    t = FESOMTracerAdvection(verbose=False)
    t.cleanup()
    try:
        assert t.initialize_mpi(0) == 0 and t.generate_analytic_mesh(nx, ny, nl) == 0
        assert t.allocate_tracers(1, nl, m.N) == 0 and t.set_schemes(1, "MUSCL", "CDIFF", "FCT") == 0
        assert t.set_precision(precision) == 0
        assert t.set_values(1, np.asfortranarray(T.T)) == 0
        assert t.init_ale_arrays() == 0 and t.init_for_advection() == 0 and t.init_complete() == 0
        for i, (vel, w) in enumerate(flows):
            uv = np.zeros((nz, m.E, 2), order="F")
            uv.reshape(-1, order="F")[: 2 * nz * m.M] = vel.reshape(-1)
            assert t.set_velocity(uv, np.asfortranarray(w.T)) == 0
            if values_too and i:
                assert t.set_values(1, t.get_tracer_values()) == 0
                vab[...] = vals
            assert t.advect_step(dt) == 0
            O.cabi_step(om, O.Work(om), dt, vel, w, vals, vab, dl, "MUSCL", "CDIFF", "FCT")
        got = t.get_tracer_values().T
    finally:
        t.cleanup()
    err = np.abs(got - vals).max()
    assert err <= (0.0 if precision == "fp64" else 1e-5 * np.abs(vals).max()), err
