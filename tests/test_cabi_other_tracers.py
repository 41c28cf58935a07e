"""tracer_set_values of a tracer other than the first between two steps of the C
interface, which advance the first one: its device values stay, so the steps are
those of an uninterrupted run, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_setting_another_tracer_keeps_the_steps(precision):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import synthetic
    from fesom2_tracer_dwarf_gb300.demo_tracer import FESOMTracerAdvection
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    nx, ny, nl, dt = 9, 8, 7, 200.0
    nz = nl - 1
    m = Mesh(nx, ny, nl, upload=False)
    rng = np.random.default_rng(3)
    vel, w = synthetic.random_flow(m, rng)
    T = synthetic.random_field(m, rng, 2)
    uv = np.zeros((nz, m.E, 2), order="F")
    uv.reshape(-1, order="F")[: 2 * nz * m.M] = vel.reshape(-1)
    out = []
    for between in (None, T[1] + 1.0):
        t = FESOMTracerAdvection(verbose=False)
        t.cleanup()
        try:
            assert t.initialize_mpi(0) == 0 and t.generate_analytic_mesh(nx, ny, nl) == 0
            assert t.allocate_tracers(2, nl, m.N) == 0 and t.set_schemes(1, "MUSCL", "PPM", "FCT") == 0
            assert t.set_precision(precision) == 0
            for i in range(2):
                assert t.set_values(i + 1, np.asfortranarray(T[i].T)) == 0
            assert t.set_velocity(uv, np.asfortranarray(w.T)) == 0
            assert t.init_ale_arrays() == 0 and t.init_for_advection() == 0 and t.init_complete() == 0
            assert t.advect_step(dt) == 0
            if between is not None:
                assert t.set_values(2, np.asfortranarray(between.T)) == 0
            assert t.advect_step(dt) == 0
            out.append(t.get_tracer_values())
        finally:
            t.cleanup()
    assert np.array_equal(out[0], out[1])
