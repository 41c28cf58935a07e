"""FP64 node kernels over tracer counts, layer counts and schemes whose chunks
differ (shared memory for the kernels' blocks, rounds of a warp, a remainder):
each tracer's values are the bits it has when it is stepped alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
@pytest.mark.parametrize("nz,K,ver,frozen", [(48, 8, "QR4C", True), (48, 7, "QR4C", True), (64, 4, "QR4C", False),
                                             (64, 5, "QR4C", True), (90, 3, "QR4C", True), (64, 6, "PPM", True),
                                             (33, 5, "CDIFF", False)])
def test_chunks_do_not_change_a_tracer(precision, nz, K, ver, frozen):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    zb = synthetic.stretched_zbar(nz)
    rng = np.random.default_rng(nz + K)
    en = rng.integers(3, nz + 2, size=2 * 8 * 7).astype(np.int32)
    en[0] = nz + 1
    m = Mesh(9, 8, nz + 1, Lx=9e3, Ly=8e3, depth=-zb[-1], periodic=False, orient_left=True, zbar=zb, elem_nlev=en)
    vel, w = synthetic.random_flow(m, rng)
    T = synthetic.random_field(m, rng, K)

    def step(k):
        e = engine.TracerAdvection(m, len(k), precision, "MUSCL", ver, "FCT", copy_ab=not frozen)
        e.set_tracers(T[k], T[k] * 1.001 if frozen else None)
        e.set_velocity(vel, w)
        e.step(100.0, 2)
        return e.values()

    together = step(list(range(K)))
    for k in range(K):
        assert np.array_equal(together[k], step([k])[0]), k
