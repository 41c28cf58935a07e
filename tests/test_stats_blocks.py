"""Tracer statistics at the edges of their block split: one block (which
writes the result itself), two, and the largest block count with one value per
thread and with more; FP64 and the grouped FP32 layout."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("precision,V", [("fp64", 1), ("fp32", 2), ("fp32", 4)])
@pytest.mark.parametrize("nx,ny,nl", [(3, 3, 3), (17, 9, 3), (18, 9, 3), (129, 129, 17), (130, 129, 17)])
def test_stats_block_split(nx, ny, nl, precision, V):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    m = Mesh(nx, ny, nl, periodic=True)
    K = 4
    T = 1e6 + np.random.default_rng(nx * nl).standard_normal((K, m.N, m.nz))
    if precision == "fp32":
        T = T.astype(np.float32).astype(np.float64)
    e = engine.TracerAdvection(m, K, precision, tracer_vec=V)
    e.set_tracers(T)
    st = e.stats()
    for t in range(K):
        v = T[t].ravel()
        exact = math.fsum(v)
        assert st[t, 0] == v.min() and st[t, 1] == v.max() and st[t, 3] == 0
        # every addition is compensated: the sum is the exact one to a few units in the last place
        assert abs(st[t, 2] - exact) <= 4 * math.ulp(exact)
