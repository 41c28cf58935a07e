"""The autotuner times the library's own choice too, so a tuned engine does not
lose a default that its candidate lists cannot express."""
from types import SimpleNamespace

import numpy as np
import pytest

from fesom2_tracer_dwarf_gb300 import autotune


def _engine(precision, K, wsplit):
    return SimpleNamespace(precision=precision, K=K, wi=object() if wsplit else None)


@pytest.mark.parametrize("K", [1, 3, 5, 6, 8])
@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
def test_fp64_default_is_a_candidate(precision, K):
    e = _engine(precision, K, False)
    for stage in ("lo", "ratio", "update"):
        cands = autotune.engine_candidates(stage, e)
        assert cands[0] == {} and cands[1:] == autotune.stage_candidates(stage, K, precision)
    assert autotune.engine_candidates("hflux", e) == [{}]  # no knob: one timing


def test_fp32_default_is_a_candidate():
    lo = autotune.engine_candidates("lo", _engine("fp32", 4, True))
    assert lo[0] == {} and lo[1:] == autotune.stage_candidates("lo", 4, "fp32", wsplit=True)
    # without w_split the default is one of the listed shapes
    assert {1: 4, 4: 3} in autotune.engine_candidates("lo", _engine("fp32", 4, False))
    assert {9: 1} in autotune.engine_candidates("hflux", _engine("fp32", 4, False))


torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("precision,K,wsplit", [("fp64", 3, False), ("fp64", 6, True), ("fp64fast", 5, False),
                                                ("fp32", 4, True)])
def test_tuned_engine_steps_as_an_untuned_one(tmp_path, precision, K, wsplit):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from fesom2_tracer_dwarf_gb300 import engine, synthetic
    from fesom2_tracer_dwarf_gb300.mesh import Mesh

    m = Mesh(30, 26, 12, periodic=True, orient_left=True)
    rng = np.random.default_rng(12)
    vel, w = synthetic.streamfunction_flow(m, rng, 200.0, cfl=0.5)
    T = synthetic.random_field(m, rng, K)
    we = 0.5 * w
    out = []
    for tuned in (True, False):
        e = engine.TracerAdvection(m, K, precision, "MUSCL", "QR4C", "FCT", copy_ab=True)
        e.set_tracers(T)
        e.set_velocity(vel, w, we if wsplit else None, w - we if wsplit else None)
        if tuned:
            path = tmp_path / "t.json"
            # a choice cached for other kernels is not used
            stale = autotune.cache_key(e).split("|", 1)[1]
            autotune._save_file(str(path), {stale: {"cfg": [2, 1, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0], "ms": {}}})
            res = autotune.tune(e, dt=200.0, reps=2, cache_path=str(path))
            assert not res["cached"] and set(res["ms"]) == {"hflux", "lo", "ratio", "update"}
            assert np.array_equal(e.values(), T if precision != "fp32" else T.astype(np.float32))
            assert autotune.tune(e, dt=200.0, cache_path=str(path))["cached"]
            if precision != "fp32":
                assert res["cfg"][0] == 0
        e.step(200.0, 2)
        out.append(e.values())
    if precision == "fp32":
        assert np.abs(out[0] - out[1]).max() <= 1e-5 * np.abs(out[1]).max()
    else:
        assert np.array_equal(out[0], out[1])
