"""Edges whose layer window of triangle gradients comes from a restart record
that no mesh builder would write: a window that starts above the surface
(ulevels_nod2D_max = 0) or ends there (nlevels_nod2D_min = 0), and one that
reaches below its up- or downwind triangle (nlevels_nod2D_min too deep). CPU:
the window function over every small window. GPU: the step's values."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from fesom2_tracer_dwarf_gb300.demo_tracer import FESOMTracerAdvection

from test_restart import MESH, frame, parse_tracer, read_record

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fesom2_tracer_dwarf_gb300", "csrc")


def test_windows_hold_the_layers_they_stand_for(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    exe = str(tmp_path / "edge_window")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, os.path.join(HERE, "edge_window_check.cpp"), "-o", exe],
                   check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "0"


torch = pytest.importorskip("torch")


def _offsets(payload):
    """Byte offset and size of every field of a t_mesh record."""
    out, p = {}, 0
    for name, kind, rank in MESH:
        dims = np.frombuffer(payload, "<i4", rank, p)
        n = int(np.prod(dims)) if rank and (dims > 0).all() else (0 if rank else 1)
        p += 4 * rank
        out[name] = (p, n)
        p += n * (8 if kind == "r8" else 4)
    assert p == len(payload)
    return out


def _patch(path, **fields):
    payload = read_record(path)
    at = _offsets(payload)
    b = bytearray(payload)
    for name, v in fields.items():
        p, n = at[name]
        b[p : p + 4 * n] = np.broadcast_to(np.asarray(v, "<i4"), (n,)).tobytes()
    open(path, "wb").write(frame(bytes(b), 1 << 30))


@pytest.fixture()
def tracer():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    t = FESOMTracerAdvection(verbose=False)
    t.cleanup()
    yield t
    t.cleanup()


def _restart(t, path, schemes, nl=12):
    assert t.generate_analytic_mesh(9, 8, nl, periodic=False) == 0
    nz, N, E = nl - 1, t.nod2D, t.edge2D
    rng = np.random.default_rng(8)
    assert t.allocate_tracers(1, nl, N) == 0
    assert t.set_values(1, np.asfortranarray(rng.uniform(1, 2, (nz, N)))) == 0
    assert t.set_schemes(1, *schemes, 0.9, 0.8) == 0
    assert t.set_velocity(np.asfortranarray(rng.uniform(-0.1, 0.1, (nz, E, 2))),
                          np.asfortranarray(rng.uniform(-1e-5, 1e-5, (nl, N)))) == 0
    assert t.finalize(str(path)) == 0
    t.cleanup()


def _step(t, path, precision):
    t.cleanup()
    assert t.initialize(str(path)) == 0
    assert t.lib.tracer_set_precision(precision) == 0
    for _ in range(2):
        assert t.advect_step(60.0) == 0
    v = t.get_tracer_values().copy()
    t.cleanup()
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("schemes", [("MUSCL", "PPM", "FCT"), ("MFCT", "UPW1", "NONE")])
@pytest.mark.parametrize("precision", [0, 1])
def test_windows_from_above_the_surface(tracer, tmp_path, schemes, precision):
    _restart(tracer, tmp_path / "a", schemes)
    for name in "bcd":
        shutil.copytree(tmp_path / "a", tmp_path / name)
    # a window that starts at layer 0 holds the layers of one that starts at layer 1
    _patch(tmp_path / "b" / "np1" / "t_mesh.0", ulevels_nod2D_max=0)
    assert np.array_equal(_step(tracer, tmp_path / "b", precision), _step(tracer, tmp_path / "a", precision))
    # one that also ends there is empty, as one that ends at layer 1: mean gradients at every layer
    _patch(tmp_path / "c" / "np1" / "t_mesh.0", ulevels_nod2D_max=0, nlevels_nod2D_min=0)
    _patch(tmp_path / "d" / "np1" / "t_mesh.0", nlevels_nod2D_min=1)
    empty = _step(tracer, tmp_path / "d", precision)
    assert np.array_equal(_step(tracer, tmp_path / "c", precision), empty)
    assert not np.array_equal(empty, _step(tracer, tmp_path / "a", precision))


@pytest.mark.gpu
@pytest.mark.parametrize("schemes", [("MUSCL", "PPM", "FCT"), ("MFCT", "QR4C", "FCT"), ("MUSCL", "CDIFF", "NONE")])
def test_windows_below_a_triangle(tracer, tmp_path, schemes):
    """Shallow elements beside deep ones, and a record whose windows go on below
    them: the gradients there come from the nodes' values, in FP64 as in FP32."""
    nl = 12
    _restart(tracer, tmp_path, schemes, nl)
    path = tmp_path / "np1" / "t_mesh.0"
    payload = read_record(path)
    at = _offsets(payload)
    get = lambda name, dt="<i4", s=4: np.frombuffer(payload, dt, at[name][1], at[name][0])  # noqa: E731
    M, N = at["nlevels"][1], at["nlevels_nod2D"][1]
    nlev = np.random.default_rng(4).integers(4, nl + 1, M).astype("<i4")
    en = get("elem2D_nodes").reshape(M, 3) - 1
    deepest = np.zeros(N, "<i4")
    np.maximum.at(deepest, en.reshape(-1), np.repeat(nlev, 3))
    _patch(path, nlevels=nlev, nlevels_nod2D=deepest, nlevels_nod2D_min=deepest)
    tri = parse_tracer(read_record(tmp_path / "np1" / "t_tracer.0"))["work%edge_up_dn_tri"] - 1
    edges = get("edges").reshape(-1, 2) - 1
    both = (tri >= 0).all(axis=0)
    assert (np.minimum(deepest[edges[both, 0]], deepest[edges[both, 1]]) > nlev[tri[:, both]].min(axis=0)).any()
    a, b = _step(tracer, tmp_path, 0), _step(tracer, tmp_path, 1)
    wet = np.arange(nl - 1)[:, None] < deepest[None, :] - 1
    assert np.abs(a - b)[wet].max() <= 1e-5 * np.abs(a[wet]).max()
