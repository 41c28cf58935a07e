"""Launch-configuration autotuner for the tracer-advection step.

The step has five stages (volume fluxes, edge fluxes, FCT low-order solution,
FCT limiting factors, update); the last four have launch knobs that do not
change results (fgb_step_desc.cfg): in the FP32 form the edge kernel (tiled, or
per edge with its block size and layers per lane), the node kernels' columns per
block and layers per lane per pass and, under w_split, the solver; in the FP64
forms the node kernels' columns per block and tracers per chunk. Zeros leave a
choice to the library's rules. The best choice depends on the mesh size, the
number of layers, the tracer count and the precision, so this module times the
candidates of each stage on the caller's own engine (its mesh, fields and
schemes) and keeps the fastest.

The library's own choice is a candidate everywhere: by itself where the others
cannot express it (FP64 chunks need not divide the tracers, the LO stage under
w_split has a rule of its own), else as the values it stands for. In the FP64
forms the edge stage has nothing to choose and is timed once.

Each stage is tuned on its own: a full step fills the workspace, then every
candidate of one stage is run ``reps`` times between CUDA events on the
engine's stream and the median is kept. Re-running the flux, LO and ratio
stages is idempotent; the update stage advances the tracers, so the tracer
fields are saved before tuning and restored afterwards.

Results are cached by (version of the kernels' choices, device, precision, K,
schemes, mesh size) in memory, and in a JSON file when ``cache_path`` (or
FGB_AUTOTUNE_CACHE) names one. Entries of another version stay in the file and
are not used: they chose among other kernels.
"""
from __future__ import annotations

import json
import os
from itertools import product

from . import _lib

EDGE_WARPS = (2, 4, 8)
NODE_WARPS = (1, 2, 4)
CHUNKS = (1, 2, 4)
SLICES = (1, 2)
CHOICES_VERSION = 2  # raise when kernels or defaults change under the knobs

_MEMO: dict = {}


def chunk_candidates(K: int):
    """Tracers per chunk that divide K (others are left to the library's rule)."""
    return [c for c in CHUNKS if K % c == 0]


def stage_candidates(stage: str, K: int, precision: str = "fp64", wsplit: bool = False):
    """Candidate knob values per tuned stage: a list of dicts of cfg index -> value.
    FP64: block size and tracers per chunk. FP32 (one tracer group at a time):
    block size and layers per lane per pass, and under w_split the solver of
    the implicit vertical step (part of the LO stage)."""
    if stage == "hflux":
        if precision == "fp32":
            # + the tiled kernel (node rows staged once per tile; its own launch shape)
            return [{0: w, 7: ns} for w, ns in product(EDGE_WARPS, SLICES)] + [{9: 1}]
        return [{0: w} for w in EDGE_WARPS]
    slot = {"lo": 0, "ratio": 1, "update": 2}[stage]
    if precision == "fp32":
        # the ratio kernel also has variants without shared memory (3; 4: fewer registers); the
        # LO stage a whole-column kernel (3: columns of at most 64 layers; its block shape is
        # fixed, so one candidate; under w_split by the library's rule, see engine_candidates)
        slices = SLICES + ((3, 4) if stage == "ratio" else ())
        cands = [{1 + slot: w, 4 + slot: ns} for w, ns in product(NODE_WARPS, slices)]
        if stage == "lo" and not wsplit:
            cands.append({1 + slot: 4, 4 + slot: 3})
        if stage == "lo" and wsplit:
            cands = [{**c, 8: solver} for c in cands for solver in (0, 1)]
        return cands
    return [{1 + slot: w, 4 + slot: c} for w, c in product(NODE_WARPS, chunk_candidates(K))]


def engine_candidates(stage: str, engine):
    """The candidates ``tune`` times for a stage of an engine: ``stage_candidates``, with the
    library's own choice ({}, all zeros) first where they do not hold it."""
    cands = stage_candidates(stage, engine.K, engine.precision, engine.wi is not None)
    if engine.precision != "fp32":
        return [{}] if stage == "hflux" else [{}, *cands]
    return [{}, *cands] if stage == "lo" and engine.wi is not None else cands


def cache_key(engine) -> str:
    import torch

    m = engine.mesh
    dev = torch.cuda.get_device_name(engine.device)
    return "|".join(str(x) for x in (f"v{CHOICES_VERSION}", dev, engine.precision, engine.K, engine.V, engine.hor, engine.ver,
                                     engine.lim, m.N, m.E, m.nz, "wsplit" if engine.wi is not None else "w"))


def _load_file(path):
    if not path or not os.path.exists(path):
        return {}
    with open(path) as f:
        return json.load(f)


def _save_file(path, table):
    if not path:
        return
    os.makedirs(os.path.dirname(os.path.abspath(path)), exist_ok=True)
    tmp = path + ".tmp"
    with open(tmp, "w") as f:
        json.dump(table, f, indent=1, sort_keys=True)
    os.replace(tmp, path)


def _time_stage(engine, mask, dt, reps):
    import torch

    stream = torch.cuda.current_stream(engine.device)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2 * reps)]
    engine.step(dt, 1, mask)  # warm-up (also sets the shared-memory attribute)
    for r in range(reps):
        ev[2 * r].record(stream)
        engine.step(dt, 1, mask)
        ev[2 * r + 1].record(stream)
    torch.cuda.synchronize(engine.device)
    ts = sorted(ev[2 * r].elapsed_time(ev[2 * r + 1]) for r in range(reps))
    return ts[reps // 2]


def tune(engine, dt: float = 1.0, reps: int = 5, cache_path: str | None = None, force: bool = False):
    """Pick the fastest launch configuration for ``engine`` and apply it.

    Returns {"cfg": [12 ints], "ms": {stage: best ms}, "cached": bool}.
    """
    import torch

    cache_path = cache_path if cache_path is not None else os.environ.get("FGB_AUTOTUNE_CACHE")
    key = cache_key(engine)
    if not force:
        hit = _MEMO.get(key) or _load_file(cache_path).get(key)
        if hit:
            _MEMO[key] = hit
            engine.set_launch(hit["cfg"])
            return dict(hit, cached=True)

    saved = [engine.T.clone()] + ([engine.TA.clone()] if engine.TA is not None else [])
    saved_lo = engine.Tlo.clone() if getattr(engine, "Tlo", None) is not None else None
    fct = engine.lim == "FCT"
    stages = [("hflux", _lib.STAGE_HFLUX)]
    stages += [("lo", _lib.STAGE_LO), ("ratio", _lib.STAGE_RATIO)] if fct else []
    stages += [("update", _lib.STAGE_UPDATE)]
    cfg = [0] * _lib.NCFG
    engine.set_launch(cfg)
    engine.step(dt, 1)  # fills every workspace array the stages read
    best_ms = {}
    for name, mask in stages:
        best = None
        for cand in engine_candidates(name, engine):
            trial = list(cfg)
            for i, v in cand.items():
                trial[i] = v
            engine.set_launch(trial)
            ms = _time_stage(engine, mask, dt, reps)
            if best is None or ms < best[0]:
                best = (ms, cand)
        for i, v in best[1].items():
            cfg[i] = v
        best_ms[name] = best[0]
    engine.set_launch(cfg)
    engine.T.copy_(saved[0])
    if engine.TA is not None:
        engine.TA.copy_(saved[1])
    if saved_lo is not None:
        engine.Tlo.copy_(saved_lo)
    torch.cuda.synchronize(engine.device)
    result = {"cfg": cfg, "ms": best_ms}
    _MEMO[key] = result
    if cache_path:
        table = _load_file(cache_path)
        table[key] = result
        _save_file(cache_path, table)
    return dict(result, cached=False)
