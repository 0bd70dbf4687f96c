"""Empirical autotuner of the 2D kernel configuration.

What it chooses among depends on the calls that the configuration is for (the family):
  * "forward": the streaming kernels, one step per launch (tile_rows 16 or 32) and two
    (step_block 2), each with shots_per_cta 1, 2, 4, ... up to 32 and the shot count; and
    the automatic configuration (two steps per launch asked for, no tiling: the resident
    kernel where the library takes it). Each is timed on a short forward (`steps` steps);
  * "gradient": the streaming ones as for a forward, and then the best of them against the
    automatic configuration, both timed as a gradient of some checkpoint segments: the
    library decides for a gradient by another estimate than for a forward;
  * "batch" (models side by side, ``tune_batch``): one or two steps per launch of the streaming
    kernels for all of its models, each at the shots per CTA that the whole batch's work gives
    it (the resident kernel does not run beside others), by the sum of their times as
    gradients. (One choice for all: 5 models of 2 shots take 4.3 ms with either, 4.65 with four
    of one kind and one of the other.)

For the forward of a gradient (and a batch) whose grid asks for the summed update form
("auto" or "summed"), the candidates are timed in that form (the kernels all have it): the
leapfrog form's accumulated rounding is what a gradient from small residuals cannot
afford.

It keeps the fastest, and caches the choice in a JSON file (default
``~/.cache/neuralmech_gb300/autotune.json``, or ``$WAVEFD_AUTOTUNE_CACHE``), by
architecture, grid shape, order, shots, family and kernel set: choices made for another
set of kernels are not taken. The candidate timings use CUDA events on the current
stream after one warm-up call per candidate. 3D columns are the library's choice (by the
grid) and are not tuned.
"""
from __future__ import annotations

import dataclasses
import json
import math
import os
import threading

_lock = threading.Lock()

KERNELS = 2  # the set of kernels and dispatch rules that cached choices hold for: count up with them
FORWARD_AUTOMATIC = {"tile_rows": 0, "shots_per_cta": 0, "step_block": 2}
GRADIENT_AUTOMATIC = {"tile_rows": 0, "shots_per_cta": 0, "step_block": 1}


def cache_path() -> str:
    return os.environ.get("WAVEFD_AUTOTUNE_CACHE",
                          os.path.join(os.path.expanduser("~"), ".cache", "neuralmech_gb300", "autotune.json"))


def _load(path):
    try:
        with open(path) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def _store(path, data):
    os.makedirs(os.path.dirname(path), exist_ok=True)
    tmp = path + ".tmp"
    with open(tmp, "w") as f:
        json.dump(data, f, indent=1, sort_keys=True)
    os.replace(tmp, path)


def problem_key(arch: str, shape, order: int, nshot: int, summed: bool = False, family: str = "forward") -> str:
    return (f"{arch}|{'x'.join(map(str, shape))}|o{order}|s{nshot}" + ("|summed" if summed else "") +
            f"|{family}|k{KERNELS}")


def candidates(nshot: int, summed: bool = False, automatic: bool = True):
    """The streaming configurations, every one with its shots per CTA; with `automatic`
    also the forward's automatic one."""
    spcs = [s for s in (1, 2, 4, 8, 16, 32) if s <= max(1, nshot)]
    if nshot <= 32 and nshot not in spcs:
        spcs.append(nshot)
    one = [{"tile_rows": tr, "shots_per_cta": s, "step_block": 1} for tr in (32, 16) for s in spcs]
    two = [{"tile_rows": 0, "shots_per_cta": s, "step_block": 2} for s in spcs]
    return one + two + ([FORWARD_AUTOMATIC] if automatic else [])


def summed_for(grid, for_gradient: bool) -> bool:
    """Whether the forward that the tuned configuration serves runs in the
    summed form (FP32 fields, lap_store auto, checkpoint adjoint; the
    same rule as the library's WFD_UPDATE_AUTO)."""
    avail = grid.field_format == "fp32" and grid.lap_store == "auto" and grid.adjoint == "checkpoint"
    return avail and (grid.update == "summed" or (grid.update == "auto" and for_gradient))


def select(timings: dict) -> dict:
    """The fastest candidate of {json(candidate): seconds}."""
    best = min(timings, key=timings.get)
    return json.loads(best)


def _times(timer, configs):
    return {json.dumps(c, sort_keys=True): float(timer(c)) for c in configs}


def _cached(path, key, refresh, measure) -> dict:
    """The cache's entry of `key`, which `measure()` makes where it is missing."""
    with _lock:
        cache = _load(path)
        if key in cache and not refresh:
            return cache[key]
    entry = measure()
    with _lock:
        cache = _load(path)
        cache[key] = entry
        _store(path, cache)
    return entry


def tune(grid, nshot: int, vel=None, steps: int = 16, device=None, path: str | None = None,
         timer=None, refresh: bool = False, for_gradient: bool = False) -> dict:
    """Best {tile_rows, shots_per_cta, step_block} for `grid` with `nshot` shots (2D), of
    forwards or of gradients (for_gradient).

    `timer(config) -> seconds` replaces the GPU timing (used by tests)."""
    if grid.ndim != 2:
        return {"tile_rows": 0, "shots_per_cta": 0, "step_block": 0}
    import torch
    arch = "cpu-timer" if timer else torch.cuda.get_device_name(device)
    summed = summed_for(grid, for_gradient)
    key = problem_key(arch, grid.shape, grid.order, nshot, summed, "gradient" if for_gradient else "forward")

    def measure():
        forward = timer or _gpu_timer(dataclasses.replace(grid, update="summed" if summed else "leapfrog"), nshot, vel,
                                      steps, device)
        entry = {"steps": steps, "timings_s": _times(forward, candidates(nshot, summed, automatic=not for_gradient))}
        entry["best"] = select(entry["timings_s"])
        if for_gradient:
            gradient = timer or _gpu_timer(grid, nshot, vel, steps, device, gradient=True)
            entry["gradient_timings_s"] = _times(gradient, [entry["best"], GRADIENT_AUTOMATIC])
            entry["best"] = select(entry["gradient_timings_s"])
        return entry

    return _cached(path or cache_path(), key, refresh, measure)["best"]


def tune_batch(grids, nshots, spcs, vels=None, steps: int = 16, device=None, path: str | None = None,
               timer=None, refresh: bool = False) -> list:
    """`grids` of models that run side by side, the 2D ones of `spcs` shots per CTA > 0 with that
    count and the steps per launch that are the faster for all of them together. Each
    model's two times are cached by themselves.

    `timer(grid, config) -> seconds` replaces the GPU timing (used by tests)."""
    import torch
    arch = "cpu-timer" if timer else torch.cuda.get_device_name(device)
    total = {1: 0.0, 2: 0.0}
    for k, (g, n, spc) in enumerate(zip(grids, nshots, spcs)):
        if g.ndim != 2 or spc <= 0:
            continue

        def measure():
            t = (lambda c: timer(g, c)) if timer else _gpu_timer(g, n, vels[k] if vels else None, steps, device,
                                                                 gradient=True)
            configs = [{"tile_rows": 0, "shots_per_cta": spc, "step_block": sb} for sb in total]
            return {"steps": steps, "gradient_timings_s": _times(t, configs)}

        key = problem_key(arch, g.shape, g.order, n, summed_for(g, True), f"batch{spc}")
        for config, seconds in _cached(path or cache_path(), key, refresh, measure)["gradient_timings_s"].items():
            total[json.loads(config)["step_block"]] += seconds * g.nt / _gradient_steps(g, steps)[0]
    sb = min(total, key=total.get)
    return [dataclasses.replace(g, tile_rows=0, shots_per_cta=spc, step_block=sb) if g.ndim == 2 and spc > 0 else g
            for g, spc in zip(grids, spcs)]


def _gradient_steps(grid, steps: int):
    """(steps, checkpoint interval) of a timed gradient: three of the grid's own segments,
    none kept, which is what the library's estimate goes by."""
    every = grid.ckpt_every if grid.ckpt_every > 0 else max(1, math.ceil(math.sqrt(grid.nt)))
    return min(grid.nt, max(steps, 3 * every)), every


def _gpu_timer(grid, nshot, vel, steps, device, gradient=False):
    import torch

    from .wavefd import misfit_gradient, wave_forward
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    nz, nx = grid.shape
    if vel is None:
        vel = torch.full((nz, nx), 2000.0, device=dev)
    R = grid.order // 2
    every = grid.ckpt_every
    if gradient:
        steps, every = _gradient_steps(grid, steps)
    g = dataclasses.replace(grid, nt=steps, ckpt_every=every, store_levels=0, group_shots=0)
    src = torch.tensor([[[max(R, nz // 8), nx // 2]]] * nshot, dtype=torch.int32)
    rec = torch.tensor([[[max(R, nz // 8), x] for x in range(R, nx - R, max(1, (nx - 2 * R) // 64))]] * nshot,
                       dtype=torch.int32)
    wav = torch.zeros((nshot, steps), device=dev)
    obs = torch.zeros((nshot, steps, rec.shape[1]), device=dev) if gradient else None

    def call(gc):
        if gradient:
            misfit_gradient(vel, wav, src, rec, obs, gc, check=False)
        else:
            wave_forward(vel, wav, src, rec, gc, check=False)

    def timer(cfg):
        gc = dataclasses.replace(g, **cfg)
        call(gc)
        best = math.inf
        for _ in range(3 if gradient else 1):  # (the few rivals of a gradient lie close together)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            call(gc)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) / 1e3)
        return best

    return timer


def tuned(grid, nshot: int, **kw):
    """`grid` with tile_rows / shots_per_cta / step_block replaced by the tuned choice."""
    best = tune(grid, nshot, **kw)
    return dataclasses.replace(grid, **best) if grid.ndim == 2 else grid
