"""Empirical autotuner of the 2D kernel configuration.

What it chooses among depends on the calls that the configuration is for (the family):
  * "forward": the streaming kernels, one step per launch (tile_rows 16 or 32) and two
    (step_block 2), each with shots_per_cta 1, 2, 4, ... up to 32 and the shot count; and
    the automatic configuration (two steps per launch asked for, no tiling: the resident
    kernel where the library takes it). Each is timed on a short forward (`steps` steps);
  * "gradient": the streaming ones as for a forward, and then the best of them against the
    automatic configuration, both timed as a gradient of some checkpoint segments: the
    library decides for a gradient by another estimate than for a forward;
  * "batch" (models side by side): the steps per launch of the best streaming one, timed as a
    forward, with no tiling: the shots per CTA come from the whole batch's work, and the
    resident kernel does not run beside others.

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


def tune(grid, nshot: int, vel=None, steps: int = 16, device=None, path: str | None = None,
         timer=None, refresh: bool = False, for_gradient: bool = False, batch: bool = False) -> dict:
    """Best {tile_rows, shots_per_cta, step_block} for `grid` with `nshot` shots (2D): of
    forwards, of gradients (for_gradient), of models of a batch (batch).

    `timer(config) -> seconds` replaces the GPU timing (used by tests)."""
    if grid.ndim != 2:
        return {"tile_rows": 0, "shots_per_cta": 0, "step_block": 0}
    import torch
    path = path or cache_path()
    arch = "cpu-timer" if timer else torch.cuda.get_device_name(device)
    summed = summed_for(grid, for_gradient or batch)
    family = "batch" if batch else "gradient" if for_gradient else "forward"
    key = problem_key(arch, grid.shape, grid.order, nshot, summed, family)
    with _lock:
        cache = _load(path)
        if key in cache and not refresh:
            return cache[key]["best"]
    gradient = timer
    if timer is None:
        timer = _gpu_timer(dataclasses.replace(grid, update="summed" if summed else "leapfrog"), nshot, vel,
                           steps, device)
        if family == "gradient":
            gradient = _gpu_timer(grid, nshot, vel, steps, device, gradient=True)

    def times(timer, configs):
        return {json.dumps(c, sort_keys=True): float(timer(c)) for c in configs}

    timings = times(timer, candidates(nshot, summed, automatic=family == "forward"))
    best = select(timings)
    entry = {"timings_s": timings, "steps": steps}
    if family == "gradient":
        entry["gradient_timings_s"] = times(gradient, [best, GRADIENT_AUTOMATIC])
        best = select(entry["gradient_timings_s"])
    elif family == "batch":
        best = {"tile_rows": 0, "shots_per_cta": 0, "step_block": best["step_block"]}
    with _lock:
        cache = _load(path)
        cache[key] = dict(entry, best=best)
        _store(path, cache)
    return best


def _gpu_timer(grid, nshot, vel, steps, device, gradient=False):
    import torch

    from .wavefd import misfit_gradient, wave_forward
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    nz, nx = grid.shape
    if vel is None:
        vel = torch.full((nz, nx), 2000.0, device=dev)
    R = grid.order // 2
    every = grid.ckpt_every
    if gradient:  # three of the grid's own checkpoint segments, none kept: what the library's estimate goes by
        every = every if every > 0 else max(1, math.ceil(math.sqrt(grid.nt)))
        steps = min(grid.nt, max(steps, 3 * every))
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
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        call(gc)
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / 1e3

    return timer


def tuned(grid, nshot: int, **kw):
    """`grid` with tile_rows / shots_per_cta / step_block replaced by the tuned choice."""
    best = tune(grid, nshot, **kw)
    return dataclasses.replace(grid, **best) if grid.ndim == 2 else grid
