"""What the tuner times and returns for forwards, gradients and batches: nothing is chosen
on the time of a kernel that the calls will not run, and a choice made for other kernels
is not taken from the cache."""
import json

import pytest

from neuralmech_gb300 import Grid, autotune

GRID = Grid((256, 512), (10.0, 10.0), 1e-3, 100)


def _tune(path, prefer, **kw):
    """The result and the configurations timed, with `prefer(config)` the fastest."""
    seen = []

    def timer(cfg):
        seen.append(cfg)
        return 1.0 if prefer(cfg) else 2.0

    return autotune.tune(GRID, 12, timer=timer, path=str(path / "cache.json"), **kw), seen


def _automatic(c):
    return c["tile_rows"] == 0 and c["shots_per_cta"] == 0


def test_forward_times_the_automatic_configuration(tmp_path):
    best, seen = _tune(tmp_path, _automatic)
    assert best == autotune.FORWARD_AUTOMATIC and sum(map(_automatic, seen)) == 1


def test_gradient_times_it_against_the_best_streaming_one(tmp_path):
    fast = {"tile_rows": 0, "shots_per_cta": 4, "step_block": 2}
    best, seen = _tune(tmp_path, lambda c: c == fast, for_gradient=True)
    assert best == fast and seen[-2:] == [fast, autotune.GRADIENT_AUTOMATIC] and not any(map(_automatic, seen[:-2]))
    best, _ = _tune(tmp_path, _automatic, for_gradient=True, refresh=True)
    assert best == autotune.GRADIENT_AUTOMATIC and best["step_block"] == 1  # (the summed form of the differences)


def test_batch_takes_the_steps_per_launch_of_the_least_sum(tmp_path):
    import dataclasses
    deep = Grid((20, 30, 40), (10.0,) * 3, 1e-3, 50)
    small, large = dataclasses.replace(GRID, shape=(100, 90)), dataclasses.replace(GRID, tile_rows=16)
    seconds = {(small, 1): 3.0, (small, 2): 1.0, (large, 1): 1.0, (large, 2): 2.0}
    seen = []

    def timer(grid, cfg):
        seen.append((grid.shape, cfg["tile_rows"], cfg["shots_per_cta"]))
        return seconds[grid, cfg["step_block"]]

    def run(*grids):
        spcs = [0 if g.ndim == 3 else 5 if g == small else 7 for g in grids]
        return autotune.tune_batch(grids, [12] * len(grids), spcs, timer=timer, path=str(tmp_path / "cache.json"))

    out = run(small, large, deep)
    assert [g.step_block for g in out[:2]] == [2, 2] and out[2] == deep
    assert [(g.tile_rows, g.shots_per_cta) for g in out[:2]] == [(0, 5), (0, 7)]
    assert seen == [(small.shape, 0, 5)] * 2 + [(large.shape, 0, 7)] * 2
    assert [g.step_block for g in run(large, large)] == [1, 1] and len(seen) == 4  # (cached)


def test_the_cache_is_by_family_and_kernel_set(tmp_path, monkeypatch):
    old = {"tile_rows": 16, "shots_per_cta": 1, "step_block": 1}
    cache = tmp_path / "cache.json"
    keys = {f"cpu-timer|256x512|o8|s12{s}": {"best": old} for s in ("", "|summed")}  # (as they were once written)
    cache.write_text(json.dumps(keys))
    for kw in ({}, dict(for_gradient=True)):
        assert _tune(tmp_path, _automatic, **kw)[1], kw   # timed ...
        assert not _tune(tmp_path, _automatic, **kw)[1], kw  # ... once
    monkeypatch.setattr(autotune, "KERNELS", autotune.KERNELS + 1)
    assert _tune(tmp_path, _automatic)[1]


@pytest.mark.gpu
@pytest.mark.parametrize("family", [dict(), dict(for_gradient=True)])
def test_on_the_gpu(cuda, tmp_path, family):
    grid = Grid((130, 250), (10.0, 10.0), 1e-3, 60)
    best = autotune.tune(grid, 3, steps=4, path=str(tmp_path / "c.json"), **family)
    assert set(best) == {"tile_rows", "shots_per_cta", "step_block"}


@pytest.mark.gpu
def test_batch_on_the_gpu(cuda, tmp_path):
    grid = Grid((130, 250), (10.0, 10.0), 1e-3, 60)
    out = autotune.tune_batch([grid, grid], [3, 4], [2, 2], steps=4, path=str(tmp_path / "c.json"))
    assert [(g.tile_rows, g.shots_per_cta) for g in out] == [(0, 2)] * 2 and out[0].step_block == out[1].step_block
