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


@pytest.mark.parametrize("fast,steps", [({"tile_rows": 16, "shots_per_cta": 2, "step_block": 1}, 1),
                                        ({"tile_rows": 0, "shots_per_cta": 1, "step_block": 2}, 2)])
def test_batch_keeps_the_steps_per_launch(tmp_path, fast, steps):
    best, seen = _tune(tmp_path, lambda c: c == fast, for_gradient=True, batch=True)
    assert not any(map(_automatic, seen))
    assert best == {"tile_rows": 0, "shots_per_cta": 0, "step_block": steps}


def test_the_cache_is_by_family_and_kernel_set(tmp_path, monkeypatch):
    old = {"tile_rows": 16, "shots_per_cta": 1, "step_block": 1}
    cache = tmp_path / "cache.json"
    keys = {f"cpu-timer|256x512|o8|s12{s}": {"best": old} for s in ("", "|summed")}  # (as they were once written)
    cache.write_text(json.dumps(keys))
    for kw in ({}, dict(for_gradient=True), dict(for_gradient=True, batch=True)):
        assert _tune(tmp_path, _automatic, **kw)[1], kw   # timed ...
        assert not _tune(tmp_path, _automatic, **kw)[1], kw  # ... once
    monkeypatch.setattr(autotune, "KERNELS", autotune.KERNELS + 1)
    assert _tune(tmp_path, _automatic)[1]


@pytest.mark.gpu
@pytest.mark.parametrize("family", [dict(), dict(for_gradient=True), dict(for_gradient=True, batch=True)])
def test_on_the_gpu(cuda, tmp_path, family):
    best = autotune.tune(Grid((130, 250), (10.0, 10.0), 1e-3, 60), 3, steps=4, path=str(tmp_path / "c.json"), **family)
    assert set(best) == {"tile_rows", "shots_per_cta", "step_block"}
    assert not family.get("batch") or _automatic(best)
