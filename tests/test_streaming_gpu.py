"""The streaming 2D kernels on problems that the dispatch gives to the resident kernel: the
tests that were written around their tiles (seams, extended regions, checkpoints at odd
steps, the recompute on a second stream, the random sweep, precision at the benchmark's
grid) run again with shots_per_cta given, at 1, 2 and 3 shots per CTA. The bounds are those
tests' own. Every forward and gradient is checked to have launched its steps' kernels: the
resident kernel launches once per checkpoint segment."""
import dataclasses
import inspect
import itertools

import pytest

import test_field_storage_gpu
import test_forward_gpu
import test_gradient_gpu
import test_precision_gpu
import test_sweep_gpu

pytestmark = pytest.mark.gpu


def _cases(*functions):
    """(function, its parametrised arguments) for every case of the functions."""
    out = []
    for f in functions:
        axes = []
        for mark in getattr(f, "pytestmark", []):
            if mark.name == "parametrize":
                names = [n.strip() for n in mark.args[0].split(",")]
                axes.append([dict(zip(names, v if len(names) > 1 else (v,))) for v in mark.args[1]])
        for combo in itertools.product(*axes):
            kw = {k: v for part in combo for k, v in part.items()}
            out.append(pytest.param(f, kw, id=f"{f.__name__[5:]}-" + "-".join(str(v)[:18] for v in kw.values())))
    return out


def _counted(call):
    """`call` (grid last of its positional arguments) that checks how many kernels it launched."""
    from neuralmech_gb300 import _lib

    def counted(*args, **kw):
        grid = args[-1]
        n0 = int(_lib.load().wfd_kernel_launches())
        out = call(*args, **kw)
        n = int(_lib.load().wfd_kernel_launches()) - n0
        assert grid.shots_per_cta > 0 and n >= grid.nt // max(1, grid.step_block)
        return out
    return counted


@pytest.fixture
def streaming(monkeypatch):
    """Gives the problems that a test module builds an explicit shots_per_cta."""
    import neuralmech_gb300
    from neuralmech_gb300 import wavefd
    for module, name in itertools.product((neuralmech_gb300, wavefd), ("wave_forward", "wave_forward_final", "misfit_gradient")):
        if hasattr(module, name):
            monkeypatch.setattr(module, name, _counted(getattr(wavefd, name)))

    def use(module, spc):
        build = module.small_problem
        monkeypatch.setattr(module, "small_problem", lambda *a, **k: build(*a, **dict(k, spc=spc)))
    return use


def _run(f, kw, cuda, orc):
    f(**dict(kw, **{k: v for k, v in (("cuda", cuda), ("orc", orc)) if k in inspect.signature(f).parameters}))


@pytest.mark.parametrize("spc", [1, 3])
@pytest.mark.parametrize("f,kw", _cases(
    test_forward_gpu.test_forward_two_step_blocking,
    test_gradient_gpu.test_gradient_two_step_blocking,
    test_gradient_gpu.test_two_step_matches_one_step_autograd,
    test_gradient_gpu.test_summed_two_step_matches_one_step,
    test_gradient_gpu.test_kept_levels_match_recompute,
    test_gradient_gpu.test_block_float_levels,
    test_gradient_gpu.test_u_store_matches_lap_store,
    test_gradient_gpu.test_adjoint_dot_product,
    test_gradient_gpu.test_shot_groups_match_one_batch))
def test_targeted(cuda, orc, streaming, f, kw, spc):
    streaming(test_forward_gpu, spc)
    streaming(test_gradient_gpu, spc)
    _run(f, kw, cuda, orc)


@pytest.mark.parametrize("f,kw", _cases(test_forward_gpu.test_forward_register_window,
                                        test_field_storage_gpu.test_forward_storage_error))
def test_three_shots_per_cta(cuda, orc, streaming, f, kw):
    """The register window and the reduced-precision fields at a count that is no power of two."""
    streaming(test_forward_gpu, 3)
    streaming(test_field_storage_gpu, 3)
    _run(f, kw, cuda, orc)


@pytest.mark.parametrize("case", [c for c in test_sweep_gpu.CASES if c["ndim"] == 2], ids=test_sweep_gpu._ids)
def test_sweep(cuda, orc, streaming, case):
    streaming(test_sweep_gpu, 1 + case["seed"] % 3)
    test_sweep_gpu.test_sweep_matches_oracle(cuda, orc, case)


def test_precision_at_fwi1024(cuda, orc, streaming, monkeypatch):
    from neuralmech_gb300 import synth
    build = synth.workload

    def workload(name):
        w = build(name)
        return dataclasses.replace(w, grid=dataclasses.replace(w.grid, shots_per_cta=2))
    monkeypatch.setattr(synth, "workload", workload)
    test_precision_gpu.test_fwi1024_two_shots_against_fp64(cuda, orc)
