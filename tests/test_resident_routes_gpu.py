"""The resident kernel on gradients that do run it, which the launch count shows (one launch
per checkpoint segment and sweep): intervals down to the shortest that is dispatched to it, with
segments of a single step at the end (nt = 61 at 5, 6 and 12), every checkpoint format, kept
levels, shot groups, both update forms. Against the streaming kernels: levels, traces and
misfits equal, wavelet gradients 1e-5 (as the resident kernel's other tests), velocity
gradients 1e-5 and twice the streaming kernels' own distance from FP64 (1e-6, but 1e-3 on
402 x 513 cells, where the waves of source and receivers hardly meet within the 61 steps and the
gradient is 1e-13: both kernels carry FP32 rounding of that size into it). And calls on two
streams at once, which share nothing."""
import dataclasses

import numpy as np
import pytest
import torch

from conftest import rel_l2
from helpers import oracle_geometry, small_problem
from test_resident_gpu import _distinct, _launches

pytestmark = pytest.mark.gpu

SHAPES = [dict(shape=(65, 128), nshot=3, order=8, sponge=0), dict(shape=(131, 129), nshot=2, order=4, sponge=10),
          dict(shape=(60, 257), nshot=5, order=2, sponge=8), dict(shape=(402, 513), nshot=1, order=8, sponge=((0, 12), (7, 0)))]


def _args(cuda, kw, seed=5):
    grid, v, wav, src, rec = small_problem(seed=seed, nt=61, nrec=40, nsrc=2, **kw)
    rng = np.random.default_rng(seed)
    src, rec = (_distinct(rng, grid.order // 2, grid.shape, src.shape[0], n) for n in (2, 40))
    obs = rng.standard_normal((src.shape[0], grid.nt, 40)).astype(np.float32)
    return grid, [torch.from_numpy(v).to(cuda), torch.from_numpy(wav).to(cuda), torch.from_numpy(src), torch.from_numpy(rec),
                  torch.from_numpy(obs).to(cuda)]


@pytest.mark.parametrize("kw", SHAPES, ids=lambda k: "x".join(map(str, k["shape"])))
@pytest.mark.parametrize("more", [dict(ckpt_every=6, ckpt_format="fp32"), dict(ckpt_every=6, ckpt_format="bf16", update="leapfrog"),
                                  dict(ckpt_every=6, ckpt_format="i16", step_block=2),
                                  dict(ckpt_every=12, ckpt_format="bf16", step_block=2, store_levels=30),
                                  dict(ckpt_every=9, ckpt_format="i16", update="leapfrog", store_levels=80),
                                  dict(ckpt_every=9, ckpt_format="fp32", update="leapfrog"),
                                  dict(ckpt_every=61, group_shots=2)],
                         ids=lambda m: "_".join(f"{k}{v}" for k, v in m.items()))
def test_gradient(cuda, orc, kw, more):
    from neuralmech_gb300 import misfit_gradient
    grid, args = _args(cuda, kw)
    grid = dataclasses.replace(grid, **more)
    n0 = _launches()
    got = misfit_gradient(*args, grid, want_wavelet=True, want_traces=True)
    n1 = _launches()
    ref = misfit_gradient(*args, dataclasses.replace(grid, shots_per_cta=1), want_wavelet=True, want_traces=True)
    groups = -(-args[2].shape[0] // grid.group_shots) if grid.group_shots else 1
    # three launches a segment, four copies of int16 checkpoints, lists and reductions
    assert n1 - n0 <= groups * (7 * -(-61 // grid.ckpt_every) + 25) and _launches() - n1 > 61
    assert torch.equal(got[3], ref[3])
    assert abs(float(got[0]) / float(ref[0]) - 1) <= 1e-12
    assert rel_l2(got[2].cpu().numpy(), ref[2].cpu().numpy()) <= 1e-5
    plain = dataclasses.replace(grid, shots_per_cta=1, ckpt_format="fp32", store_levels=0, group_shots=0)
    exact = orc.gradient(oracle_geometry(orc, plain, *(a.cpu().numpy() for a in args[:4])), args[4].cpu().numpy())[1]
    floor = rel_l2(misfit_gradient(*args, plain)[1].cpu().numpy(), exact)
    assert rel_l2(got[1].cpu().numpy(), ref[1].cpu().numpy()) <= 1e-5 + 2 * floor


@pytest.mark.parametrize("kw", SHAPES[:3], ids=lambda k: "x".join(map(str, k["shape"])))
def test_the_shortest_interval(cuda, orc, kw):
    """Intervals of 5 steps (4 stream)."""
    test_gradient(cuda, orc, kw, dict(ckpt_every=5, ckpt_format="bf16"))


def test_autograd_pair(cuda):
    """wfd_forward / wfd_backward, each deriving the route for itself."""
    from neuralmech_gb300 import misfit_gradient, wave_forward
    grid, args = _args(cuda, SHAPES[1])
    vel = args[0].clone().requires_grad_(True)
    n0 = _launches()
    t = wave_forward(vel, *args[1:4], grid)
    (g,) = torch.autograd.grad(t, vel, t.detach() - args[4])
    assert _launches() - n0 < 100
    ref = misfit_gradient(*args, grid)[1]
    assert rel_l2(g.cpu().numpy(), ref.cpu().numpy()) <= 1e-6


def test_two_streams(cuda):
    """Gradients of two problems issued to two streams without waiting, several times over:
    each as when it has the GPU to itself."""
    from neuralmech_gb300.wavefd import _misfit_gradient_into, _prepare, _workspace
    calls = []
    for kw, seed in ((SHAPES[3], 5), (dict(shape=(300, 700), nshot=1, order=8, sponge=9), 6)):
        grid, args = _args(cuda, kw, seed)
        call = _prepare(*args[:4], grid, args[2].shape[0])
        outs = [(torch.empty_like(call.vel), torch.zeros((), dtype=torch.float64, device=cuda)) for _ in range(7)]
        calls.append((call, args[4], _workspace(call, True), outs, torch.cuda.Stream()))
    torch.cuda.synchronize()
    for call, obs, ws, outs, _ in calls:
        n0 = _launches()
        _misfit_gradient_into(call, obs, ws, *outs[0])
        assert _launches() - n0 < 61
        torch.cuda.synchronize()
    for k in range(1, 7):
        for call, obs, ws, outs, stream in calls:
            with torch.cuda.stream(stream):
                _misfit_gradient_into(call, obs, ws, *outs[k])
    torch.cuda.synchronize()
    for _, _, _, outs, _ in calls:
        for g, J in outs[1:]:
            assert abs(float(J) / float(outs[0][1]) - 1) <= 1e-12
            assert rel_l2(g.cpu().numpy(), outs[0][0].cpu().numpy()) <= 1e-6
