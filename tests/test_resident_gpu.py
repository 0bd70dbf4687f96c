"""The resident 2D kernel (fields on the chip for many steps) against the
streaming kernels, which an explicit shots_per_cta asks for. Both evaluate the
same expressions in the same order, so levels, traces and misfits agree value
for value; the gradients differ by the order of their FP32 sums and by the form
of L u (1e-5, the bound the streaming kernels are held to among themselves).
Sizes lie at the edges of the 128-column tiles and of the row splits.
"""
import ctypes
import dataclasses

import numpy as np
import pytest
import torch

from conftest import rel_l2
from helpers import small_problem

pytestmark = pytest.mark.gpu


def _launches():
    from neuralmech_gb300 import _lib
    return int(_lib.load().wfd_kernel_launches())


def _distinct(rng, R, shape, nshot, n):
    """n different interior cells per shot (sums at one cell have no fixed order)."""
    nz, nx = shape[0] - 2 * R, shape[1] - 2 * R
    out = np.stack([rng.permutation(nz * nx)[:n] for _ in range(nshot)])
    return np.stack([R + out // nx, R + out % nx], -1).astype(np.int32)


CASES = [
    dict(shape=(24, 127), nshot=1, order=8, sponge=6),
    dict(shape=(65, 128), nshot=3, order=8, sponge=0),
    dict(shape=(131, 129), nshot=2, order=4, sponge=10),
    dict(shape=(33, 257), nshot=5, order=2, sponge=8),
    dict(shape=(402, 513), nshot=2, order=8, sponge=((0, 12), (7, 0))),
    dict(shape=(150, 300), nshot=40, order=8, sponge=12),
    dict(shape=(1030, 1025), nshot=1, order=8, sponge=20, nt=41),
    dict(shape=(2040, 2047), nshot=1, order=8, sponge=20, nt=21),
]


@pytest.mark.parametrize("kw", CASES, ids=lambda k: "x".join(map(str, k["shape"])) + f"_{k['nshot']}shots_o{k['order']}")
@pytest.mark.parametrize("sb", [0, 2])
def test_resident_forward_equals_streaming(cuda, kw, sb):
    from neuralmech_gb300.wavefd import wave_forward_final
    kw = dict(dict(nt=70, nrec=33, nsrc=1), **kw)
    grid, v, wav, src, rec = small_problem(seed=3, step_block=sb, **kw)
    args = (torch.from_numpy(v).to(cuda), torch.from_numpy(wav).to(cuda), torch.from_numpy(src), torch.from_numpy(rec))
    n0 = _launches()
    t, u = wave_forward_final(*args, grid)
    assert _launches() - n0 < grid.nt  # (the streaming kernels launch once per step or two)
    ts, us = wave_forward_final(*args, dataclasses.replace(grid, shots_per_cta=1))
    assert float(us.abs().max()) > 0
    assert torch.equal(t, ts) and torch.equal(u, us)


@pytest.mark.parametrize("kw", [
    dict(shape=(65, 128), nshot=3, order=8, sponge=0, ckpt_format="fp32"),
    dict(shape=(131, 129), nshot=2, order=4, sponge=10, ckpt_format="bf16"),
    dict(shape=(60, 257), nshot=5, order=2, sponge=8, ckpt_format="i16"),
    dict(shape=(402, 513), nshot=2, order=8, sponge=((0, 12), (7, 0)), ckpt_format="bf16"),
], ids=lambda k: "x".join(map(str, k["shape"])))
@pytest.mark.parametrize("more", [dict(), dict(step_block=2, store_levels=40), dict(update="leapfrog", ckpt_every=1),
                                  dict(store_levels=80, ckpt_every=9), dict(group_shots=2, ckpt_every=61)],
                         ids=lambda m: "_".join(f"{k}{v}" for k, v in m.items()) or "default")
def test_resident_gradient_equals_streaming(cuda, kw, more):
    from neuralmech_gb300 import misfit_gradient
    grid, v, wav, src, rec = small_problem(seed=5, nt=61, nrec=40, nsrc=2, **kw)
    rng = np.random.default_rng(1)
    src = _distinct(rng, grid.order // 2, grid.shape, src.shape[0], 2)
    rec = _distinct(rng, grid.order // 2, grid.shape, src.shape[0], 40)
    grid = dataclasses.replace(grid, **more)
    obs = torch.from_numpy(rng.standard_normal((src.shape[0], grid.nt, 40)).astype(np.float32)).to(cuda)
    args = (torch.from_numpy(v).to(cuda), torch.from_numpy(wav).to(cuda), torch.from_numpy(src), torch.from_numpy(rec), obs)
    got = misfit_gradient(*args, grid, want_wavelet=True, want_traces=True)
    ref = misfit_gradient(*args, dataclasses.replace(grid, shots_per_cta=1), want_wavelet=True, want_traces=True)
    assert torch.equal(got[3], ref[3])
    assert abs(float(got[0]) / float(ref[0]) - 1) <= 1e-12
    assert rel_l2(got[1].cpu().numpy(), ref[1].cpu().numpy()) <= 1e-5
    assert rel_l2(got[2].cpu().numpy(), ref[2].cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("update", ["leapfrog", "auto"])
def test_resident_points_past_the_linked_ones(cuda, update):
    """600 sources and 700 receivers in one tile (256 are staged per tile)."""
    from neuralmech_gb300 import misfit_gradient
    grid, v, _, _, _ = small_problem(shape=(60, 120), nshot=2, nt=40, order=8, sponge=5, seed=9, ckpt_every=7)
    grid = dataclasses.replace(grid, update=update)
    rng = np.random.default_rng(2)
    src, rec = _distinct(rng, 4, grid.shape, 2, 600), _distinct(rng, 4, grid.shape, 2, 700)
    wav = torch.from_numpy(rng.standard_normal((2, 40, 600)).astype(np.float32)).to(cuda)
    obs = torch.zeros((2, 40, 700), device=cuda)
    args = (torch.from_numpy(v).to(cuda), wav, torch.from_numpy(src), torch.from_numpy(rec), obs)
    got = misfit_gradient(*args, grid, want_wavelet=True, want_traces=True)
    ref = misfit_gradient(*args, dataclasses.replace(grid, shots_per_cta=1), want_wavelet=True, want_traces=True)
    assert torch.equal(got[3], ref[3])
    assert rel_l2(got[1].cpu().numpy(), ref[1].cpu().numpy()) <= 1e-5
    assert rel_l2(got[2].cpu().numpy(), ref[2].cpu().numpy()) <= 1e-5


def test_a_workspace_without_mailboxes_streams(cuda):
    """A workspace of the streaming kernels' size (which the library reported before it
    had the resident one) is accepted, and gives the same traces."""
    from neuralmech_gb300 import _lib, wave_forward
    from neuralmech_gb300.wavefd import _prepare, _ptr, _stream, workspace_bytes
    grid, v, wav, src, rec = small_problem(shape=(90, 200), nshot=2, nt=50, seed=4)
    args = (torch.from_numpy(v).to(cuda), torch.from_numpy(wav).to(cuda), torch.from_numpy(src), torch.from_numpy(rec))
    ref = wave_forward(*args, grid)
    n = workspace_bytes(dataclasses.replace(grid, shots_per_cta=1), 2, 1, rec.shape[1], False)
    assert n < workspace_bytes(grid, 2, 1, rec.shape[1], False)
    c = _prepare(*args, grid)
    ws = torch.empty(n + 256, dtype=torch.uint8, device=cuda)
    ws = ws[(-ws.data_ptr()) % 256:][:n]
    t = torch.empty_like(ref)
    gz, gy, gx = c.sponges
    n0 = _launches()
    _lib.check(_lib.load().wfd_forward(ctypes.byref(c.problem), _ptr(c.vel), _ptr(gz), _ptr(gy), _ptr(gx), _ptr(c.wavelet),
                                       _ptr(c.src), _ptr(c.rec), _ptr(t), 0, _ptr(ws), n, _stream()), "wfd_forward")
    assert _launches() - n0 > grid.nt
    assert torch.equal(t, ref)
