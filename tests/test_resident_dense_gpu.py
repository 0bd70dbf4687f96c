"""Tiles of the resident kernel that hold as many points as it links (256), one more, and
one point in every cell. Values against the streaming kernels at distinct cells, as the
resident kernel's other tests: levels, traces and misfits equal, gradients 1e-5. A dense
cotangent must not cost many times what it costs the streaming kernels (the measured ratio
is 0.65; a walk of every thread through the list took 3.5)."""
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


def _block(R, shape, n):
    """n distinct cells, of the first tile as long as it has them."""
    z, x = np.mgrid[R:shape[0] - R, R:shape[1] - R]
    cells = np.stack([z.ravel(), x.ravel()], -1)
    first = (cells[:, 0] < 8) & (cells[:, 1] < 128)
    return np.concatenate([cells[first], cells[~first]])[:n].astype(np.int32)


@pytest.mark.parametrize("nsrc,nrec", [(1, 256), (1, 257), (256, 5), (257, 300), (1, 12500)])
@pytest.mark.parametrize("order,update", [(2, "auto"), (4, "leapfrog"), (8, "auto"), (8, "leapfrog")])
def test_points_at_the_linked_count(cuda, order, update, nsrc, nrec):
    from neuralmech_gb300 import misfit_gradient
    grid, v, _, _, _ = small_problem(shape=(70, 200), nshot=2, nt=37, order=order, sponge=5, seed=9, ckpt_every=9)
    grid = dataclasses.replace(grid, update=update)
    R, rng = order // 2, np.random.default_rng(nrec)
    src, rec = _block(R, grid.shape, nsrc), _block(R, grid.shape, nrec)
    wav = torch.from_numpy(rng.standard_normal((2, 37, len(src))).astype(np.float32)).to(cuda)
    obs = torch.zeros((2, 37, len(rec)), device=cuda)
    args = (torch.from_numpy(v).to(cuda), wav, torch.from_numpy(src), torch.from_numpy(rec), obs)
    n0 = _launches()
    got = misfit_gradient(*args, grid, want_wavelet=True, want_traces=True)
    assert _launches() - n0 < 37  # the resident kernel
    ref = misfit_gradient(*args, dataclasses.replace(grid, shots_per_cta=1), want_wavelet=True, want_traces=True)
    assert torch.equal(got[3], ref[3]) and float(got[3].abs().max()) > 0
    assert rel_l2(got[1].cpu().numpy(), ref[1].cpu().numpy()) <= 1e-5
    assert rel_l2(got[2].cpu().numpy(), ref[2].cpu().numpy()) <= 1e-5


def test_a_receiver_in_every_cell_is_not_slow(cuda):
    from neuralmech_gb300 import Grid, misfit_gradient
    grid = Grid((256, 256), (10.0, 10.0), 1e-3, 60, order=8, sponge=10)
    rec = torch.from_numpy(_block(4, grid.shape, 248 * 248)).to(cuda)
    src = torch.tensor([[128, 128]], device=cuda)
    wav = torch.ones(60, device=cuda)
    obs = torch.zeros((1, 60, rec.shape[0]), device=cuda)
    vel = torch.full((256, 256), 2500.0, device=cuda)

    def ms(g):
        best = float("inf")
        for _ in range(4):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            misfit_gradient(vel, wav, src, rec, obs, g, check=False)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    assert ms(grid) < 1.5 * ms(dataclasses.replace(grid, shots_per_cta=1))
