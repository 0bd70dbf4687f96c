"""Checkpoints of the resident kernel: FP32 ones are its launches' own state, BF16
ones are written beside it and read by the recompute, int16 ones go through the
packing kernels. In each format the gradient of a small problem with several
recomputed segments against the streaming kernels' (the same steps from the same
checkpoints; sums in another order: 2e-5), the misfit to FP64 rounding of its sum."""
import dataclasses

import numpy as np
import pytest
import torch

from conftest import rel_l2
from helpers import small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["fp32", "bf16", "i16"])
@pytest.mark.parametrize("order,update,every,nt", [(8, "auto", 7, 50), (8, "leapfrog", 1, 20), (4, "auto", 16, 33),
                                                   (2, "leapfrog", 9, 28)])
def test_checkpoint_formats(cuda, fmt, order, update, every, nt):
    from neuralmech_gb300.wavefd import misfit_gradient
    grid, v, wav, src, rec = small_problem(shape=(61, 133), nshot=3, nt=nt, nrec=17, order=order, sponge=9, seed=8)
    grid = dataclasses.replace(grid, ckpt_format=fmt, ckpt_every=every, update=update)
    vel = torch.from_numpy(v).to(cuda)
    obs = (1e-3 * np.random.default_rng(3).standard_normal((3, nt, rec.shape[1]))).astype(np.float32)
    args = (vel, torch.from_numpy(wav).to(cuda), torch.from_numpy(src), torch.from_numpy(rec), torch.from_numpy(obs).to(cuda))
    m, g = misfit_gradient(*args, grid)[:2]
    ms, gs = misfit_gradient(*args, dataclasses.replace(grid, shots_per_cta=1))[:2]
    assert float(gs.abs().max()) > 0
    assert abs(float(m) - float(ms)) <= 1e-12 * abs(float(ms))
    assert rel_l2(g.cpu().numpy(), gs.cpu().numpy()) <= 2e-5
