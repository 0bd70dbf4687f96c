"""The 3D kernel's two column shapes (64 x 16 and 32 x 32 cells): the shape follows
from the grid and the number of shots, the values do not. On these grids one shot
runs on the first shape and 60 equal ones on the second: levels and traces value
for value the same, and the gradient 60 times that of one shot (60 sums in FP32 of
values that agree to FP32 rounding: 2e-5)."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from helpers import small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,order", [((40, 64, 95), 8), ((24, 63, 157), 8), ((24, 64, 160), 4), ((40, 61, 93), 2)])
def test_column_shapes_agree(cuda, shape, order):
    from neuralmech_gb300.wavefd import misfit_gradient, wave_forward_final
    S = 60
    grid, v, wav, src, rec = small_problem(shape=shape, nshot=1, nt=24, nrec=23, order=order, sponge=4, seed=5, cfl=0.4)
    vel = torch.from_numpy(v).to(cuda)
    rng = np.random.default_rng(1)
    obs = (1e-3 * rng.standard_normal((1, grid.nt, rec.shape[1]))).astype(np.float32)
    one = [torch.from_numpy(a) for a in (wav, src, rec, obs)]
    many = [torch.from_numpy(np.repeat(a, S, axis=0)) for a in (wav, src, rec, obs)]
    t1, u1 = wave_forward_final(vel, one[0].to(cuda), one[1], one[2], grid)
    tS, uS = wave_forward_final(vel, many[0].to(cuda), many[1], many[2], grid)
    assert float(u1.abs().max()) > 0
    assert torch.equal(tS, t1.expand_as(tS)) and torch.equal(uS, u1.expand_as(uS))
    g1 = misfit_gradient(vel, one[0].to(cuda), one[1], one[2], one[3].to(cuda), grid)[1]
    gS = misfit_gradient(vel, many[0].to(cuda), many[1], many[2], many[3].to(cuda), grid)[1]
    assert rel_l2(gS.cpu().numpy(), S * g1.cpu().numpy()) <= 2e-5
