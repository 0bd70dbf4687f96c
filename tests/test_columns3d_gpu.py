"""The 3D kernel's z columns: how many planes a CTA marches depends on the grid
and on the number of shots, the levels do not. Each grid runs with one shot
(short columns) and with many equal ones (longer columns): every shot value for
value the same, and the first against the FP64 oracle (1e-5)."""
import dataclasses

import numpy as np
import pytest
import torch

from conftest import rel_l2
from helpers import oracle_geometry, small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,order", [((9, 12, 70), 8), ((65, 17, 33), 8), ((67, 33, 64), 4), ((130, 16, 40), 2)])
def test_columns_do_not_change_the_levels(cuda, orc, shape, order):
    from neuralmech_gb300.wavefd import wave_forward_final
    grid, v, wav, src, rec = small_problem(shape=shape, nshot=1, nt=40, nrec=19, order=order, sponge=3, seed=2, cfl=0.4)
    vel = torch.from_numpy(v).to(cuda)
    t1, u1 = wave_forward_final(vel, torch.from_numpy(wav).to(cuda), torch.from_numpy(src), torch.from_numpy(rec), grid)
    S = 60
    many = [np.repeat(a, S, axis=0) for a in (wav, src, rec)]
    tS, uS = wave_forward_final(vel, torch.from_numpy(many[0]).to(cuda), torch.from_numpy(many[1]),
                                torch.from_numpy(many[2]), grid)
    assert float(u1.abs().max()) > 0
    assert torch.equal(tS, t1.expand_as(tS)) and torch.equal(uS, u1.expand_as(uS))
    ref = orc.forward(oracle_geometry(orc, grid, v, wav, src, rec))
    assert rel_l2(t1.cpu().numpy(), ref) <= 1e-5
