"""The eight-step stream kernel (wfd_temporal_step_fast) where its strips and row
groups end: columns about multiples of the 112 stored ones, rows about the
groups' ends, padded and unpadded rows (16-byte and 4-byte copies), against eight
single steps in FP64 (1e-6 after one launch: 8 roundings of 6e-8 grow at most
linearly with the steps in both levels)."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _eight(u0, u1, cx, cy):
    a, b = u0.astype(np.float64), u1.astype(np.float64)
    for _ in range(8):
        n = a.copy()  # (fixed cells keep the value of two levels before)
        c = b[1:-1, 1:-1]
        n[1:-1, 1:-1] = 2 * c - a[1:-1, 1:-1] + cx * (b[:-2, 1:-1] - 2 * c + b[2:, 1:-1]) + cy * (b[1:-1, :-2] - 2 * c + b[1:-1, 2:])
        a, b = b, n
    return a, b


@pytest.mark.parametrize("N", [3, 17, 64, 401])
@pytest.mark.parametrize("M", [3, 9, 111, 112, 113, 119, 120, 121, 127, 128, 129, 225, 1000])
@pytest.mark.parametrize("pad", [0, 5])
def test_strips_and_row_groups(cuda, N, M, pad):
    from neuralmech_gb300.wavefd import temporal_step_fast
    Mp = M if pad == 0 else (M + pad + 3) // 4 * 4
    rng = np.random.default_rng(N * M)
    u0, u1 = (rng.standard_normal((N, Mp)).astype(np.float32) for _ in range(2))
    u0[:, M:] = u1[:, M:] = np.nan  # (never used)
    u1[:, :M] = u0[:, :M] + 0.01 * u1[:, :M]
    v0, v1 = torch.full((N, Mp), 3.0, device=cuda), torch.full((N, Mp), 4.0, device=cuda)
    dx, dy, dt = np.float32(0.01), np.float32(0.013), np.float32(0.005)
    temporal_step_fast(torch.from_numpy(u0).to(cuda), torch.from_numpy(u1).to(cuda), v0, v1, 1.0, float(dt), float(dx),
                       float(dy), N, M)
    k = float(dt * dt)
    a, b = _eight(u0[:, :M], u1[:, :M], k / float(dx * dx), k / float(dy * dy))
    assert rel_l2(v0[:, :M].cpu().numpy(), a) < 1e-6 and rel_l2(v1[:, :M].cpu().numpy(), b) < 1e-6
    assert bool((v0[:, M:] == 3.0).all()) and bool((v1[:, M:] == 4.0).all())
