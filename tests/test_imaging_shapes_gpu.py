"""The imaging kernels at the sizes where their splits end: traces of any length
modulo 8 (analytic signal, 1e-5 as its other test), and pixel lists that are
ragged grids, rows, columns or no grid at all, with early times (t0 < 0) and
times past the traces' end (TFM, 1e-4 as its other test)."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [2, 3, 7, 8, 9, 15, 16, 17, 63, 255, 256, 257, 1501, 2055])
def test_analytic_signal_lengths(cuda, nt):
    from scipy.signal import hilbert

    from neuralmech_gb300.imaging import analytic_signal
    x = np.random.default_rng(nt).standard_normal((5, nt)).astype(np.float32)
    h = analytic_signal(torch.from_numpy(x).to(cuda)).cpu().numpy()
    assert rel_l2(h, hilbert(x.astype(np.float64), axis=-1)) < 1e-5


@pytest.mark.parametrize("pixels", ["grid", "transposed", "row", "scattered", "one"])
@pytest.mark.parametrize("E,t0,reciprocity", [(9, 0.02, True), (6, -0.004, False), (4, 1.4, True)])
def test_tfm_pixel_lists(cuda, pixels, E, t0, reciprocity):
    from oracle.tfm_ref import tfm_kernel_semantics

    from neuralmech_gb300.imaging import tfm
    rng = np.random.default_rng(E)
    nt = 300
    a = (rng.standard_normal((E, E, nt)) + 1j * rng.standard_normal((E, E, nt))).astype(np.complex64)
    h = a + a.transpose(1, 0, 2)
    el = np.stack([np.linspace(0.1, 0.9, E), np.full(E, 1.0)], axis=1).astype(np.float32)
    gx, gy = np.meshgrid(np.linspace(0, 1, 37), np.linspace(0, 0.99, 21), indexing="ij" if pixels != "transposed" else "xy")
    x, y = {"row": (gx[:, 0], 0 * gx[:, 0]), "one": (gx[:1, 0], gy[:1, 0])}.get(pixels, (gx, gy))
    if pixels == "scattered":
        x, y = rng.random(203), 0.9 * rng.random(203)
    x, y = x.astype(np.float32), y.astype(np.float32)
    img = tfm(torch.from_numpy(h).to(cuda), el, t0, 0.005, 1.0, x, y, reciprocity=reciprocity)
    ref = tfm_kernel_semantics(h.astype(np.complex128), el[:, 0].astype(np.float64), el[:, 1].astype(np.float64), t0, 0.005,
                               1.0, x, y, reciprocity=reciprocity)
    assert rel_l2(img.cpu().numpy().ravel(), ref) < 1e-4
