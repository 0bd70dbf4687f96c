"""TFM at element counts around 96, whose times of flight fill the default limit of shared
memory, and at the most there may be (1e-4, the bound of the other TFM tests)."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 95, 96, 97, 256])
def test_tfm_element_counts(cuda, E):
    from oracle.tfm_ref import tfm_kernel_semantics

    from neuralmech_gb300.imaging import tfm
    rng = np.random.default_rng(E)
    h = (rng.standard_normal((E, E, 60)) + 1j * rng.standard_normal((E, E, 60))).astype(np.complex64)
    el = np.stack([np.linspace(0.1, 0.9, E), np.full(E, 1.0)], axis=1).astype(np.float32)
    x, y = np.meshgrid(np.linspace(0, 1, 20, dtype=np.float32), np.linspace(0, 0.9, 7, dtype=np.float32))
    img = tfm(torch.from_numpy(h).to(cuda), el, 0.01, 0.04, 1.0, x, y)
    ref = tfm_kernel_semantics(h.astype(np.complex128), el[:, 0].astype(np.float64), el[:, 1].astype(np.float64), 0.01, 0.04,
                               1.0, x, y)
    assert rel_l2(img.cpu().numpy().ravel(), ref) < 1e-4
