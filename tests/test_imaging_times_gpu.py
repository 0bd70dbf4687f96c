"""Delay and sum at times that the index from the bits of t + 2^23 does not hold: traces of
more than 2^23 samples, and times that are no numbers. One element at the origin, pixels
on it or at whole numbers of samples, so that every time is a sample's own and the image
is that sample's modulus (FP32 rounding of hypotf: 1e-6)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("late", [2.0 ** 23 - 8, 9000001.0 - 2, 2.0 ** 24 - 16])
def test_tfm_samples_past_2_to_23(cuda, late):
    from neuralmech_gb300.imaging import tfm
    nt = 2 ** 24 + 3
    gen = torch.Generator(device=cuda).manual_seed(1)
    h = torch.randn((1, 1, nt, 2), generator=gen, device=cuda)
    x = torch.arange(0, 8, device=cuda, dtype=torch.float32)  # sample late + 2 x
    img = tfm(torch.view_as_complex(h), [[0.0, 0.0]], late, 1.0, 1.0, x, torch.zeros_like(x))
    at = (late + 2 * x.double()).long()
    ref = h[0, 0, at].double().norm(dim=-1)
    assert float((img.double() / ref - 1).abs().max()) < 1e-6


@pytest.mark.parametrize("t0,dt", [(float("nan"), 1.0), (0.0, 1e-40)])
def test_tfm_times_that_are_no_numbers(cuda, t0, dt):
    """No image where a pair's time is not a number: t0 is none, or 0 / 0 samples
    (1 / dt is infinite, the pixel on the element)."""
    from neuralmech_gb300.imaging import tfm
    h = torch.ones((1, 1, 16), dtype=torch.complex64, device=cuda)
    img = tfm(h, [[0.0, 0.0]], t0, dt, 1.0, torch.zeros(1, device=cuda), torch.zeros(1, device=cuda))
    assert bool(img.isnan().all())
