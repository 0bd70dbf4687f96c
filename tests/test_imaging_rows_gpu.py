"""TFM over grids of pixels with rows of any length: values as the pixel-by-pixel call (the
same sums: equal), and narrow rows take no longer than the same number of pixels in long
ones by more than their own spread (measured 1.1 to 1.5; blocks of 16 columns on rows of
two took 5.3)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(cuda, E, nt, w, h):
    gen = torch.Generator(device=cuda).manual_seed(w)
    traces = torch.view_as_complex(torch.randn((E, E, nt, 2), generator=gen, device=cuda))
    el = torch.stack([torch.linspace(0, 1, E), torch.zeros(E)], 1)
    x, y = np.meshgrid(np.linspace(0.2, 0.8, w, dtype=np.float32), np.linspace(0.05, 0.9, h, dtype=np.float32))
    return traces, el, torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)


@pytest.mark.parametrize("w,h", [(2, 301), (15, 77), (16, 9), (17, 33), (32, 8), (33, 40), (127, 3), (512, 9), (513, 5)])
def test_rows_of_any_length(cuda, w, h):
    from neuralmech_gb300.imaging import tfm
    traces, el, x, y = _setup(cuda, 7, 200, w, h)
    img = tfm(traces, el, 0.0, 0.012, 1.0, x, y)
    order = torch.randperm(w * h, device=cuda)
    mixed = tfm(traces, el, 0.0, 0.012, 1.0, x.reshape(-1)[order], y.reshape(-1)[order])
    assert float(img.max()) > 0 and torch.equal(img.reshape(-1)[order], mixed)


@pytest.mark.parametrize("w", [2, 4, 17])
def test_narrow_rows_are_not_slow(cuda, w):
    from neuralmech_gb300.imaging import tfm

    def ms(w):
        args = _setup(cuda, 32, 1500, w, 262144 // w)
        best = float("inf")
        for _ in range(5):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            tfm(args[0], args[1], 0.0, 2.0 / 1500, 1.0, args[2], args[3])
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    assert ms(w) < 2.0 * ms(512)
