"""wfd_backward after a forward of another layout (a different workspace_bytes, whose
kernels and point lists are others'), after one without checkpoints, and after none:
WFD_ERR_STATE and gradients of NaN; after its own forward, the gradient."""
import ctypes

import pytest
import torch

from helpers import small_problem

pytestmark = pytest.mark.gpu


class _Calls:
    """The C forward / backward pair of one problem on one buffer, each call given its own size."""

    def __init__(self, cuda, **kw):
        from neuralmech_gb300 import _lib
        from neuralmech_gb300.wavefd import _prepare, workspace_bytes
        self.lib, self.check = _lib.load(), _lib.check
        grid, v, wav, src, rec = small_problem(**kw)
        self.c = _prepare(torch.from_numpy(v).to(cuda), torch.from_numpy(wav).to(cuda), src, rec, grid)
        n = [c.shape[1] for c in (self.c.src, self.c.rec)]
        self.full = workspace_bytes(grid, src.shape[0], *n, True)
        self.ws = torch.zeros(self.full + 256, dtype=torch.uint8, device=cuda)
        self.ws = self.ws[(-self.ws.data_ptr()) % 256:][:self.full]
        self.traces = torch.empty((src.shape[0], grid.nt, rec.shape[1]), device=cuda)
        self.grad = torch.empty_like(self.c.vel)

    def _args(self):
        from neuralmech_gb300.wavefd import _ptr
        c = self.c
        return [ctypes.byref(c.problem), _ptr(c.vel), *map(_ptr, c.sponges), _ptr(c.wavelet), _ptr(c.src), _ptr(c.rec)]

    def forward(self, nbytes, save=1):
        from neuralmech_gb300.wavefd import _ptr, _stream
        self.check(self.lib.wfd_forward(*self._args(), _ptr(self.traces), save, _ptr(self.ws), nbytes, _stream()), "forward")

    def backward(self, nbytes):
        """Status after the call, and whether the gradient is NaN throughout its interior."""
        from neuralmech_gb300.wavefd import _ptr, _stream
        self.check(self.lib.wfd_backward(*self._args(), _ptr(self.traces), _ptr(self.grad), None, _ptr(self.ws), nbytes,
                                         _stream()), "backward")
        rc = self.lib.wfd_status(_ptr(self.ws), _stream())
        R = self.c.grid.order // 2
        inner = self.grad[tuple(slice(R, n - R) for n in self.grad.shape)]
        return rc, bool(inner.isnan().all()), bool(self.grad.isfinite().all() and self.grad.abs().max() > 0)


CASES = [dict(shape=(65, 128), nshot=3, nt=61, sponge=4, seed=2),
         dict(shape=(61, 133), nshot=2, nt=50, sponge=4, seed=3, step_block=2),
         dict(shape=(40, 140, 70), nshot=4, nt=20, sponge=4, seed=4)]


@pytest.mark.parametrize("kw", CASES, ids=lambda k: "x".join(map(str, k["shape"])))
def test_backward_wants_its_own_forward(cuda, kw):
    from neuralmech_gb300 import _lib
    p = _Calls(cuda, **kw)
    # the smallest size the library takes: the general kernels' layout
    lo, hi = 0, p.full
    while hi - lo > 256:
        mid = (lo + hi) // 512 * 256
        try:
            p.forward(mid)
            hi = mid
        except RuntimeError:
            lo = mid
    small = hi
    assert small < p.full
    torch.cuda.synchronize()
    p.ws.zero_()
    for n in (p.full, small):
        assert p.backward(n)[:2] == (_lib.WFD_ERR_STATE, True)  # no forward
        p.forward(n, save=0)
        assert p.backward(n)[:2] == (_lib.WFD_ERR_STATE, True)  # none with checkpoints
        p.forward(n)
        assert p.backward(n) == (0, False, True)
        p.forward(n)
        assert p.backward(p.full + small - n)[:2] == (_lib.WFD_ERR_STATE, True)  # another layout's
        p.ws.zero_()
