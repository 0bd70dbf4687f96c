"""A backward on a thread that has made no CUDA call yet: autograd runs it on a
thread of its own, whose first use of CUDA is then the library's (a child
process, since the thread lives as long as its process)."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import dataclasses, torch
from helpers import small_problem
from neuralmech_gb300 import wave_forward
grid, v, wav, src, rec = small_problem(shape=(60, 150), nshot=2, nt=30, step_block=2)
vel = torch.from_numpy(v).cuda().requires_grad_(True)
t = wave_forward(vel, torch.from_numpy(wav).cuda(), torch.from_numpy(src), torch.from_numpy(rec),
                 dataclasses.replace(grid, shots_per_cta=1))
g, = torch.autograd.grad(t, vel, t.detach())  # (no kernel of torch's own on that thread first)
assert torch.isfinite(g).all() and float(g.abs().max()) > 0
print("gradient ok")
"""


def test_first_backward_of_a_process(cuda):
    import os
    tests = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", CODE.format(root=os.path.dirname(tests), tests=tests)], capture_output=True,
                       text=True, timeout=300)
    assert "gradient ok" in r.stdout, r.stderr[-2000:]
