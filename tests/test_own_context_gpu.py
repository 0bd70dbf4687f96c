"""A caller with a driver context of its own (not the device's primary one, as PyCUDA
makes them): the library's calls run in that context and leave it current. In a process
of its own, which has no other context."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes, sys
cu = ctypes.CDLL("libcuda.so.1")
lib = ctypes.CDLL(sys.argv[1])
def ok(rc):
    assert rc == 0, rc
ok(cu.cuInit(0))
dev, ctx, now = ctypes.c_int(), ctypes.c_void_p(), ctypes.c_void_p()
ok(cu.cuDeviceGet(ctypes.byref(dev), 0))
ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev))
N, M = 40, 64
bufs = []
for k in range(4):
    p = ctypes.c_void_p()
    ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(4 * N * M)))
    ok(cu.cuMemsetD32_v2(p, ctypes.c_uint(0x3f800000), ctypes.c_size_t(N * M)))
    bufs.append(p)
f = ctypes.c_float
for rep in range(2):
    rc = lib.wfd_temporal_step(*bufs, f(1), f(0.1), f(1), f(1), N, M, M, None)
    ok(cu.cuCtxGetCurrent(ctypes.byref(now)))
    assert now.value == ctx.value, "another context is current"
    assert rc == 0
    ok(cu.cuCtxSynchronize())
out = (ctypes.c_float * (N * M))()
ok(cu.cuMemcpyDtoH_v2(out, bufs[3], ctypes.c_size_t(4 * N * M)))
assert all(v == 1.0 for v in out), "a constant field is a fixed point of the step"
print("fine")
"""


def test_the_callers_context_stays(cuda):
    from neuralmech_gb300.build import LIB
    r = subprocess.run([sys.executable, "-c", PROGRAM, LIB], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "fine", r.stdout + r.stderr
