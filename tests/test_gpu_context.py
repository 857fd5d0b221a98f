"""A second CUDA context on a device the library has already served: kernels
that need more than 48 KB of shared memory must be allowed it there too."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

# One cell per call, in the primary context and then in a driver context of its own: the device memory comes
# from the driver, the LLRs of both are compared.
CHILD = r"""
import ctypes, importlib, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
aeq = importlib.import_module("aerial-mimo-tc-optimization_b200")
wl = importlib.import_module("aerial-mimo-tc-optimization_b200.workload")
cu = ctypes.CDLL("libcuda.so.1")
def ok(s): assert s == 0, s
ok(cu.cuInit(0))
dev = ctypes.c_int(); ok(cu.cuDeviceGet(ctypes.byref(dev), 0))
primary, second = ctypes.c_void_p(), ctypes.c_void_p()
ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(primary), dev))
ok(cu.cuCtxCreate_v2(ctypes.byref(second), 0, dev))
c = wl.make_cell(2, 128, 8, 11, 16, 20.0, seed=5)
H, Y = c.H.numpy(), c.Y.numpy()

def alloc(n, src=None):
    p = ctypes.c_uint64()
    ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(n)))
    if src is not None:
        ok(cu.cuMemcpyHtoD_v2(p, src.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(n)))
    return p.value

def run(ctx):
    ok(cu.cuCtxSetCurrent(ctx))
    out = np.zeros((2, c.llr_numel), np.float32)
    h, y = alloc(H.nbytes, H), alloc(Y.nbytes, Y)
    d = aeq.CellDesc()
    d.H, d.Y_rx, d.sigma2 = h, y, c.sigma2
    d.nPRB, d.nAnt, d.nLayers, d.nSym, d.nPamBits = c.nPRB, c.nAnt, c.nLayers, c.nSym, c.nPamBits
    arr = (aeq.CellDesc * 1)(d)
    for i, call in enumerate((lambda: aeq.lib().aerial_pusch_eq_plain_static(arr, 1, None),
                              lambda: aeq.lib().aerial_pusch_eq_fused(arr, 1, None, None))):
        arr[0].llr = alloc(out[i].nbytes)
        s = call()
        assert s == 0, (i, s, aeq.lib().aerial_error_string(s))
        ok(cu.cuCtxSynchronize())
        ok(cu.cuMemcpyDtoH_v2(out[i].ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(arr[0].llr),
                              ctypes.c_size_t(out[i].nbytes)))
    return out

a = run(primary)
b = run(second)
again = run(primary)
assert np.isfinite(a).all() and np.abs(a).max() > 0
assert (a == b).all() and (a == again).all()
print("same")
"""


def test_second_context_on_a_device():
    root = os.path.join(os.path.dirname(__file__), "..")
    r = subprocess.run([sys.executable, "-c", CHILD, root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
