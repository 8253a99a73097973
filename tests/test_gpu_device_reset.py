"""The library's memory pool belongs to a CUDA context: after a device reset
(of this process's own context, in a process of its own) the next call makes
another and gives the same result."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r'''
import ctypes
import numpy as np
from stablebear_gb300 import _native as nat

cu = ctypes.CDLL("libcuda.so.1")


def ok(status):
    assert status == 0, status


def run():
    ctx = ctypes.c_void_p()
    ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(ctx), 0))
    ok(cu.cuCtxSetCurrent(ctx))
    rng = np.random.default_rng(1)
    n, k = 200, 30
    t = np.concatenate([np.r_[0.0, np.cumsum(rng.exponential(1, k - 1))] for _ in range(n)])
    v = rng.standard_normal(n * k)
    v[k - 1::k] = 0
    arrays = (np.ascontiguousarray(np.stack([t, v], 1)), np.arange(n + 1, dtype=np.uint64) * k,
              np.zeros(n * (n - 1) // 2))
    on = []
    for a in arrays:
        d = ctypes.c_uint64()
        ok(cu.cuMemAlloc_v2(ctypes.byref(d), ctypes.c_size_t(a.nbytes)))
        ok(cu.cuMemcpyHtoD_v2(d, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes)))
        on.append(ctypes.c_void_p(d.value))
    nat.check(nat.lib().sbg_pairwise_device(nat.F64, nat.OP_L1, 1.0, nat.SKIP_LOWER_NODIAG, on[0], on[1], n, None,
                                            None, 0, None, None, k, on[2], 0, 0, 0, None))
    ok(cu.cuCtxSynchronize())
    out = arrays[2]
    ok(cu.cuMemcpyDtoH_v2(out.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(on[2].value), ctypes.c_size_t(out.nbytes)))
    return out


ok(cu.cuInit(0))
first = run()
ok(cu.cuDevicePrimaryCtxReset_v2(0))
assert first.any() and np.array_equal(first, run())
print("the same")
'''


def test_a_call_after_a_device_reset():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "the same" in r.stdout, r.stderr
