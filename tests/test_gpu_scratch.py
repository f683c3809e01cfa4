"""The library's pool of call scratch: it follows its device's context, keeps a
bounded amount and gives it back."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

AFTER_RESET = """
import ctypes
import numpy as np
from salsaa_b200 import lib, params as P
L, rt = lib(), ctypes.CDLL("libcudart.so.12")

def run():
    n = 1 << 16
    w = np.arange(n, dtype=np.uint64) * np.uint64(123457) % np.uint64(P.Q0)
    outs = [np.zeros(1, np.uint64), np.zeros(2 * 16 * 3, np.uint64)]
    dev = []
    for a in (w, *outs):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)) == 0
        assert rt.cudaMemcpy(p, ctypes.c_void_p(a.ctypes.data), ctypes.c_size_t(a.nbytes), 1) == 0
        dev.append(p)
    assert L.salsaa_sumcheck(dev[0], 1, n, 128, P.Q0, 3, 1, dev[1], dev[2], None) == 0, L.salsaa_last_error()
    assert rt.cudaDeviceSynchronize() == 0
    for a, p in zip(outs, dev[1:]):
        assert rt.cudaMemcpy(ctypes.c_void_p(a.ctypes.data), p, ctypes.c_size_t(a.nbytes), 2) == 0
    return np.concatenate(outs)

first = run()
assert first.any() and np.array_equal(run(), first)
assert rt.cudaDeviceReset() == 0
assert np.array_equal(run(), first) and np.array_equal(run(), first)
"""


def test_scratch_after_device_reset(gpu_lib):
    """A pool ends with its context; calls after a reset get one of their own."""
    r = subprocess.run([sys.executable, "-c", AFTER_RESET], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_scratch_release(gpu_lib, cuda):
    """Without a context or dense key nothing else gives the memory back."""
    from salsaa_b200 import api, params as P
    w = cuda.ones((8, 1 << 15, 128), dtype=cuda.int64, device="cuda")
    c = cuda.ones((8, 128), dtype=cuda.int64, device="cuda")
    api.fold(w, P.Q0, c)
    cuda.cuda.synchronize()
    kept = cuda.cuda.mem_get_info()[0]
    api.scratch_release()
    free = cuda.cuda.mem_get_info()[0]
    assert free - kept >= w.numel() * 8  # the rows' slot form alone is that large
    cuda.cuda.synchronize()
    assert cuda.equal(api.fold(w, P.Q0, c), api.fold(w, P.Q0, c))
    api.scratch_release()
