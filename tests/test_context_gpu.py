"""Calls after a context reset: kernel attributes are set again in the new context.

A child process calls the C entry points with buffers of its own, ends its context
with cudaDeviceReset (which touches no other process) and calls them again.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, sys
import numpy as np
rt = ctypes.CDLL("libcudart.so.12")
L = ctypes.CDLL(sys.argv[1])
vp, u = ctypes.c_void_p, ctypes.c_uint
rt.cudaMalloc.argtypes = [ctypes.POINTER(vp), ctypes.c_size_t]
rt.cudaMemcpy.argtypes = [vp, vp, ctypes.c_size_t, ctypes.c_int]
L.wino_dropin_conv2d.argtypes = [vp] * 6 + [u] * 9 + [vp]


def conv(n, c, h, w, k):
    rng = np.random.default_rng(n + c)
    x = rng.standard_normal((n, c, h, w)).astype(np.float16)
    wt = (rng.standard_normal((k, c, 3, 3)) / (9 * c) ** 0.5).astype(np.float16)
    y = np.zeros((n, k, h, w), np.float16)
    ptr = []
    for nbytes in (x.nbytes, wt.nbytes, y.nbytes, 8 * h * h * n * c, 32 * k * c, 8 * k * h * w * n):
        p = vp()
        assert rt.cudaMalloc(ctypes.byref(p), nbytes) == 0
        ptr.append(p)
    assert rt.cudaMemcpy(ptr[0], x.ctypes.data, x.nbytes, 1) == 0 and rt.cudaMemcpy(ptr[1], wt.ctypes.data, wt.nbytes, 1) == 0
    rc = L.wino_dropin_conv2d(*ptr, n, c, h, w, k, 3, 3, 1, 1, None)
    assert rc == 0, rc
    assert rt.cudaMemcpy(y.ctypes.data, ptr[2], y.nbytes, 2) == 0
    return y


# shift kernel, two-stage, fused
shapes = [(8, 64, 32, 32, 64), (2, 64, 16, 16, 32), (2, 32, 9, 7, 32)]
first = [conv(*s) for s in shapes]
assert all(np.isfinite(y).all() and y.any() for y in first)
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    for s, y in zip(shapes, first):
        assert np.array_equal(conv(*s).view(np.uint16), y.view(np.uint16)), s
print("ok")
"""


def test_calls_after_a_context_reset(wino, cuda):
    import torch
    env = dict(os.environ)
    lib = os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib")
    env["LD_LIBRARY_PATH"] = lib + os.pathsep + env.get("LD_LIBRARY_PATH", "")
    out = subprocess.run([sys.executable, "-c", CHILD, wino.LIB_PATH], env=env, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stderr[-2000:]
