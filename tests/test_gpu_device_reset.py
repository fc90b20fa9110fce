"""tgb_bin_transform keeps nothing across a cudaDeviceReset: its shared-memory opt-in (64 KB for
float64) is made on every call.  In a process of its own, which owns the context it resets."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from tidegbm_b200 import native
rt = C.CDLL(sys.argv[2])
n, nf = 1000, 5
rng = np.random.default_rng(0)
X = rng.standard_normal((n, nf))
E = np.full((nf, 256), np.inf)
E[:, :254] = np.sort(rng.standard_normal((nf, 254)), 1)
want = np.stack([np.searchsorted(E[f, :254], X[:, f], side="right") + 1 for f in range(nf)], 1)

def device(a):
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
    return p

for k in range(2):
    out = np.zeros((n, 16), np.uint8)
    c = device(out)
    native.check(native.lib().tgb_bin_transform(device(X), 1, n, nf, device(E), device(np.full(nf, 254, np.int32)), c, 16, None))
    assert rt.cudaMemcpy(out.ctypes.data_as(C.c_void_p), c, C.c_size_t(out.nbytes), 2) == 0
    assert np.array_equal(out[:, :nf], want)
    if k == 0:
        assert rt.cudaDeviceReset() == 0
print("ok")
"""


def test_transform_after_a_device_reset(native):
    import torch

    runtime = os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so.12")
    out = subprocess.run([sys.executable, "-c", PROGRAM, ROOT, runtime], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == "ok"
