"""The host-array entry points across cudaDeviceReset: what they keep between
calls belongs to a CUDA context that is gone then."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# A process of its own, without torch (whose state does not survive a reset).
PROGRAM = r"""
import ctypes, glob, os, site, sys
import numpy as np
lib = ctypes.CDLL(sys.argv[1])
P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
found = [f for d in sys.path for f in glob.glob(os.path.join(d, "nvidia", "cuda_runtime", "lib", "libcudart.so.*"))]
found += glob.glob("/usr/local/cuda/lib64/libcudart.so.1?")
rt = ctypes.CDLL(found[0])
rng = np.random.default_rng(0)
n, count = 20022, 120000
v = rng.normal(0, 1, (n, 9)).astype(np.float32)
rays = np.zeros((count, 8), np.float32)
rays[:, 3] = 10.0
rays[:, 4:7] = rng.normal(0, 1, (count, 3))


def calls():
    hits = np.zeros((count, 4), np.float32)
    assert lib.vlrbTraceRaysHost(P(v), ctypes.c_uint32(n), ctypes.c_uint32(3), P(rays), ctypes.c_uint32(count),
                                 ctypes.c_uint32(0), P(hits), None) == 0
    out = [np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(2 * n - 2, np.int32), np.zeros(6 * n - 6, np.float32)]
    assert lib.vlrbBvhBuildOptimizedHost(P(v), ctypes.c_uint32(n), ctypes.c_uint32(3), *(P(a) for a in out), None,
                                         None) == 0
    return [hits] + out


want = calls()
for _ in range(3):
    assert rt.cudaDeviceReset() == 0
    for _ in range(2):
        assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(calls(), want))
print("same")
"""


def test_host_calls_before_and_after_a_device_reset():
    lib = os.path.join(ROOT, "vlr_b200", "libvlr_b200.so")
    p = subprocess.run([sys.executable, "-c", PROGRAM, lib], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip() == "same", p.stdout + p.stderr
