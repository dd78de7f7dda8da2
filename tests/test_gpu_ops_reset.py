"""Per-slice operators across a reset of the process's own CUDA context: idle
device blocks of the old context are not used in the new one, where their
addresses are given out again (a child process, so that the reset ends no other
test's context)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, sys
sys.path[:0] = [sys.argv[1] + "/verb-4d_b200", sys.argv[1] + "/tests"]
import numpy as np
from verb4d_b200 import _lib
from test_gpu_ops_threads import convection_call, diffusion_call, tridag_call

_lib.load()
rt = ctypes.CDLL("libcudart.so.12")  # the one the library is linked with
calls = [convection_call(12, 13, 1), diffusion_call(9, 9, 2), tridag_call(500, 3),
         diffusion_call(31, 31, 4)]
ref = [f() for f in calls]
for turn in range(3):
    assert rt.cudaDeviceReset() == 0
    # memory of another owner, at the addresses that the idle blocks had
    p, size = ctypes.c_void_p(), 1 << 20
    mine = []
    for i in range(8):
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0
        assert rt.cudaMemset(p, i + 1, ctypes.c_size_t(size)) == 0
        mine.append(p.value)
    for f, x in zip(calls, ref):
        assert np.array_equal(f(), x)
    host = np.empty(size, np.uint8)
    for i, q in enumerate(mine):
        assert rt.cudaMemcpy(host.ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(q),
                             ctypes.c_size_t(size), 2) == 0
        assert (host == i + 1).all()
print("same")
"""


def test_after_a_reset(gpu):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["same"]
