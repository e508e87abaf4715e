"""A device reset between two batches.

cudaDeviceReset ends the process's context on the device and everything in
it; the documented limit is that only the allocation-free entry point does not
survive one.  In a process of its own, through the driver's form of the call
(the library has its own copy of the runtime).
"""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes, sys
sys.path[:0] = [%r, %r]
from conftest import make_kw
from smili_b200 import _lib, synth
prob = _lib.Problem(make_kw(synth.small_crescent(seed=1, nx=32, niter=3)))

def solve():
    b = _lib.Batch([prob], niter=3, options=_lib.make_options(64, 1e-12))
    b.run()
    cost = b.fetch(0)[1]["cost"]
    b.close()
    return cost

driver, dev = ctypes.CDLL("libcuda.so.1"), ctypes.c_int()
want = [solve(), solve()][0]
assert driver.cuDeviceGet(ctypes.byref(dev), 0) == 0
for _ in range(2):
    assert driver.cuDevicePrimaryCtxReset_v2(dev) == 0
    for _ in range(3):
        assert abs(solve() - want) <= 1e-9 * abs(want)
print("survived")
"""


@pytest.mark.gpu
def test_batches_survive_a_device_reset():
    r = subprocess.run([sys.executable, "-c", PROGRAM % (ROOT, os.path.join(ROOT, "tests"))], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "survived" in r.stdout, r.stderr[-2000:]
