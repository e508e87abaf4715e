"""Host packing where no further threads can be made: the calling thread packs
everything itself, and no exception leaves the C entry points.

A child process whose threads would get stacks larger than the address space
(the default stack size is the stack limit).
"""
import os
import resource
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys, threading
sys.path[:0] = [%r, %r]
from conftest import make_kw
from test_oracle3d import movie_kw
from smili_b200 import _lib, synth
from smili_b200.fortlib import fftim3d
m, _ = movie_kw(nframes=4)
prob = _lib.Problem(make_kw(synth.small_crescent(seed=1, nx=32, niter=2)))
t = threading.Thread(target=print)
try:
    t.start()
    raise SystemExit("threads can be made here")
except RuntimeError:
    pass
for call in (lambda: fftim3d.calc_cost(m["iin"], **m), lambda: _lib.Batch([prob] * 4, niter=2).close()):
    try:
        call()
    except _lib.SmiliError as e:
        assert e.code == -4, e  # no CUDA device
print("no abort")
"""


def test_packing_without_threads():
    _, hard = resource.getrlimit(resource.RLIMIT_STACK)
    want = 1 << 47
    if hard != resource.RLIM_INFINITY and hard < want:
        import pytest
        pytest.skip("the stack limit cannot be raised")
    env = dict(os.environ, OMP_NUM_THREADS="1", OPENBLAS_NUM_THREADS="1", MKL_NUM_THREADS="1", CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, "-c", PROGRAM % (ROOT, os.path.join(ROOT, "tests"))], env=env,
                       preexec_fn=lambda: resource.setrlimit(resource.RLIMIT_STACK, (want, hard)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "no abort" in r.stdout, (r.returncode, r.stderr[-1500:])
