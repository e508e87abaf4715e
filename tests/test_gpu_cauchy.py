"""The Cauchy search where more breakpoints share a bucket than one batch
holds (1024), against the oracle.

One visibility of a zero baseline pulls every pixel alike, so pixels of one
value have breakpoints that differ by rounding only.
"""
import numpy as np
import pytest

from conftest import make_kw

pytestmark = pytest.mark.gpu


def _zero_baseline(iin, flux, var, niter):
    """64 x 64 pixels under one visibility, flux, of variance var."""
    from smili_b200 import synth
    kw = dict(make_kw(synth.small_crescent(seed=3, nx=64, niter=niter)))
    kw.update(dict.fromkeys(("isamp", "iscp", "isca"), False))
    kw.update(dict.fromkeys([r + "_l" for r in ("l1", "tv", "tsv", "kl", "gs", "tfd", "cen", "sm")], -1.0))
    kw.update(iin=iin, u=np.zeros(1), v=np.zeros(1), isfcv=True, uvidxfcv=np.array([1]), wfcv=1.0,
              vfcvr=np.array([flux]), vfcvi=np.zeros(1), varfcv=np.array([var]), niter=niter)
    return kw


@pytest.mark.parametrize("ctas", [1, 3, 0])
def test_breakpoints_that_underflow_to_zero(ctas):
    """The least double everywhere and gradients of 1000: 4096 breakpoints at
    t = 0, index 0 among them, are taken in batches and the solve ends."""
    from smili_b200 import _lib
    kw = _zero_baseline(np.full(4096, 5e-324), -1.0, 1e-3, 5)
    b = _lib.Batch([kw], niter=5, options=_lib.make_options(64, 1e-12, ctas))
    b.run()
    x, terms, _, info = b.fetch(0)
    b.close()
    assert info["task"] != _lib.TASK_ERROR and info["niter"] <= 5
    assert not x.any() and abs(terms["cost"] - 500.0) <= 1e-9 * 500.0
