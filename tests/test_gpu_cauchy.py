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


# (flux over the start's, variance over its square, l1, tsv): the search passes
# all of the crowded bucket in the first iteration, with no pairs stored; and
# in the fourth, with three
CROWDED = [(0.0, 1e-4, -1.0, 1e-3), (0.3, 1.0, 1e-2, 1e-3)]


@pytest.mark.parametrize("ctas", [1, 2, 16, 0])
@pytest.mark.parametrize("flux,var,l1,tsv", CROWDED)
def test_bucket_of_many_breakpoints(oracle, flux, var, l1, tsv, ctas):
    """Some 2450 of 4096 pixels have one value, the others values around it:
    their breakpoints fall into one bucket, taken 1024 at a time by radix
    selection.  Six iterations agree with the oracle's to 1e-9 (perturbing
    the start by 1e-13 moves the oracle by 6e-11 at most)."""
    from smili_b200 import _lib
    rng = np.random.default_rng(0)
    x0 = np.full(4096, 1.0)
    m = rng.random(4096) < 0.4
    x0[m] = rng.uniform(0.3, 3.0, m.sum())
    kw = _zero_baseline(x0, flux * x0.sum(), var * x0.sum() ** 2, 6)
    kw.update(l1_l=l1, tsv_l=tsv, l1_wgt=np.ones(4096), l1_nwgt=4096, tsv_wgt=np.ones(4096), tsv_nwgt=4096)
    want = oracle.imaging(kw, eps=1e-12)[2]["trace"][:6]
    b = _lib.Batch([kw], niter=6, options=_lib.make_options(64, 1e-12, ctas))
    b.run()
    got = b.trace(0, 6)
    b.close()
    np.testing.assert_allclose(got, want, rtol=1e-9)
