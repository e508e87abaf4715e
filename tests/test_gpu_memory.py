"""Batches on a device that is nearly full.

The kernel weights' tables are kept where there is room for them; without it
a batch is made and solved without them, with the same results.
"""
import numpy as np
import pytest

from conftest import make_kw

pytestmark = pytest.mark.gpu


def _many_points(nuv):
    """A small image under nuv visibilities (the crescent's, repeated and shifted)."""
    from smili_b200 import synth
    kw = dict(make_kw(synth.small_crescent(seed=2, nx=32, niter=1), l1_lambda=-1, tsv_lambda=-1))
    kw.update(dict.fromkeys(("isamp", "iscp", "isca"), False))
    n0, rng = np.size(kw["u"]), np.random.default_rng(0)
    pick = rng.integers(0, n0, nuv)
    kw.update(u=np.asarray(kw["u"])[pick] * rng.uniform(0.9, 1.1, nuv),
              v=np.asarray(kw["v"])[pick] * rng.uniform(0.9, 1.1, nuv), uvidxfcv=np.arange(1, nuv + 1),
              vfcvr=np.asarray(kw["vfcvr"])[pick], vfcvi=np.asarray(kw["vfcvi"])[pick],
              varfcv=np.asarray(kw["varfcv"])[pick])
    return kw


def test_batch_without_room_for_the_weight_tables():
    """1.5e6 points at eps 1e-12 (w = 13): 312 MB of tables and some 120 MB of
    everything else, with 200 MB free.  A second batch, with 40 MB free, has
    no room at all; its error is reported once and does not turn up in later calls."""
    import torch
    from smili_b200 import _lib
    from smili_b200.fortlib import fftlib
    prob = _lib.Problem(_many_points(1500000))

    def cost():
        b = _lib.Batch([prob], niter=1, options=_lib.make_options(64, 1e-12))
        b.run(fg_only=1)
        _, t, g, _ = b.fetch(0)
        return b, t["cost"], g

    b, want, grad = cost()
    b.close()
    img, u = np.ones((32, 32)), np.linspace(-1.0, 1.0, 100)
    vis = fftlib.nufft_fwd_real(u, u, img)
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (200 << 20), dtype=torch.uint8, device="cuda")
    more = None
    try:
        b, got, g = cost()
        rest = max(torch.cuda.mem_get_info()[0] - (40 << 20), 0)
        more = torch.empty(rest, dtype=torch.uint8, device="cuda")
        with pytest.raises(_lib.SmiliError) as e:
            cost()
        assert e.value.code == -3 and "allocation" in str(e.value)
        again = fftlib.nufft_fwd_real(u, u, img)
        b.close()
    finally:
        hold = more = None
        torch.cuda.empty_cache()
    assert abs(got - want) <= 1e-12 * abs(want)
    assert np.abs(g - grad).max() <= 1e-11 * np.abs(grad).max()
    assert np.array_equal(vis, again)


def test_small_call_where_the_pool_cannot_grow():
    """The library's memory pool grows by 32 MB.  With 12 to 24 MB left, a
    transform that needs a megabyte or two still goes through."""
    import torch
    from smili_b200.fortlib import fftlib
    img, u = np.ones((32, 32)), np.linspace(-1.0, 1.0, 100)
    vis = fftlib.nufft_fwd_real(u, u, img)
    hold = []
    try:
        for size in (4 << 30, 256 << 20, 12 << 20):
            while True:
                try:
                    hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                except torch.cuda.OutOfMemoryError:
                    break
        hold.pop()
        torch.cuda.empty_cache()
        again = fftlib.nufft_fwd_real(u, u, img)
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    assert np.array_equal(vis, again)
