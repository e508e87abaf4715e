"""uv coordinates far beyond the transform's fine grid.

The kernels place a point in the band of touched cells by differences of
32-bit cell numbers.  Coordinates that those cannot hold are refused by every
entry point before a device is touched (so this runs without one); the
transforms are periodic and take everything below.
"""
import numpy as np
import pytest

from conftest import make_kw
from test_oracle3d import movie_kw

ERR_DATA, ERR_NODEV = -2, -4
CELLS = 64 / (2 * np.pi)  # fine-grid cells per radian of a 32-pixel axis (eps 1e-6)


def _code(call):
    from smili_b200 import _lib
    try:
        call()
    except _lib.SmiliError as e:
        return e.code
    return 0


def _bare(u, v, precision):
    from smili_b200.fortlib import fftlib
    n = u.size
    return [lambda: fftlib.nufft_fwd_real(u, v, np.ones((32, 32)), precision=precision),
            lambda: fftlib.nufft_adj_real1d(u, v, np.ones(n), np.zeros(n), 32, 32, precision=precision)]


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("u", [1.01 * 2 ** 30 / CELLS, -1.01 * 2 ** 30 / CELLS, 1e12, -1e300])
def test_bare_transforms_refuse_what_cells_cannot_hold(u, precision):
    few = u * (1 + 1e-16 * np.arange(5))  # a narrow band
    for a, b in ((few, np.zeros(5)), (np.zeros(5), few), (np.append(few, 0.0), np.zeros(6))):
        for call in _bare(a, b, precision):
            assert _code(call) == ERR_DATA


@pytest.mark.parametrize("precision", [64, 32])
def test_bare_transforms_take_what_cells_can_hold(precision):
    u = np.full(5, 0.99 * 2 ** 30 / CELLS)
    for call in _bare(u, -u, precision):
        assert _code(call) in (0, ERR_NODEV)


def test_solves_and_movies_refuse_what_cells_cannot_hold(crescent32):
    from smili_b200 import _lib
    from smili_b200.fortlib import fftim2d, fftim3d
    kw = make_kw(crescent32, niter=2)
    bad = dict(kw, u=np.asarray(kw["u"]) + 1e12)
    assert _code(lambda: fftim2d.imaging(**bad)) == ERR_DATA
    assert _code(lambda: fftim2d.calc_cost(kw["iin"], **bad)) == ERR_DATA
    assert _code(lambda: fftim2d.calc_cost_noalloc(kw["iin"], **bad)) == ERR_DATA
    assert _code(lambda: _lib.Batch([kw, bad], niter=2)) == ERR_DATA
    m, _ = movie_kw(nframes=2)
    bad = dict(m, v=np.asarray(m["v"]) - 1e12)
    assert _code(lambda: fftim3d.calc_cost(m["iin"], **bad)) == ERR_DATA
