"""The device sort of a bare transform's points.

Transforms against the oracle's exact sums at the tolerances of the other
transform tests (1e-10 at eps = 1e-12, 2e-5 in FP32 at 1e-6), for point
counts around the 128-point work items, points piled into one cell, points
in a narrow band away from zero, and points over the whole fine grid and
beyond it (periodic in 2 pi).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


def _points(kind, n, rng):
    if kind == "one cell":
        return np.full(n, 0.31), np.full(n, -1.2)
    if kind == "narrow":
        return rng.uniform(1.0, 1.2, n), rng.uniform(-2.9, -2.8, n)
    if kind == "line":
        return np.linspace(-3.1, 3.1, n), np.zeros(n)
    return rng.uniform(-7.0, 7.0, n), rng.uniform(-3.2, 3.2, n)


@pytest.mark.parametrize("kind", ["one cell", "narrow", "line", "everywhere"])
@pytest.mark.parametrize("nx,ny,nuv", [(32, 32, 1), (31, 45, 127), (45, 31, 129), (1, 7, 300), (64, 50, 5000)])
def test_bare_transforms(oracle, kind, nx, ny, nuv):
    from smili_b200.fortlib import fftlib
    rng = np.random.default_rng(nuv)
    u, v = _points(kind, nuv, rng)
    img = rng.standard_normal((ny, nx))
    c = rng.standard_normal(nuv) + 1j * rng.standard_normal(nuv)
    ex2 = oracle.nufft2d2(u, v, img, 0)
    ex1 = oracle.nufft2d1(u, v, c, nx, ny, 0).real.reshape(-1)
    # cancellation: errors scale with the sums of magnitudes
    s2, s1 = np.abs(img).sum(), np.abs(c).sum()
    for prec, eps, tol in ((64, 1e-12, 1e-10), (32, 1e-6, 2e-5)):
        vr, vi = fftlib.nufft_fwd_real(u, v, img.T, precision=prec, nufft_eps=eps)
        assert np.abs(vr + 1j * vi - ex2).max() <= tol * s2
        got = fftlib.nufft_adj_real1d(u, v, c.real, c.imag, nx, ny, precision=prec, nufft_eps=eps)
        assert np.abs(got - ex1).max() <= tol * s1


def test_bare_transforms_refuse_bad_points():
    from smili_b200.fortlib import fftlib
    img = np.ones((8, 8))
    for bad in (np.nan, np.inf, -np.inf):
        for k in (0, 7, 8, 19):
            u = np.zeros(20)
            u[k] = bad
            with pytest.raises(Exception):
                fftlib.nufft_fwd_real(u, np.zeros(20), img)
            with pytest.raises(Exception):
                fftlib.nufft_adj_real1d(np.zeros(20), u, np.ones(20), np.ones(20), 8, 8)
