"""How a problem is split over CTAs does not show in its results.

Group sizes from one CTA to all of the device, at sizes that leave some
CTAs without image rows, band columns, uv points or breakpoints.  One
evaluation in FP64 at the tight NUFFT tolerance (1e-12) agrees with the
oracle to 1e-9 (objective) and 1e-8 (gradient, max-norm), in FP32 (1e-6) to
1e-4 and 5e-3; the first ten iterations of a solve agree with the oracle's
to 1e-9, as those at the automatic group size do.  (Visibilities and closure phases of bright baselines: sums in
another order change them by rounding only.)
"""
import numpy as np
import pytest

from conftest import make_kw
from test_oracle3d import movie_kw

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from smili_b200 import _lib
    return _lib


def _rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


def _obs(nx, **over):
    from smili_b200 import synth
    return make_kw(synth.small_crescent(seed=nx, nx=nx, niter=10), **over)


@pytest.fixture(scope="module")
def odd(oracle):
    """33 x 33 pixels: a remainder in every split of rows and columns"""
    kw = _obs(33)
    x = np.asarray(kw["iin"]) * np.random.default_rng(1).uniform(0.5, 1.5, np.size(kw["iin"]))
    return kw, x, oracle.calc_cost(kw, x, eps=0.0)


@pytest.mark.parametrize("transform", [1, 2])
@pytest.mark.parametrize("ctas", [1, 2, 5, 32, 33, 148, 296])
def test_evaluation_over_group_sizes(odd, lib, ctas, transform):
    kw, x, (t, g) = odd
    for prec, eps, tol_t, tol_g in ((64, 1e-12, 1e-9, 1e-8), (32, 1e-6, 1e-4, 5e-3)):
        b = lib.Batch([lib.Problem(dict(kw, iin=x))], niter=1,
                      options=lib.make_options(prec, eps, ctas, transform=transform))
        b.run(fg_only=1)
        _, tb, gb, _ = b.fetch(0)
        b.close()
        assert abs(tb["cost"] - t["cost"]) <= tol_t * abs(t["cost"])
        assert _rel(gb, g) <= tol_g


@pytest.fixture(scope="module")
def short_trace(oracle, crescent32):
    kw = make_kw(crescent32, niter=10)
    return kw, oracle.imaging(kw, eps=1e-12)[2]["trace"]


@pytest.mark.parametrize("ctas", [0, 1, 3, 64, 296])
def test_solve_over_group_sizes(short_trace, lib, ctas):
    """1024 breakpoints: four rounds of the Cauchy search on one CTA, none
    left for most of 296"""
    kw, trace = short_trace
    b = lib.Batch([kw], niter=10, options=lib.make_options(64, 1e-12, ctas))
    b.run()
    tr = b.trace(0, 12)
    b.close()
    np.testing.assert_allclose(tr[:10], trace[:10], rtol=1e-9)


@pytest.mark.parametrize("ctas", [0, 1, 60, 200])
def test_mixed_sizes_share_a_launch(lib, ctas):
    """24^2 to 96^2 pixels, automatic groups (each problem its own size) and
    fixed ones (60: four groups and a queue of six; 200: one group)."""
    kws = [_obs(n, niter=5) for n in (24, 96, 33, 64, 25, 48)]
    b = lib.Batch(kws, niter=5, options=lib.make_options(64, 1e-12, ctas))
    for _ in range(2):
        b.run()
    for p, kw in enumerate(kws):
        s = lib.Batch([kw], niter=5, options=lib.make_options(64, 1e-12, 1))
        s.run()
        x1, t1, _, i1 = s.fetch(0)
        s.close()
        x, t, _, i = b.fetch(p)
        assert i["niter"] == i1["niter"]
        assert abs(t["cost"] - t1["cost"]) <= 1e-9 * abs(t1["cost"])
    b.close()


def test_more_problems_than_groups(lib):
    """300 problems on 296 CTAs: one CTA each and a queue; equal problems
    give equal results wherever they ran."""
    kw = _obs(24, niter=3)
    prob = lib.Problem(kw)
    b = lib.Batch([prob] * 300, niter=3, options=lib.make_options(64, 1e-12))
    b.run()
    cost = np.array([b.fetch(p)[1]["cost"] for p in range(300)])
    b.close()
    assert np.max(np.abs(cost - cost[0])) <= 1e-9 * abs(cost[0])


@pytest.mark.parametrize("ctas", [0, 1, 4, 5, 7, 17, 296])
def test_movie_over_group_sizes(oracle, ctas):
    """five frames on fewer CTAs than frames, one each, one and a remainder,
    several each; one frame has no data"""
    from smili_b200 import synth
    from smili_b200.fortlib import fftim3d
    from smili_b200.imaging.lbfgs3d import prepare_imaging3d
    m = synth.dynamic_problem(seed=4, nframes=5, nx=33, nst=6, vis_per_frame=90, niter=10)
    vt = m.vistable[m.vistable.frmidx != 3].reset_index(drop=True)
    bt = m.bstable[m.bstable.frmidx != 3].reset_index(drop=True)
    kw, _ = prepare_imaging3d(m.frames, vistable=vt, bstable=bt, niter=10, l1_lambda=1.0, tsv_lambda=1.0,
                              rt_lambda=1.0, ri_lambda=0.5, tfd_lambda=1.0)
    x = np.asarray(kw["iin"], dtype=np.float64) * np.random.default_rng(5).uniform(0.5, 1.5, np.size(kw["iin"]))
    t_o, g_o = oracle.calc_cost3d(kw, x, eps=0.0)
    t, g = fftim3d.calc_cost(x, nufft_eps=1e-12, ctas_per_problem=ctas, **kw)
    for k in t_o:
        if k in t:
            assert abs(t[k] - t_o[k]) <= 1e-9 * abs(t_o["cost"]), k
    assert _rel(g, g_o) <= 1e-8


def test_movie_solves_agree_over_group_sizes():
    from smili_b200.fortlib import fftim3d
    kw, _ = movie_kw(extra={"ri_lambda": 0.5})
    kw["niter"] = 5
    out = [fftim3d.imaging(nufft_eps=1e-12, ctas_per_problem=g, **kw)[20] for g in (1, 3, 50, 0)]
    assert np.max(np.abs(np.array(out) - out[0])) <= 1e-9 * abs(out[0])


def test_batches_from_threads(lib):
    """Batches made, run and freed by several threads at once, on the
    library's streams and on the caller's, share the pooled device memory."""
    import threading
    import torch
    kw = _obs(24, niter=3)
    prob = lib.Problem(kw)

    def solve(stream=None):
        b = lib.Batch([prob], niter=3, options=lib.make_options(64, 1e-12, 2, stream=stream))
        b.run()
        c = b.fetch(0)[1]["cost"]
        b.close()
        return c

    want, got = solve(), []

    def work(own):
        s = torch.cuda.Stream() if own else None
        for _ in range(10):
            got.append(solve(s.cuda_stream if own else None))

    ts = [threading.Thread(target=work, args=(k % 2 == 0,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(got) == 60 and np.max(np.abs(np.array(got) - want)) <= 1e-9 * abs(want)


def test_batch_refuses_a_capturing_stream(lib):
    import torch
    prob = lib.Problem(_obs(24, niter=3))
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    x = torch.zeros(1, device="cuda")
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        with pytest.raises(Exception):
            lib.Batch([prob], niter=3, options=lib.make_options(64, 1e-12, 1, stream=s.cuda_stream))
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert float(x) == 1.0


def test_movie_group_counts_its_points():
    """4 frames of 32^2 pixels with 2000 points each: 16 CTAs for the pixels
    and 10 for the points.  Sums depend on the group size in their last bits
    and on nothing else, so the automatic size shows in the cost terms."""
    from smili_b200 import synth
    from smili_b200.fortlib import fftim3d
    from smili_b200.imaging.lbfgs3d import prepare_imaging3d
    m = synth.dynamic_problem(seed=4, nframes=4, nx=32, nst=16, vis_per_frame=2000, niter=1)
    kw, _ = prepare_imaging3d(m.frames, vistable=m.vistable, bstable=m.bstable, niter=1, l1_lambda=1.0,
                              tsv_lambda=1.0, rt_lambda=1.0)
    x = np.asarray(kw["iin"], dtype=np.float64) * np.random.default_rng(5).uniform(0.5, 1.5, np.size(kw["iin"]))
    points = np.size(kw["u"])
    want = int(4096 / 256 + points / 800)
    assert want >= 20

    def terms(ctas):
        return fftim3d.calc_cost(x, nufft_eps=1e-6, ctas_per_problem=ctas, **kw)[0]

    auto = terms(0)
    assert auto == terms(0) == terms(want)
    assert auto != terms(16)  # four CTAs per frame instead of six


@pytest.mark.parametrize("ctas", [1, 3, 16, 148])
@pytest.mark.parametrize("eps", [1e-6, 1e-7, 1e-8])
def test_register_spreading_over_group_sizes(odd, oracle, lib, eps, ctas):
    """FP64 kernel widths 7, 8 and 9 spread with the subgrid in registers,
    the points cut into one range per warp: the objective and the gradient of
    the oracle at the same width (rounding only, at the bounds above)."""
    kw, x, _ = odd
    t, g = oracle.calc_cost(kw, x, eps=eps)
    b = lib.Batch([lib.Problem(dict(kw, iin=x))], niter=1, options=lib.make_options(64, eps, ctas))
    b.run(fg_only=1)
    _, tb, gb, _ = b.fetch(0)
    b.close()
    assert abs(tb["cost"] - t["cost"]) <= 1e-9 * abs(t["cost"])
    assert _rel(gb, g) <= 1e-8


@pytest.mark.parametrize("ctas", [1, 3, 148])
@pytest.mark.parametrize("eps", [0.5, 1e-2, 1e-6, 1e-8])
def test_register_spreading_equals_general_spreading(odd, lib, eps, ctas):
    """Widths 2, 3, 7 and 9 against the general spreading (16 x 16 tiles) at
    the same group size: the gradient differs by the order of at most 2016
    additions per cell and 64 per transform."""
    kw, x, _ = odd
    got = []
    for spread_bin in (8, 16):
        b = lib.Batch([lib.Problem(dict(kw, iin=x))], niter=1,
                      options=lib.make_options(64, eps, ctas, spread_bin=spread_bin))
        b.run(fg_only=1)
        got.append(b.fetch(0))
        b.close()
    assert abs(got[0][1]["cost"] - got[1][1]["cost"]) <= 1e-13 * abs(got[1][1]["cost"])
    assert _rel(got[0][2], got[1][2]) <= 1e-11
