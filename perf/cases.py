"""The performance cases of this framework: what its users have it do, over
the range of sizes they do it at.

``listed()`` names the cases that are always measured and ``draw(rng)`` makes
one more of the same ranges.  A case's ``kind`` says which public entry point
it goes through:

- ``solve``: one imaging problem kept on the device (``_lib.Batch`` of one
  problem) and solved again, FP64;
- ``evaluate``: one objective and gradient evaluation of a resident problem
  for an outer optimiser (``set_start``, ``run(fg_only=True)``, ``fetch``);
- ``batch``: many 256 x 256 problems in one FP32 launch, the image hand-over
  to the warm-start network included (``Batch.run``, ``Batch.images``);
- ``survey``: many problems of different sizes in one FP64 launch;
- ``imaging``: the drop-in call ``fortlib.fftim2d.imaging`` on host arrays;
- ``movie``: the dynamic-imaging call ``fortlib.fftim3d.imaging`` on host
  arrays;
- ``nufft``: ``fortlib.fftlib`` forward and adjoint transforms of host arrays;
- ``network``: the warm-start U-Net's forward pass;
- ``train``: one U-Net training step (forward, loss, backward, Adam);
- ``layer``: one 3x3 convolution layer, forward and backward from stored
  activations, through ``warmstart.kernels``.

Solves run a few iterations only: L-BFGS-B on closure data is chaotic, and
after some tens of iterations (in FP32 some five) two runs of the same code
differ visibly.
"""
import math
import os

import numpy as np
import torch

from smili_b200 import _lib, synth
from smili_b200.fortlib import fftim2d, fftim3d, fftlib
from smili_b200.imaging.lbfgs import prepare_imaging
from smili_b200.imaging.lbfgs3d import prepare_imaging3d
from smili_b200.warmstart import closure, kernels
from smili_b200.warmstart.unet import CHANNELS, UNet, layer_specs

DEV = "cuda"
WEIGHTS = os.path.join(os.path.dirname(closure.__file__), "unet_closure256.npz")  # the trained network


def listed():
    return [
        # the smallest imaging run: 64 x 64, 2 uas, a crescent seen by 8 stations in 10 min scans
        {"name": "solve-64", "kind": "solve", "nx": 64, "ny": 64, "pix": 2.0, "data": "vis", "nst": 8,
         "nscan": 72, "window": False, "niter": 10},
        # the headline problem: 256 x 256, 1 uas, 10 stations, ~97 000 amplitudes, closure phases and
        # log closure amplitudes, l1 + TV + MEM
        {"name": "solve-256", "kind": "solve", "nx": 256, "ny": 256, "pix": 1.0, "data": "closure", "nst": 10,
         "nscan": 2160, "window": False, "niter": 10},
        # a wide field: 1024 x 1024, 16 stations, 240 000 complex visibilities + closure phases
        {"name": "solve-1024", "kind": "solve", "nx": 1024, "ny": 1024, "pix": 1.0, "data": "vis", "nst": 16,
         "nscan": 2000, "window": False, "niter": 5},
        # an outer optimiser's call on the headline problem: start image in, cost terms and gradient out
        {"name": "evaluate-256", "kind": "evaluate", "nx": 256, "ny": 256, "pix": 1.0, "data": "closure",
         "nst": 10, "nscan": 2160, "window": False},
        # the benchmark's step at a third of its size: 148 headline problems in one FP32 launch
        {"name": "batch-256", "kind": "batch", "nx": 256, "nprob": 148, "nst": 10, "nscan": 2160, "niter": 3},
        # a hyper-parameter survey: 48 problems of 64^2 to 256^2 pixels and 2e3 to 5e4 visibilities
        {"name": "survey-48", "kind": "survey", "nprob": 48, "first": 0, "niter": 10},
        # the drop-in call with an image window and an odd field of view, every regularizer on
        {"name": "imaging-150x90", "kind": "imaging", "nx": 150, "ny": 90, "pix": 1.3, "data": "all", "nst": 8,
         "nscan": 150, "window": True, "niter": 20},
        # dynamic imaging of a rotating crescent: 16 frames of 64 x 64
        {"name": "movie-16x64", "kind": "movie", "nz": 16, "nx": 64, "nst": 10, "vis": 900, "niter": 10},
        # simulated visibilities and their dirty map, 200 000 uv points on an odd grid
        {"name": "nufft-200k", "kind": "nufft", "nx": 200, "ny": 162, "nuv": 200000, "band": 0.35, "eps": 1e-6},
        # the network's part of a warm-started step
        {"name": "network-64x128", "kind": "network", "n": 64, "side": 128},
        # one training step of the warm-start network, the batch and image size of its training script
        {"name": "train-32x128", "kind": "train", "n": 32, "side": 128},
        # the widest layer of the network's decoder on a full batch
        {"name": "layer-192", "kind": "layer", "n": 32, "h": 64, "w": 64, "cin": 192, "cout": 192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "evaluate", "batch", "survey", "imaging", "movie", "nufft", "network",
                       "train", "layer"])
    if kind in ("solve", "evaluate"):
        nx = _log(rng, 48, 512)
        c = {"kind": kind, "nx": nx, "ny": max(32, int(nx * rng.uniform(0.7, 1.3))),
             "pix": round(rng.uniform(0.8, 2.0), 3), "data": rng.choice(["vis", "closure", "all"]),
             "nst": rng.randint(6, 12), "nscan": _log(rng, 40, 1500), "window": rng.random() < 0.3}
        return c if kind == "evaluate" else dict(c, niter=rng.randint(4, 10))
    if kind == "batch":
        return {"kind": kind, "nx": 256, "nprob": rng.randint(20, 148), "nst": rng.randint(8, 10),
                "nscan": _log(rng, 500, 2160), "niter": rng.randint(2, 3)}
    if kind == "survey":
        return {"kind": kind, "nprob": rng.randint(6, 48), "first": rng.randint(0, 400), "niter": rng.randint(5, 10)}
    if kind == "imaging":
        return {"kind": kind, "nx": _log(rng, 40, 256), "ny": _log(rng, 40, 256), "pix": round(rng.uniform(0.8, 2.0), 3),
                "data": rng.choice(["vis", "closure", "all"]), "nst": rng.randint(6, 10), "nscan": _log(rng, 20, 400),
                "window": rng.random() < 0.5, "niter": rng.randint(5, 20)}
    if kind == "movie":
        return {"kind": kind, "nz": rng.randint(4, 24), "nx": _log(rng, 32, 96), "nst": rng.randint(6, 12),
                "vis": _log(rng, 200, 2000), "niter": rng.randint(5, 10)}
    if kind == "nufft":
        return {"kind": kind, "nx": _log(rng, 48, 512), "ny": _log(rng, 48, 512), "nuv": _log(rng, 1000, 400000),
                "band": round(rng.uniform(0.1, 0.8), 3), "eps": rng.choice([1e-6, 1e-6, 1e-9, 1e-12])}
    if kind in ("network", "train"):
        side = 8 * rng.randint(6, 20)  # as many pixels as the listed case at most
        return {"kind": kind, "n": _log(rng, 2, (64 if kind == "network" else 32) * min(1.0, (128 / side) ** 2)),
                "side": side}
    cin, cout = (8 * rng.randint(2, 24) for _ in range(2))
    return {"kind": "layer", "n": rng.randint(2, 32), "h": 8 * rng.randint(2, 8), "w": 8 * rng.randint(2, 8),
            "cin": cin, "cout": cout}


# ---------------------------------------------------------------------------
# observations
# ---------------------------------------------------------------------------
def _dft(truth, img, u, v, chunk=1 << 15):
    """Exact model visibilities (synth.exact_dft on the GPU)."""
    x, y = (torch.as_tensor(a.copy(), device=DEV) for a in img.get_xygrid(twodim=False, angunit="rad"))
    im = torch.as_tensor(np.array(truth, dtype=np.float64), device=DEV)
    ud, vd = (torch.as_tensor(np.array(a, dtype=np.float64), device=DEV) for a in (u, v))
    out = []
    for s in range(0, ud.numel(), chunk):
        a = 2 * math.pi * ud[s:s + chunk, None] * x
        b = 2 * math.pi * vd[s:s + chunk, None] * y
        ar, ai = torch.cos(a) @ im.T, torch.sin(a) @ im.T
        c, d = torch.cos(b), torch.sin(b)
        out.append(torch.complex((ar * c - ai * d).sum(1), (ai * c + ar * d).sum(1)))
    return torch.cat(out).cpu().numpy()


def _kwargs(nx, ny, pix, data, nst, nscan, niter, rng, window=False):
    """fftim2d.imaging keywords of one observation, started from a blurred
    earlier image as a pipeline restarts it."""
    img = synth.Image(nx, ny, pix)
    ext = 0.25 * pix * min(nx, ny)
    truth = synth.multigauss_gp_image(img, rng, ngauss=8, flux=1.0, extent_uas=ext, gp_corr_uas=6 * pix)
    vis = data in ("vis", "all")
    t = synth.observe(truth, img, rng, nst=nst, dec_deg=float(rng.uniform(-30, 60)), freq_hz=230e9, hours=12.0,
                      scan_min=720.0 / nscan, gain_amp=0.0 if vis else 0.1, gain_phase=not vis, fcv=vis,
                      amp=not vis or data == "all", cp=True, ca=not vis or data == "all",
                      amp_frac_err=0.0 if vis else 0.05, model=_dft)
    start = img.copy()
    start.data[0, 0] = synth._gauss_blur(truth, 4.0).clip(0) * (1 + 0.1 * rng.uniform(-1, 1, truth.shape)) + 1e-6
    reg = {"vis": {"l1_lambda": 1.0, "tsv_lambda": 1.0},
           "closure": {"l1_lambda": 1.0, "tv_lambda": 1.0, "kl_lambda": 0.1},
           "all": {"l1_lambda": 1.0, "tv_lambda": 0.5, "tsv_lambda": 0.5, "gs_lambda": 0.1, "tfd_lambda": 1.0,
                   "cen_lambda": 0.1, "cen_alpha": 3}}[data]
    if window:
        yy, xx = np.mgrid[0:ny, 0:nx]
        reg["imregion"] = ((xx - nx / 2) / (0.45 * nx)) ** 2 + ((yy - ny / 2) / (0.4 * ny)) ** 2 < 1
    kw, _ = prepare_imaging(start, vistable=t["vistable"], amptable=t["amptable"], bstable=t["bstable"],
                            catable=t["catable"], niter=niter, **reg)
    return kw


def _rng(*seed):
    return np.random.default_rng([int(s) & 0x7fffffff for s in seed])


def _survey_size(i):
    """Grid side, stations and scans of survey problem i (2e3 to 5e4 visibilities)."""
    r = np.random.default_rng([3, i])
    nst = int(r.integers(6, 13))
    return int(r.choice([64, 96, 128, 192, 256])), nst, int(10 ** r.uniform(3.3, 4.7) / (nst * (nst - 1) / 2)) + 1


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    k = case["kind"]
    rng = _rng(seed)
    if k in ("solve", "evaluate", "imaging"):
        kw = _kwargs(case["nx"], case["ny"], case["pix"], case["data"], case["nst"], case["nscan"],
                     case.get("niter", 1), rng, case["window"])
        if k == "imaging":
            return {"case": case, "kw": kw}
        s = {"case": case, "batch": _lib.Batch([kw], niter=case.get("niter", 1), options=_lib.make_options(64)),
             "kw": kw, "x": np.array(kw["iin"])}
        return s
    if k == "batch":  # four observations, each from many starts
        kws = [_kwargs(case["nx"], case["nx"], 1.0, "closure", case["nst"], case["nscan"], case["niter"], _rng(seed, i))
               for i in range(4)]
        probs = [_lib.Problem(dict(kws[i % 4], iin=kws[i % 4]["iin"] * rng.uniform(0.9, 1.1, kws[i % 4]["npix"])))
                 for i in range(case["nprob"])]
        b = _lib.Batch(probs, niter=case["niter"], options=_lib.make_options(32, 1e-6, 4))
        return {"case": case, "batch": b,
                "images": torch.empty(case["nprob"], case["nx"], case["nx"], dtype=torch.float32, device=DEV)}
    if k == "survey":
        kws = []
        for i in range(case["nprob"]):
            nx, nst, nscan = _survey_size(case["first"] + i)
            kws.append(_kwargs(nx, nx, 160.0 / nx, "vis", nst, nscan, case["niter"], _rng(seed, i)))
        return {"case": case, "batch": _lib.Batch(kws, niter=case["niter"], options=_lib.make_options(64))}
    if k == "movie":
        m = synth.dynamic_problem(seed=int(seed) & 0x7fffffff, nframes=case["nz"], nx=case["nx"], nst=case["nst"],
                                  vis_per_frame=case["vis"], niter=case["niter"], model=_dft)
        kw, _ = prepare_imaging3d(m.frames, vistable=m.vistable, bstable=m.bstable, niter=case["niter"], **m.reg)
        return {"case": case, "kw": kw}
    if k == "nufft":
        r, a = case["band"] * np.sqrt(rng.random(case["nuv"])), rng.uniform(0, 2 * np.pi, case["nuv"])
        c = rng.standard_normal((2, case["nuv"]))
        return {"case": case, "u": r * np.cos(a), "v": r * np.sin(a), "img": rng.random((case["nx"], case["ny"])),
                "cr": c[0], "ci": c[1]}
    g = torch.Generator(device=DEV).manual_seed(int(seed) & 0x7fffffff)
    if k == "network":
        return {"case": case, "net": UNet.load(WEIGHTS),
                "x": _blobs(case["n"], case["side"], g)}
    if k == "train":
        x = _blobs(case["n"], case["side"], g)
        return {"case": case, "net": UNet(seed=int(seed) & 0x7fffffff), "x": x, "t": _blobs(case["n"], case["side"], g)}
    n, h, w, ci, co = (case[q] for q in ("n", "h", "w", "cin", "cout"))

    def rand(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    bf = torch.bfloat16
    s = {"case": case, "x": rand(n, h, w, ci).relu().to(bf), "w": (rand(co, 3, 3, ci) / math.sqrt(4.5 * ci)).to(bf),
         "b": 0.1 * rand(co), "act": rand(n, h, w, co).relu().to(bf), "dy": rand(n, h, w, co).to(bf),
         "y": torch.empty(n, h, w, co, dtype=bf, device=DEV), "dx": torch.empty(n, h, w, ci, dtype=bf, device=DEV),
         "wt": torch.empty(ci, 3, 3, co, dtype=bf, device=DEV), "dw": torch.empty(co, 3, 3, ci, device=DEV),
         "db": torch.empty(co, device=DEV)}
    kernels.flip_weights(s["w"], s["wt"], co, ci)
    tiles = n * -(-h // 8) * -(-w // 16)
    s["nsplit"] = max(1, min(tiles, 296 // (-(-co // 64) * -(-ci // 16))))
    s["partial"] = torch.empty(s["nsplit"], co, 3, 3, ci, device=DEV)
    return s


def _blobs(n, side, g):
    """Images of a few smooth components scaled to max 1, as the network gets them."""
    t = torch.linspace(-1, 1, side, device=DEV)
    p = torch.rand(n, 6, 4, generator=g, device=DEV)
    w = 0.05 + 0.25 * p[..., 2]
    gx = torch.exp(-((t - (p[..., :1] - 0.5)) / w[..., None]) ** 2)
    gy = torch.exp(-((t - (p[..., 1:2] - 0.5)) / w[..., None]) ** 2)
    im = torch.einsum("nk,nky,nkx->nyx", p[..., 3], gy, gx)
    return im / im.amax(dim=(1, 2), keepdim=True)


def _solution(b, p):
    x, terms, grad, info = b.fetch(p)
    return x, np.array([terms[q] for q in _lib.TERM_NAMES]), grad, info["nfg"]


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "solve":
        state["batch"].run()
        return _solution(state["batch"], 0)
    if k == "evaluate":
        b = state["batch"]
        b.set_start(0, state["x"])
        b.run(fg_only=True)
        _, terms, grad, _ = b.fetch(0)
        return np.array([terms[q] for q in _lib.TERM_NAMES]), grad
    if k == "batch":
        state["batch"].run()
        state["batch"].images(state["images"])
        return state["images"]
    if k == "survey":
        state["batch"].run()
        got = [_solution(state["batch"], p) for p in range(case["nprob"])]
        return tuple(np.concatenate([np.atleast_1d(q[i]) for q in got]) for i in range(4))
    if k == "imaging":
        out = fftim2d.imaging(**state["kw"])
        return out[0], np.array(out[1:])
    if k == "movie":
        out = fftim3d.imaging(**state["kw"])
        return out[0], np.array(out[1:])
    if k == "nufft":
        vr, vi = fftlib.nufft_fwd_real(state["u"], state["v"], state["img"], nufft_eps=case["eps"])
        dirty = fftlib.nufft_adj_real1d(state["u"], state["v"], state["cr"], state["ci"], case["nx"], case["ny"],
                                        nufft_eps=case["eps"])
        return vr, vi, dirty
    if k == "network":
        return state["net"].forward(state["x"])
    if k == "train":
        net = state["net"]
        net.forward(state["x"])
        loss = net.loss(state["t"])
        net.backward()
        net.adam_step(1e-3)
        return loss, net.grad
    n, h, w, ci, co = (case[q] for q in ("n", "h", "w", "cin", "cout"))
    s = state
    kernels.conv3x3(s["x"], n, h, w, ci, ci, s["w"], s["b"], s["y"], co, co, True)
    kernels.relu_mask(s["act"], co, s["dy"], co, n * h * w, co)
    kernels.conv3x3_wgrad(s["x"], ci, s["dy"], co, n, h, w, ci, co, s["partial"], s["nsplit"], s["dw"])
    kernels.bias_grad(s["dy"], co, n * h * w, co, s["db"])
    kernels.conv3x3(s["dy"], n, h, w, co, co, s["wt"], None, s["dx"], ci, ci, False)
    return s["y"], s["dw"], s["db"], s["dx"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _fg_work(npix, nvis, data, nst, size, w=7):
    """Bytes and operations of one evaluation: image and gradient, uv points,
    values, variances and uv references of the data; interpolation, spreading
    and the data terms (the transforms' few operations a pixel included)."""
    nbl = nst * (nst - 1) / 2
    nscan = nvis / nbl
    cp, ca = nscan * (nst - 1) * (nst - 2) / 2, nscan * nst * (nst - 3) / 2
    nf = nvis if data in ("vis", "all") else 0
    na = nvis if data in ("closure", "all") else 0
    nc = ca if data in ("closure", "all") else 0
    by = 2 * size * npix + 2 * size * nvis + nf * (3 * size + 4) + na * (2 * size + 4) + cp * (2 * size + 12) + nc * (2 * size + 16)
    fl = 8 * w * w * nvis + 40 * (nf + na) + 120 * cp + 150 * nc + 100 * npix
    return by, fl


def _solve_work(npix, nvis, data, nst, size, niter, m=5):
    by, fl = _fg_work(npix, nvis, data, nst, size)
    n_fg = niter + 2
    return n_fg * by + niter * npix * 8 * (10 + 4 * m), n_fg * fl + niter * npix * (16 * m + 40)


def _net_flops(n, side):
    s = {"1": 1, "2": 2, "3": 4, "a": 8, "b": 8}
    return sum(2 * 9 * ci * co * n * (side / (8 if q[0] == "b" else s.get(q[1], 1))) ** 2
               for q, ci, co, _ in layer_specs(CHANNELS))


def work(case):
    k = case["kind"]
    if k in ("solve", "imaging", "evaluate"):
        npix = case["nx"] * case["ny"] * (0.56 if case["window"] else 1.0)
        nvis = case["nscan"] * case["nst"] * (case["nst"] - 1) / 2
        if k == "evaluate":
            b, f = _fg_work(npix, nvis, case["data"], case["nst"], 8)
        else:
            b, f = _solve_work(npix, nvis, case["data"], case["nst"], 8, case["niter"])
    elif k == "batch":
        nvis = case["nscan"] * case["nst"] * (case["nst"] - 1) / 2
        b, f = (case["nprob"] * q for q in _solve_work(case["nx"] ** 2, nvis, "closure", case["nst"], 4, case["niter"]))
    elif k == "survey":
        b = f = 0.0
        for i in range(case["nprob"]):
            nx, nst, nscan = _survey_size(case["first"] + i)
            q = _solve_work(nx * nx, nscan * nst * (nst - 1) / 2, "vis", nst, 8, case["niter"])
            b, f = b + q[0], f + q[1]
    elif k == "movie":
        q = _solve_work(case["nx"] ** 2, case["vis"], "vis", case["nst"], 8, case["niter"])
        b, f = case["nz"] * q[0], case["nz"] * q[1]
    elif k == "nufft":
        w = math.ceil(math.log10(1 / case["eps"])) + 1
        b = 8 * (2 * case["nx"] * case["ny"] + 8 * case["nuv"])
        f = 16 * w * w * case["nuv"] + 40 * case["nx"] * case["ny"]
    elif k in ("network", "train"):
        # every activation written once and read once (forward), weights once; a training step reads the
        # activations again and writes and reads their gradients
        px = case["n"] * case["side"] ** 2
        c1, c2, c3, c4 = CHANNELS
        act = 2 * px * (2 + 4 * c1 + 4 * c2 / 4 + 4 * c3 / 16 + 2 * c4 / 64)
        wts = sum(9 * ci * co for _, ci, co, _ in layer_specs(CHANNELS))
        b, f = 2 * act + 2 * wts, _net_flops(case["n"], case["side"])
        if k == "train":
            b, f = 3 * b + 32 * wts, 3 * f
    else:
        px = case["n"] * case["h"] * case["w"]
        ci, co = case["cin"], case["cout"]
        b = 2 * px * (2 * ci + 3 * co) + 9 * ci * co * 8
        f = 3 * 2 * 9 * ci * co * px
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _grid_phase(kw):
    """exp(i u x) and exp(i v y) factors, pixels counted from nx/2, ny/2 as fortlib counts them."""
    u, v = (torch.as_tensor(np.array(kw[q], dtype=np.float64), device=DEV) for q in ("u", "v"))
    x = torch.arange(int(kw["nx"]), device=DEV, dtype=torch.float64) - int(kw["nx"]) // 2
    y = torch.arange(int(kw["ny"]), device=DEV, dtype=torch.float64) - int(kw["ny"]) // 2
    return u, v, x, y


def _visibilities(img, u, v, x, y, chunk=1 << 14):
    """sum img[y, x] exp(i (u x + v y)), differentiable in img."""
    re, im = [], []
    for s in range(0, u.numel(), chunk):
        a, b = u[s:s + chunk, None] * x, v[s:s + chunk, None] * y
        ar, ai = torch.cos(a) @ img.T, torch.sin(a) @ img.T
        c, d = torch.cos(b), torch.sin(b)
        re.append((ar * c - ai * d).sum(1))
        im.append((ai * c + ar * d).sum(1))
    return torch.cat(re), torch.cat(im)


def _exact_cost(kw, xvec):
    """The cost terms (in _lib.TERM_NAMES' order) and the gradient of the imaging objective."""
    t64 = lambda q: torch.as_tensor(np.array(kw[q], dtype=np.float64).reshape(-1), device=DEV)  # noqa: E731
    nx, ny = int(kw["nx"]), int(kw["ny"])
    pos = torch.as_tensor((np.array(kw["yidx"], dtype=np.int64) - 1) * nx + np.array(kw["xidx"]) - 1, device=DEV)
    x = torch.as_tensor(np.array(xvec), device=DEV).requires_grad_(True)
    img = torch.zeros(ny * nx, dtype=torch.float64, device=DEV).index_put((pos,), x).reshape(ny, nx)
    u, v, gx, gy = _grid_phase(kw)
    vr, vi = _visibilities(img, u, v, gx, gy)
    n = {"fcv": np.size(kw["uvidxfcv"]) if kw["isfcv"] else 0, "amp": np.size(kw["uvidxamp"]) if kw["isamp"] else 0,
         "cp": np.size(kw["cp"]) if kw["iscp"] else 0, "ca": np.size(kw["ca"]) if kw["isca"] else 0}
    w = {q: float(kw["w" + q]) for q in n}
    tot = 2 * n["fcv"] * w["fcv"] + n["amp"] * w["amp"] + n["cp"] * w["cp"] + n["ca"] * w["ca"]
    idx = lambda q: torch.as_tensor(np.array(kw["uvidx" + q], dtype=np.int64), device=DEV)  # noqa: E731
    raw = dict.fromkeys(n, torch.zeros((), dtype=torch.float64, device=DEV))
    amp, ph = torch.sqrt(vr * vr + vi * vi), torch.atan2(vi, vr)
    if n["fcv"]:
        i = idx("fcv")
        j, sg = i.abs() - 1, torch.sign(i).double()
        shift = sg * (u[j] * (float(kw["nxref"]) - nx / 2.0 - 1) + v[j] * (float(kw["nyref"]) - ny / 2.0 - 1))
        dr, di = t64("vfcvr"), t64("vfcvi")
        yr, yi = dr * torch.cos(shift) - di * torch.sin(shift), dr * torch.sin(shift) + di * torch.cos(shift)
        raw["fcv"] = (((yr - vr[j]) ** 2 + (yi - sg * vi[j]) ** 2) / t64("varfcv")).sum()
    if n["amp"]:
        raw["amp"] = ((t64("vamp") - amp[idx("amp").abs() - 1]) ** 2 / t64("varamp")).sum()
    if n["cp"]:
        i = idx("cp")
        raw["cp"] = (2 * (1 - torch.cos(t64("cp") - (ph[i.abs() - 1] * torch.sign(i)).sum(0))) / t64("varcp")).sum()
    if n["ca"]:
        la = torch.log(amp)[idx("ca").abs() - 1]
        raw["ca"] = ((t64("ca") - (la[0] + la[1] - la[2] - la[3])) ** 2 / t64("varca")).sum()
    sab = lambda z: torch.sqrt(z * z + 1e-10)  # noqa: E731
    dx = torch.cat([img[:, 1:] - img[:, :-1], torch.zeros(ny, 1, dtype=img.dtype, device=DEV)], 1).reshape(-1)[pos]
    dy = torch.cat([img[1:] - img[:-1], torch.zeros(1, nx, dtype=img.dtype, device=DEV)], 0).reshape(-1)[pos]
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    lam = {q: float(kw[q + "_l"]) for q in ("l1", "tv", "tsv", "kl", "gs", "tfd", "cen", "sm")}
    reg = dict.fromkeys(lam, zero)
    if lam["l1"] > 0:
        reg["l1"] = lam["l1"] * (t64("l1_wgt") * sab(x)).sum()
    if lam["tv"] > 0:
        e = dx * dx + dy * dy
        reg["tv"] = lam["tv"] * (t64("tv_wgt") * torch.where(e > 1e-20, torch.sqrt(e.clamp_min(1e-20)), zero)).sum()
    if lam["tsv"] > 0:
        reg["tsv"] = lam["tsv"] * (t64("tsv_wgt") * (dx * dx + dy * dy)).sum()
    if lam["kl"] > 0:
        p = t64("kl_wgt")
        reg["kl"] = lam["kl"] * (sab(x) * torch.log(sab(x) / p) + p / math.e).sum()
    if lam["gs"] > 0:
        p = t64("gs_wgt")
        reg["gs"] = lam["gs"] * (sab(x) * (torch.log(sab(x) / p) - 1) + p).sum()
    if lam["tfd"] > 0:
        reg["tfd"] = lam["tfd"] * (x.sum() - float(kw["tfd_tgtfd"])) ** 2
    chi = {q: raw[q] * (w[q] / tot) for q in n}
    f = sum(chi.values()) + sum(reg.values())
    g, = torch.autograd.grad(f, x)
    per = [raw["fcv"] / max(1, 2 * n["fcv"]), raw["amp"] / max(1, n["amp"]), raw["cp"] / max(1, n["cp"]),
           raw["ca"] / max(1, n["ca"])]
    terms = [sum(chi.values())] + per + [sum(reg.values())] + [reg[q] for q in ("l1", "tv", "tsv", "kl", "gs", "tfd", "cen", "sm")] + [f]
    return np.array([float(q) for q in terms]), g.cpu().numpy()


def _conv(x, w, b):
    """3x3 convolution with padding 1 of an NHWC tensor in 64 bits."""
    y = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2), w.permute(0, 3, 1, 2), b, padding=1)
    return y.permute(0, 2, 3, 1)


def _exact_net(x, params):
    pool = lambda t: torch.nn.functional.avg_pool2d(t.permute(0, 3, 1, 2), 2).permute(0, 2, 3, 1)  # noqa: E731
    up = lambda t: t.repeat_interleave(2, 1).repeat_interleave(2, 2)  # noqa: E731
    lay = lambda q, t: torch.relu(_conv(t, *params[q]))  # noqa: E731
    s1 = lay("e1b", lay("e1a", x))
    s2 = lay("e2b", lay("e2a", pool(s1)))
    s3 = lay("e3b", lay("e3a", pool(s2)))
    t = lay("bb", lay("ba", pool(s3)))
    t = lay("d3b", lay("d3a", torch.cat([up(t), s3], 3)))
    t = lay("d2b", lay("d2a", torch.cat([up(t), s2], 3)))
    t = lay("d1b", lay("d1a", torch.cat([up(t), s1], 3)))
    return _conv(t, *params["head"])


def _params64(net):
    """The network's weights as its kernels use them, in 64 bits."""
    return {q: tuple(torch.as_tensor(a, dtype=torch.float64, device=DEV) for a in p) for q, p in net.params_bf16().items()}


def exact(case, seed):
    k = case["kind"]
    if k == "evaluate":
        if case["data"] == "all":  # the centroid term's exponent is left to the framework's tests
            return None
        kw = _kwargs(case["nx"], case["ny"], case["pix"], case["data"], case["nst"], case["nscan"], 1, _rng(seed),
                     case["window"])
        return _exact_cost(kw, kw["iin"])
    if k == "nufft":
        s = prepare(case, seed)
        u, v, x, y = _grid_phase({"u": s["u"], "v": s["v"], "nx": case["nx"], "ny": case["ny"]})
        vr, vi = _visibilities(torch.as_tensor(s["img"], device=DEV).T.contiguous(), u, v, x, y)
        cr, ci = torch.as_tensor(s["cr"], device=DEV), torch.as_tensor(s["ci"], device=DEV)
        dirty = torch.zeros(case["ny"], case["nx"], dtype=torch.float64, device=DEV)
        for a in range(0, case["nuv"], 1 << 14):
            p, q = u[a:a + (1 << 14), None] * x, v[a:a + (1 << 14), None] * y
            c, d = cr[a:a + (1 << 14), None], ci[a:a + (1 << 14), None]
            dirty += (c * torch.cos(q) - d * torch.sin(q)).T @ torch.cos(p) - (c * torch.sin(q) + d * torch.cos(q)).T @ torch.sin(p)
        return vr.cpu().numpy(), vi.cpu().numpy(), dirty.reshape(-1).cpu().numpy()
    if k == "network":
        s = prepare(case, seed)
        with torch.no_grad():
            return torch.cat([_exact_net(q[..., None].to(torch.bfloat16).double(), _params64(s["net"]))
                              for q in s["x"].split(16)])
    if k == "train":
        s = prepare(case, seed)
        par = {q: tuple(a.clone().requires_grad_(True) for a in p) for q, p in _params64(s["net"]).items()}
        total = 0.0
        for q, t in zip(s["x"].split(8), s["t"].split(8)):
            y = _exact_net(q[..., None].to(torch.bfloat16).double(), par)[..., 0]
            loss = ((y - t.double()) ** 2).sum() / s["t"].numel()
            loss.backward()
            total += float(loss.detach())
        grads = [a.grad.reshape(-1) for q, _, _, _ in layer_specs(CHANNELS) for a in par[q]]
        return torch.tensor(total, dtype=torch.float64), torch.cat(grads)
    if k == "layer":
        s = prepare(case, seed)
        x = s["x"].double().requires_grad_(True)
        w, b = s["w"].double().requires_grad_(True), s["b"].double().requires_grad_(True)
        dy = torch.where(s["act"] > 0, s["dy"], torch.zeros_like(s["dy"])).double()
        ys = []
        for a in range(0, case["n"], 8):
            y = _conv(x[a:a + 8], w, b)
            y.backward(dy[a:a + 8])
            ys.append(torch.relu(y.detach()))
        return torch.cat(ys), w.grad, b.grad, x.grad
    return None  # an iterative solve has no value of its own beside the one its steps give
