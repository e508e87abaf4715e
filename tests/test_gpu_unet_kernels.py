"""U-Net kernels at the sizes where their paths change: 16-byte and scalar
channel access, one-channel convolutions, few and many splits.

Elementwise results and the one-channel layers are exact (the same products
in the same order as the general kernels); sums are held to the worst case of
an FP32 summation, n 2^-24 times the sum of magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand(shape, seed, scale=1.0):
    import torch
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("C,ld,npix", [(24, 24, 1000), (24, 72, 333), (8, 16, 1), (192, 288, 70), (1, 1, 4097),
                                       (5, 7, 129)])
@pytest.mark.parametrize("masked", [False, True])
def test_bias_grad_and_mask(C, ld, npix, masked):
    import torch
    from smili_b200.warmstart import kernels as K
    dy, y = _rand((npix, ld), 1), _rand((npix, ld), 2)
    y[::3, 0] = 0.0
    y[0, 0] = float("nan")
    want = dy.clone()
    db = torch.full((C,), 3.0, device="cuda")
    if masked:
        want[:, :C] = torch.where(y[:, :C] > 0, dy[:, :C], torch.zeros_like(dy[:, :C]))
        separate = dy.clone()
        K.relu_mask(y, ld, separate, ld, npix, C)
        assert torch.equal(separate, want)
        K.relu_bias_grad(y, ld, dy, ld, npix, C, db, accumulate=True)
    else:
        K.bias_grad(dy, ld, npix, C, db, accumulate=True)
    assert torch.equal(dy, want)  # masked in place, nothing past C touched
    ref = 3.0 + want[:, :C].double().sum(0)
    bound = (npix + 1) * 2.0 ** -24 * (3.0 + want[:, :C].double().abs().sum(0))
    assert ((db.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("C,pad", [(24, 0), (24, 16), (8, 3), (5, 0)])
def test_pool_and_upsample(C, pad):
    import torch
    from smili_b200.warmstart import kernels as K
    N, H, W, ld = 3, 6, 10, C + pad
    x = _rand((N, H, W, ld), 3)
    f = x[..., :C].float()
    y = torch.zeros(N, H // 2, W // 2, ld, dtype=torch.bfloat16, device="cuda")
    K.avgpool2(x, ld, y, ld, N, H, W, C)
    s = ((f[:, ::2, ::2] + f[:, ::2, 1::2]) + f[:, 1::2, ::2]) + f[:, 1::2, 1::2]
    assert torch.equal(y[..., :C], (0.25 * s).to(torch.bfloat16))
    up = torch.zeros(N, 2 * H, 2 * W, ld, dtype=torch.bfloat16, device="cuda")
    K.upsample2(x, ld, up, ld, N, H, W, C)
    assert torch.equal(up[..., :C], x[..., :C].repeat_interleave(2, 1).repeat_interleave(2, 2))
    for acc in (False, True):
        old = _rand((N, H, W, ld), 4)
        d = old.clone()
        K.avgpool2_bwd(y, ld, d, ld, N, H, W, C, accumulate=acc)
        want = 0.25 * y[..., :C].float().repeat_interleave(2, 1).repeat_interleave(2, 2)
        assert torch.equal(d[..., :C], (want + old[..., :C].float() if acc else want).to(torch.bfloat16))
        old = _rand((N, H // 2, W // 2, ld), 5)
        d = old.clone()
        K.upsample2_bwd(x, ld, d, ld, N, H // 2, W // 2, C, accumulate=acc)
        assert torch.equal(d[..., :C], (s + old[..., :C].float() if acc else s).to(torch.bfloat16))
        assert torch.equal(d[..., C:], old[..., C:])


@pytest.mark.parametrize("Cout,H,W,ldy", [(24, 64, 32, 24), (1, 5, 7, 1), (13, 70, 19, 15), (40, 65, 16, 72)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_one_channel_conv_equals_general_kernel(Cout, H, W, ldy, accumulate):
    import torch
    from smili_b200.warmstart import kernels as K
    x, w = _rand((2, H, W, 1), 6), _rand((Cout, 3, 3, 1), 7, 0.3)
    b = torch.randn(Cout, device="cuda")
    out = []
    for path in (0, 1):
        K.set_conv_path(path)
        y = _rand((2, H, W, ldy), 8)
        K.conv3x3(x, 2, H, W, 1, 1, w, b, y, ldy, Cout, True, accumulate)
        out.append(y)
    K.set_conv_path(0)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("thin_x", [True, False])
@pytest.mark.parametrize("C,H,W,nsplit", [(24, 40, 33, 5), (8, 3, 2, 1), (48, 16, 16, 40)])
def test_one_channel_weight_gradient(thin_x, C, H, W, nsplit):
    import torch
    from smili_b200.warmstart import kernels as K
    N, ci, co = 3, 1 if thin_x else C, C if thin_x else 1
    x, dy = _rand((N, H, W, ci), 9), _rand((N, H, W, co), 10)
    got = []
    for path in (0, 1):  # the general kernel makes the same products in the same order
        K.set_conv_path(path)
        part = torch.full((nsplit, co, 9, ci), float("nan"), device="cuda")
        dw = torch.ones(co, 9, ci, device="cuda")
        K.conv3x3_wgrad(x, ci, dy, co, N, H, W, ci, co, part, nsplit, dw, accumulate=True)
        got.append(dw)
    K.set_conv_path(0)
    assert torch.equal(got[0], got[1])
    xp = np.pad(x.double().cpu().numpy(), ((0, 0), (1, 1), (1, 1), (0, 0)))
    d = dy.double().cpu().numpy()
    ref, mag = np.ones((co, 9, ci)), np.ones((co, 9, ci))
    for t in range(9):
        s = xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W]
        ref[:, t] += np.einsum("nhwo,nhwi->oi", d, s)
        mag[:, t] += np.einsum("nhwo,nhwi->oi", np.abs(d), np.abs(s))
    # products exact in FP32; additions on the tensor cores may truncate (2^-23 each)
    assert (np.abs(dw.double().cpu().numpy() - ref) <= (N * H * W + nsplit) * 2.0 ** -23 * mag).all()


# (N, H, W, Cin, Cout, ldx, ldy): tiles and groups with remainders, 32- and
# 64-channel planes, resident and streamed weights, one to four tiles per
# group, several output-channel and input-channel blocks
CONV = [(2, 5, 3, 8, 1, 8, 1), (3, 17, 9, 24, 24, 72, 40), (150, 20, 12, 24, 24, 24, 24), (40, 33, 20, 72, 24, 72, 24),
        (2, 16, 16, 48, 48, 48, 48), (3, 32, 32, 144, 48, 144, 48), (2, 16, 24, 96, 192, 96, 192),
        (40, 32, 32, 192, 192, 192, 288), (1, 16, 16, 192, 272, 192, 272), (1, 20, 12, 640, 40, 640, 40)]


@pytest.mark.parametrize("N,H,W,Cin,Cout,ldx,ldy", CONV)
@pytest.mark.parametrize("accumulate", [False, True])
def test_tensor_core_convolution(N, H, W, Cin, Cout, ldx, ldy, accumulate):
    import torch
    from smili_b200.warmstart import kernels as K
    x, w = _rand((N, H, W, ldx), 11), _rand((Cout, 3, 3, Cin), 12, 1 / (3 * Cin ** 0.5))
    b = torch.randn(Cout, device="cuda")
    y = _rand((N, H, W, ldy), 13)
    old = y.clone()
    K.conv3x3(x, N, H, W, Cin, ldx, w, b, y, ldy, Cout, True, accumulate)
    assert K.tc_status() == 0
    xd, wd = x[..., :Cin].double().permute(0, 3, 1, 2), w.double().permute(0, 3, 1, 2)
    add = old[..., :Cout].double() if accumulate else 0.0
    ref = torch.relu(torch.nn.functional.conv2d(xd, wd, b.double(), padding=1)).permute(0, 2, 3, 1) + add
    mag = torch.nn.functional.conv2d(xd.abs(), wd.abs(), b.double().abs(), padding=1).permute(0, 2, 3, 1) + abs(add)
    # FP32 sums of 9 Cin products and the bf16 rounding of the result
    bound = (9 * Cin + 2) * 2.0 ** -23 * mag + 2.0 ** -8 * ref.abs()
    assert ((y[..., :Cout].double() - ref).abs() <= bound).all()
    assert torch.equal(y[..., Cout:], old[..., Cout:])


# (N, H, W, Cin, Cout, nsplit): one, three and nine taps per CTA, either side
# on M, several M and N tiles, splits with and without pixels
WGRAD = [(1, 8, 16, 8, 16, 1), (3, 17, 9, 24, 24, 4), (2, 32, 32, 72, 24, 7), (64, 16, 32, 24, 24, 128),
         (2, 20, 40, 96, 96, 5), (2, 16, 16, 288, 96, 3), (4, 32, 32, 192, 192, 8), (1, 16, 16, 16, 272, 2),
         (1, 9, 9, 24, 24, 30)]


@pytest.mark.parametrize("N,H,W,Cin,Cout,nsplit", WGRAD)
def test_tensor_core_weight_gradient(N, H, W, Cin, Cout, nsplit):
    import torch
    from smili_b200.warmstart import kernels as K
    ldx, ldd = Cin + 8, Cout + 16
    x, dy = _rand((N, H, W, ldx), 14), _rand((N, H, W, ldd), 15)
    part = torch.full((nsplit, Cout, 9, Cin), float("nan"), device="cuda")
    dw = torch.ones(Cout, 3, 3, Cin, device="cuda")
    K.conv3x3_wgrad(x, ldx, dy, ldd, N, H, W, Cin, Cout, part, nsplit, dw, accumulate=True)
    assert K.tc_status() == 0

    def grad(a, d):
        w = torch.zeros(Cout, Cin, 3, 3, dtype=torch.float64, device="cuda", requires_grad=True)
        y = torch.nn.functional.conv2d(a.double().permute(0, 3, 1, 2), w, padding=1)
        y.backward(d.double().permute(0, 3, 1, 2))
        return w.grad.permute(0, 2, 3, 1) + 1.0
    xs, ds = x[..., :Cin], dy[..., :Cout]
    bound = (N * H * W + nsplit) * 2.0 ** -23 * grad(xs.abs(), ds.abs())
    assert ((dw.double() - grad(xs, ds)).abs() <= bound).all()


@pytest.mark.parametrize("C,ld,npix", [(24, 24, 1000), (8, 8, 1), (5, 7, 70001), (192, 288, 4097)])
@pytest.mark.parametrize("masked", [False, True])
def test_bias_grad_without_clusters(C, ld, npix, masked):
    """The kernels for a device that cannot hold a 16-CTA cluster add in the
    same order: equal results."""
    import torch
    from smili_b200.warmstart import kernels as K
    y, got = _rand((npix, ld), 2), []
    for path in (0, 1):
        K.set_conv_path(path)
        dy, db = _rand((npix, ld), 1), torch.full((C,), 3.0, device="cuda")
        if masked:
            K.relu_bias_grad(y, ld, dy, ld, npix, C, db, accumulate=True)
        else:
            K.bias_grad(dy, ld, npix, C, db, accumulate=True)
        got.append((dy, db))
    K.set_conv_path(0)
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
