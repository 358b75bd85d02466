"""Depthwise layers on the staged-plane kernels: kernel sizes, strides, paddings, multipliers and maps that the bulk-copy 3x3 path
does not take, at the edges of strips, bands, channel groups and clusters."""
import numpy as np
import pytest

from conftest import assert_parity

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def F():
    from cunn_b200 import functional
    return functional


@pytest.mark.parametrize("shape", [
    # N, C, H, W, M, k, d, padH, padW
    (3, 10, 57, 43, 1, 5, 2, 2, 2),      # one plane per tile, ragged strips
    (2, 3, 200, 33, 1, 5, 1, 2, 2),      # several bands
    (2, 2, 150, 131, 1, 7, 2, 3, 3),     # bands at stride 2, odd rows
    (17, 6, 7, 7, 1, 7, 1, 3, 3),        # many planes per tile; more images than ranks
    (5, 7, 14, 14, 2, 5, 1, 2, 2),       # multiplier 2
    (2, 5, 29, 37, 3, 3, 2, 1, 1),       # multiplier 3 at stride 2
    (2, 8, 37, 29, 1, 3, 1, 1, 1),       # 3x3 with planes of an odd size
    (2, 4, 16, 18, 1, 3, 1, 0, 2),       # paddings that differ
    (2, 4, 11, 9, 1, 5, 2, 4, 0),        # padding of k - 1 and none
    (2, 3, 12, 12, 1, 3, 2, 3, 3),       # padding of the kernel size: outer outputs see padding only
    (1, 1, 5, 1200, 1, 7, 1, 3, 3),      # long rows: strips of one band row group
    (1, 2, 3, 4000, 1, 7, 1, 3, 3),      # rows too long for a tile: the kernels for any shape
    (1, 3, 1, 1, 1, 5, 2, 2, 2),         # a single pixel
    (40, 2, 20, 20, 1, 3, 1, 0, 0),      # more terms per thread than one fp32 chain takes
])
def test_staged_plane_shapes(F, ref64, ref32, shape):
    N, C, H, W, M, k, d, pH, pW = shape
    rng = np.random.default_rng(abs(hash(shape)) % 99991)
    oH, oW = (H + 2 * pH - k) // d + 1, (W + 2 * pW - k) // d + 1
    x, gy = rng.standard_normal((N, C, H, W)).astype(np.float32), rng.standard_normal((N, C * M, oH, oW)).astype(np.float32)
    w, b = rng.uniform(-1, 1, (M, C, k, k)).astype(np.float32), rng.uniform(-1, 1, (M, C)).astype(np.float32)
    gw0, gb0 = rng.standard_normal((M, C, k, k)).astype(np.float32), rng.standard_normal((M, C)).astype(np.float32)
    y = F.dwconv_forward(dev(x), dev(w), dev(b), d, d, pH, pW).cpu().numpy()
    assert_parity("y", y, ref64.dwconv_forward(x, w, b, d, d, pH, pW), 1e-5, port=lambda: ref32.dwconv_forward(x, w, b, d, d, pH, pW))
    gx = F.dwconv_grad_input(dev(gy), dev(w), H, W, d, d, pH, pW).cpu().numpy()
    assert_parity("gx", gx, ref64.dwconv_grad_input(gy, w, H, W, d, d, pH, pW), 1e-5, port=lambda: ref32.dwconv_grad_input(gy, w, H, W, d, d, pH, pW))
    gw, gb = dev(gw0), dev(gb0)
    F.dwconv_acc_grad(dev(x), dev(gy), gw, gb, d, d, pH, pW, 0.75)
    want = ref64.dwconv_acc_grad(x, gy, gw0.copy(), gb0.copy(), d, d, pH, pW, 0.75)
    port = ref32.dwconv_acc_grad(x, gy, gw0.copy(), gb0.copy(), d, d, pH, pW, 0.75)
    assert_parity("gw", gw.cpu().numpy(), want[0], 1e-5, port=port[0])
    assert_parity("gb", gb.cpu().numpy(), want[1], 1e-5, port=port[1])
    # the order of the sums is fixed: the same bits again, without a bias gradient too
    gw2 = dev(gw0)
    F.dwconv_acc_grad(dev(x), dev(gy), gw2, None, d, d, pH, pW, 0.75)
    assert np.array_equal(gw.cpu().numpy(), gw2.cpu().numpy())


@pytest.mark.parametrize("d", [1, 2])
def test_weights_that_are_not_finite_stay_off_the_padding(F, d):
    import torch
    x, w = torch.ones(1, 3, 9, 9, device="cuda"), torch.full((1, 3, 5, 5), 0.25, device="cuda")
    w[0, 1, 0, 2] = float("inf")
    w[0, 2, 4, 4] = float("nan")
    y = F.dwconv_forward(x, w, None, d, d, 2, 2)
    xd, wd = x.cpu().double(), w.cpu().double().view(3, 1, 5, 5)
    cols = torch.nn.functional.unfold(torch.ones(1, 3, 9, 9).double(), 5, padding=2, stride=d).view(3, 25, -1)     # 0: padding
    want = torch.where(cols > 0, wd.view(3, 25, 1), torch.zeros(1, dtype=torch.double)).sum(1).view(y.shape)
    assert torch.allclose(y.cpu().double(), want, equal_nan=True)
    gx = F.dwconv_grad_input(torch.ones_like(y), w, 9, 9, d, d, 2, 2).cpu()
    o = y.shape[2]
    ref = torch.zeros(3, 9, 9, dtype=torch.double)
    for oh in range(o):
        for ow in range(o):
            for kh in range(5):
                for kw in range(5):
                    h, q = oh * d - 2 + kh, ow * d - 2 + kw
                    if 0 <= h < 9 and 0 <= q < 9:
                        ref[:, h, q] += wd[:, 0, kh, kw]
    assert torch.allclose(gx[0].double(), ref, equal_nan=True)


@pytest.mark.parametrize("what", ["inf", "nan", "gpu nan"])
@pytest.mark.parametrize("shape", [
    # N, C, H, W, M, k, d, padH, padW
    (3, 4, 10, 12, 1, 5, 1, 0, 0),       # the kernel for any shape
    (20, 40, 10, 12, 1, 5, 1, 0, 0),     # six rows of outputs: the second strip of four ends in two that do not exist
    (12, 60, 23, 21, 2, 5, 2, 2, 2),     # rows past the last window, padding on every side
    (40, 2, 9, 9, 1, 3, 1, 1, 0),        # several ranks
    (1, 2, 90, 70, 1, 7, 1, 3, 2),       # several bands
])
def test_parameter_gradient_not_finite(F, shape, what):
    """An infinity or a NaN in x or gy reaches exactly the taps whose products read it."""
    import torch
    N, C, H, W, M, k, d, pH, pW = shape
    oH, oW = (H + 2 * pH - k) // d + 1, (W + 2 * pW - k) // d + 1
    value = {"inf": float("inf"), "nan": float("nan")}.get(what)
    if value is None:
        value = torch.full((1,), float("inf"), device="cuda")
        value = (value - value)[0]
    g = torch.Generator(device="cuda").manual_seed(5)
    for where in ("x last row", "x inside", "gy corner", "gy inside"):
        x, gy = torch.randn(N, C, H, W, device="cuda", generator=g), torch.randn(N, C * M, oH, oW, device="cuda", generator=g)
        if where == "x last row":
            x[N - 1, C - 1, H - 1, W // 2] = value
        elif where == "x inside":
            x[0, 0, H // 2, W // 2] = value
        elif where == "gy corner":
            gy[N - 1, C * M - 1, oH - 1, oW - 1] = gy[0, 0, 0, 0] = value
        else:
            gy[0, 0, oH // 2, oW // 2] = value
        gw, gb = torch.zeros(M, C, k, k, device="cuda"), torch.zeros(M, C, device="cuda")
        F.dwconv_acc_grad(x, gy, gw, gb, d, d, pH, pW)
        # tap by tap over the windows that are inside the image
        xd, gd = x.cpu().double(), gy.cpu().double().view(N, C, M, oH, oW)
        want = torch.zeros(M, C, k, k, dtype=torch.double)
        for kh in range(k):
            for kw in range(k):
                oh = [o for o in range(oH) if 0 <= o * d - pH + kh < H]
                ow = [o for o in range(oW) if 0 <= o * d - pW + kw < W]
                if oh and ow:
                    xs = xd[:, :, [o * d - pH + kh for o in oh]][:, :, :, [o * d - pW + kw for o in ow]]
                    want[:, :, kh, kw] = (xs[:, :, None] * gd[:, :, :, oh][..., ow]).sum((0, 3, 4)).t()
        assert torch.allclose(gw.cpu().double(), want, rtol=1e-4, atol=1e-3, equal_nan=True), where
        assert torch.allclose(gb.cpu().double(), gd.sum((0, 3, 4)).t(), rtol=1e-4, atol=1e-3, equal_nan=True), where


@pytest.mark.parametrize("shape", [(16, 64, 56, 56, 5, 1), (29, 36, 37, 42, 7, 1), (98, 32, 51, 39, 3, 2)])
def test_parameter_gradient_sums_in_fp64(F, shape):
    """2-norm of the error: eight fp32 terms, then fp64, for the taps; fp64 throughout for the bias."""
    import torch
    N, C, H, W, k, d = shape
    p, g = k // 2, torch.Generator(device="cuda").manual_seed(7)
    oH, oW = (H + 2 * p - k) // d + 1, (W + 2 * p - k) // d + 1
    x, gy = torch.randn(N, C, H, W, device="cuda", generator=g), torch.randn(N, C, oH, oW, device="cuda", generator=g)
    cols = torch.nn.functional.unfold(x.double(), k, padding=p, stride=d).view(N, C, k * k, oH * oW)
    want = torch.einsum("nckp,ncp->ck", cols, gy.double().view(N, C, -1)).view(1, C, k, k)
    gw, gb = torch.zeros(1, C, k, k, device="cuda"), torch.zeros(1, C, device="cuda")
    F.dwconv_acc_grad(x, gy, gw, gb, d, d, p, p)
    # a chain of n FMAs is about 1.8e-8 sqrt(n + 1) off, the result's rounding 3.5e-8: 6.4e-8 for n = 8 (1.1e-7 for 32)
    assert float((gw.double() - want).norm() / want.norm()) <= 7e-8
    b = gy.double().sum((0, 2, 3)).view(1, C)
    assert float((gb.double() - b).abs().max() / b.abs().max()) <= 2.0 ** -24


@pytest.mark.parametrize("shape", [
    # N, C, H, W, M, k, d, padH, padW: the same edges with as much work as the staged form is chosen for in every pass
    (8, 200, 57, 43, 1, 5, 2, 2, 2), (6, 60, 200, 33, 1, 5, 1, 2, 2), (6, 40, 150, 131, 1, 7, 2, 3, 3), (64, 300, 7, 7, 1, 7, 1, 3, 3),
    (40, 70, 14, 14, 2, 5, 1, 2, 2), (30, 50, 29, 37, 3, 3, 2, 1, 1), (12, 144, 37, 29, 1, 3, 1, 1, 1), (40, 100, 16, 18, 1, 3, 1, 0, 2),
    (12, 300, 30, 26, 1, 5, 2, 4, 0), (40, 90, 33, 33, 1, 3, 2, 3, 3), (300, 40, 20, 20, 1, 3, 1, 0, 0), (24, 90, 40, 12, 1, 5, 1, 0, 0),
    (30, 100, 31, 29, 1, 7, 2, 3, 3),
    # layers that the kernels for any shape take although a tile plan exists
    (70, 56, 9, 9, 1, 5, 2, 2, 2), (12, 47, 12, 9, 1, 3, 2, 1, 1), (1, 23, 35, 35, 2, 3, 2, 1, 1),
])
def test_both_sides_of_the_staging_rule(F, ref64, ref32, shape):
    test_staged_plane_shapes(F, ref64, ref32, shape)


@pytest.mark.parametrize("width", [8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257, 512, 517])
@pytest.mark.parametrize("d", [1, 2])
def test_rows_that_lanes_share(F, width, d):
    """Rows of staged columns at the edges of what 8 to 256 lanes copy, two columns each, and of one round of them.  Against fp64, with the
    bound of a chain of n fp32 multiply-adds: (n + 1) units of 2^-24 of the sum of the terms' magnitudes; n = 25 taps for y and gx, eight
    products and fp64 for gw and gb."""
    import torch
    N, C, H, k, p = 7, 24, 11, 5, 2
    W = max((width - k) // d * d + k - 2 * p, 4)          # staged columns: (oW - 1) d + k
    g = torch.Generator(device="cuda").manual_seed(width)
    x, w = torch.randn(N, C, H, W, device="cuda", generator=g), torch.randn(1, C, k, k, device="cuda", generator=g)
    b = torch.randn(1, C, device="cuda", generator=g)
    x64, w64 = x.double().requires_grad_(), w.double().view(C, 1, k, k).requires_grad_()
    y64 = torch.nn.functional.conv2d(x64, w64, b.double().view(-1), d, p, groups=C)
    gy = torch.randn(y64.shape, device="cuda", generator=g)
    gx64, gw64 = torch.autograd.grad(y64, (x64, w64), gy.double())
    xa, wa = x64.detach().abs().requires_grad_(), w64.detach().abs().requires_grad_()
    ya = torch.nn.functional.conv2d(xa, wa, b.double().abs().view(-1), d, p, groups=C)
    gxa, gwa = torch.autograd.grad(ya, (xa, wa), gy.double().abs())
    gw, gb = torch.zeros_like(w), torch.zeros_like(b)
    F.dwconv_acc_grad(x, gy, gw, gb, d, d, p, p)
    gb64, gba = gy.double().sum((0, 2, 3)).view(1, C), gy.double().abs().sum((0, 2, 3)).view(1, C)
    for what, got, want, size, n in (("gb", gb, gb64, gba, 8), ("y", F.dwconv_forward(x, w, b, d, d, p, p), y64, ya, k * k),
                                     ("gx", F.dwconv_grad_input(gy, w, H, W, d, d, p, p), gx64, gxa, k * k),
                                     ("gw", gw.view(C, 1, k, k), gw64, gwa, 8)):
        assert bool(((got.double() - want).abs() <= (n + 1) * 2.0 ** -24 * size).all()), what
