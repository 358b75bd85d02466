"""SpatialConvolutionMM: tcgen05 implicit-GEMM kernels (flat C ABI) against the CPU oracle and the committed
PyTorch-CPU fixtures.  GEMM-path tolerance 1e-4 (element-wise relative error with a 1 % floor)."""
import numpy as np
import pytest

from conftest import golden, rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-4


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.detach().cpu().numpy()


@pytest.fixture(scope="module")
def F():
    import cunn_b200.functional as F
    from cunn_b200 import device_status
    yield F
    assert device_status() == 0


def make_case(seed, N, C, H, W, K, k, d, pad, bias=True):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    w = (rng.standard_normal((K, C, k, k)) * np.sqrt(2.0 / (C * k * k))).astype(np.float32)
    b = rng.uniform(-0.5, 0.5, K).astype(np.float32) if bias else None
    oH, oW = (H + 2 * pad - k) // d + 1, (W + 2 * pad - k) // d + 1
    gy = rng.standard_normal((N, K, oH, oW)).astype(np.float32)
    gw0 = rng.standard_normal((K, C, k, k)).astype(np.float32)
    gb0 = rng.standard_normal(K).astype(np.float32) if bias else None
    return x, w, b, gy, gw0, gb0


def run_all(F, x, w, b, gy, gw0, gb0, d, pad, scale):
    H, W = x.shape[2:]
    y = F.convmm_forward(dev(x), dev(w), None if b is None else dev(b), d, d, pad, pad)
    gx = F.convmm_grad_input(dev(gy), dev(w), H, W, d, d, pad, pad)
    gw = dev(gw0)
    gb = None if gb0 is None else dev(gb0)
    F.convmm_acc_grad(dev(x), dev(gy), gw, gb, d, d, pad, pad, scale)
    torch.cuda.synchronize()
    return host(y), host(gx), host(gw), None if gb is None else host(gb)


def check_against_oracle(ref64, F, x, w, b, gy, gw0, gb0, d, pad, scale):
    H, W = x.shape[2:]
    y, gx, gw, gb = run_all(F, x, w, b, gy, gw0, gb0, d, pad, scale)
    assert rel_err(y, ref64.convmm_forward(x, w, b, d, d, pad, pad)) < TOL
    assert rel_err(gx, ref64.convmm_grad_input(gy, w, H, W, d, d, pad, pad)) < TOL
    rgw, rgb = ref64.convmm_acc_grad(x, gy, gw0, gb0, d, d, pad, pad, scale)
    assert rel_err(gw, rgw) < TOL
    if gb0 is not None:
        assert rel_err(gb, rgb) < TOL


@pytest.mark.parametrize("name", ["convmm_3x3", "convmm_1x1", "convmm_s2"])
def test_convmm_golden(F, name):
    g = golden(name)
    K, k, d, pad, has_b = [int(v) for v in g["params"]]
    y, gx, gw, gb = run_all(F, g["x"], g["w"], g["b"] if has_b else None, g["gy"], g["gw0"],
                            g["gb0"] if has_b else None, d, pad, float(g["scale"]))
    assert rel_err(y, g["y"]) < TOL
    assert rel_err(gx, g["gx"]) < TOL
    assert rel_err(gw, g["gw"]) < TOL
    if has_b:
        assert rel_err(gb, g["gb"]) < TOL


@pytest.mark.parametrize("shape", [
    # N, C, H, W, K, k, d, pad, bias
    (2, 16, 14, 14, 32, 3, 1, 1, True),      # small 3x3
    (3, 64, 14, 14, 256, 1, 1, 0, True),     # 1x1, several N tiles
    (2, 3, 32, 32, 32, 3, 2, 1, True),       # MobileNet stem geometry (reduced): Kd = 27
    (2, 32, 28, 28, 64, 1, 1, 0, True),      # MobileNet pointwise geometry
    (4, 256, 7, 7, 256, 1, 1, 0, False),     # 7x7 planes (49 pixels: no 16-byte alignment)
    (2, 24, 9, 11, 40, 3, 1, 1, True),       # odd sizes, K not a multiple of 8
    (1, 8, 12, 12, 300, 3, 1, 0, True),      # pad 0, K > 256
    (2, 5, 10, 10, 7, 5, 2, 2, True),        # 5x5 stride 2 (generic k decomposition, gather dgrad)
    (2, 130, 6, 6, 20, 3, 1, 1, True),       # Kd = 1170: many k-blocks, ragged tail
    (9, 4, 5, 5, 4, 1, 2, 0, True),          # 1x1 stride 2
    (2, 3, 20, 20, 8, 7, 2, 3, True),        # 7x7 (49 taps): the kernel for more than 32 taps
    (2, 6, 12, 12, 10, 7, 1, 3, False),      # 7x7 stride 1: tensor-core input gradient of that kernel
    (3, 3, 17, 19, 32, 3, 1, 1, True),       # first-layer kernels: stride 1, odd sizes
    (2, 3, 16, 16, 32, 3, 2, 0, False),      # first-layer kernels: no padding, no bias
    (80, 3, 64, 64, 32, 3, 2, 1, True),      # first-layer kernels: more pixel tiles than CTAs
    (8, 32, 56, 56, 64, 1, 1, 0, True),      # pointwise, one k-block, more tiles than SMs (persistent loop)
    (16, 128, 28, 28, 128, 1, 1, 0, True),   # pointwise, four k-blocks, two accumulator sets
    (2, 1024, 14, 14, 192, 1, 1, 0, False),  # pointwise, long reduction, ragged second column tile
    (2, 30, 6, 6, 50, 1, 1, 0, True),        # pointwise, channel counts not multiples of 4
    (3, 20, 5, 5, 36, 1, 1, 0, True),        # pointwise, 25-pixel planes (scalar loads)
    (40, 512, 7, 7, 96, 1, 1, 0, True),      # pointwise, 49-pixel planes, several row tiles
    (64, 1024, 1, 1, 1000, 1, 1, 0, True),   # classifier geometry: one pixel per image
])
def test_convmm_shapes(F, ref64, shape):
    N, C, H, W, K, k, d, pad, bias = shape
    case = make_case(abs(hash(shape)) % 99991, N, C, H, W, K, k, d, pad, bias)
    check_against_oracle(ref64, F, *case, d, pad, 0.75)


@pytest.fixture(params=[1, 0], ids=["tma", "element-copy"])
def pointwise_loader(request):
    """1x1 convolutions have two operand loaders: tensor-map copies (aligned tensors) and element copies."""
    from cunn_b200._lib import lib
    lib.cunn_b200_convmm_set_tma(request.param)
    yield request.param
    lib.cunn_b200_convmm_set_tma(1)


@pytest.mark.parametrize("shape", [
    # N, C, H, W, K, bias
    (3, 64, 14, 14, 256, True),      # 196-pixel planes: 7 groups of 32, the last one 4 pixels wide; two column tiles
    (5, 96, 14, 14, 40, False),      # row tiles that end inside an image and past the last image; K < 64
    (2, 32, 28, 28, 64, True),       # 784 pixels: 24.5 groups
    (3, 32, 56, 56, 64, True),       # 3136 = 98 x 32 pixels: bulk-store epilogue, one k-block
    (2, 256, 32, 32, 200, True),     # 1024-pixel planes, 8 k-blocks, ragged column tile
    (16, 128, 28, 28, 128, True),    # four k-blocks, two accumulator sets, several tiles per CTA
    (4, 1024, 14, 14, 256, False),   # long reduction: four accumulators, one set
    (3, 40, 64, 64, 24, True),       # 4096-pixel planes, narrow column tile (32): per-column bulk stores
    (2, 64, 40, 40, 128, False),     # 1600-pixel planes: tiles that cross an image boundary in the bulk-store epilogue
    (6, 100, 6, 6, 20, True),        # 36-pixel planes (2 groups per image), C not a multiple of 32
    (2, 36, 2, 2, 24, True),         # 4-pixel planes
    (130, 64, 2, 4, 32, True),       # many tiny images: more groups than one wave of row tiles
])
def test_convmm_pointwise_both_loaders(F, ref64, shape, pointwise_loader):
    N, C, H, W, K, bias = shape
    case = make_case(abs(hash(shape)) % 99991, N, C, H, W, K, 1, 1, 0, bias)
    check_against_oracle(ref64, F, *case, 1, 0, 0.75)


def test_convmm_depthwise_equivalence(F):
    # The reference's own depthwise test (test.lua:6602-6661): depthwise forward == per-channel
    # SpatialConvolution(1, m, 3,3,1,1,1,1) on weight[:, c] / bias[:, c]; n=3, m=4, 28x28, batch 3, within 1e-5.
    rng = np.random.default_rng(7)
    n, m = 3, 4
    x = rng.random((3, n, 28, 28)).astype(np.float32)
    w = rng.random((m, n, 3, 3)).astype(np.float32)
    b = rng.random((m, n)).astype(np.float32)
    y = host(F.dwconv_forward(dev(x), dev(w), dev(b), 1, 1, 1, 1))
    for c in range(n):
        yc = host(F.convmm_forward(dev(x[:, c:c + 1]), dev(w[:, c:c + 1]), dev(b[:, c]), 1, 1, 1, 1))
        assert np.max(np.abs(y[:, c * m:(c + 1) * m] - yc)) < 1e-5


def test_convmm_empty_batch_and_errors(F):
    from cunn_b200 import CunnError
    x = torch.empty((0, 4, 8, 8), device="cuda")
    w = torch.ones((8, 4, 3, 3), device="cuda")
    assert tuple(F.convmm_forward(x, w, None, 1, 1, 1, 1).shape) == (0, 8, 8, 8)
    with pytest.raises(CunnError, match="Output size is too small"):
        F.convmm_forward(torch.zeros((1, 4, 2, 2), device="cuda"), torch.zeros((8, 4, 5, 5), device="cuda"), None,
                         1, 1, 0, 0, out=torch.zeros(1, device="cuda"))


@pytest.mark.parametrize("cfg", [(128, 256, 256, 14, 3, 1), (128, 1024, 256, 14, 1, 0)])
def test_convmm_full_size_adjoint_identities(F, cfg):
    # The two benchmarked GEMM convolutions at full size (a size-independent property beside the whole-tensor
    # oracle comparison of test_full_size_gpu.py): the three passes are the three partial
    # derivatives of one trilinear form, so <conv(x, W), gy> == <x, dgrad(gy, W)> == <wgrad(x, gy), W>, and the
    # bias gradient is the plain sum of gy.  Inner products are taken in fp64; 1e-4 is the GEMM-path bar.
    N, C, K, HW, k, pad = cfg
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((N, C, HW, HW), device="cuda", generator=g)
    w = torch.randn((K, C, k, k), device="cuda", generator=g) * (2.0 / (C * k * k)) ** 0.5
    gy = torch.randn((N, K, HW, HW), device="cuda", generator=g)
    y = F.convmm_forward(x, w, None, 1, 1, pad, pad)
    gx = F.convmm_grad_input(gy, w, HW, HW, 1, 1, pad, pad)
    gw, gb = torch.zeros_like(w), torch.zeros(K, device="cuda")
    F.convmm_acc_grad(x, gy, gw, gb, 1, 1, pad, pad, 1.0)
    a = float((y.double() * gy.double()).sum())
    b = float((x.double() * gx.double()).sum())
    c = float((gw.double() * w.double()).sum())
    scale = float((y.double().abs() * gy.double().abs()).sum())
    assert abs(a - b) < 1e-6 * scale and abs(a - c) < 1e-6 * scale
    ref_gb = gy.double().sum((0, 2, 3))
    assert float((gb.double() - ref_gb).abs().max()) < 1e-4 * float(ref_gb.abs().max())
    # linearity in x at full size: conv(2 x1 - 3 x2) == 2 conv(x1) - 3 conv(x2)
    x2 = torch.randn((N, C, HW, HW), device="cuda", generator=g)
    lhs = F.convmm_forward(2 * x - 3 * x2, w, None, 1, 1, pad, pad)
    rhs = 2 * y - 3 * F.convmm_forward(x2, w, None, 1, 1, pad, pad)
    assert float((lhs - rhs).abs().max()) < 1e-4 * float(rhs.abs().max())


@pytest.mark.parametrize("shape", [
    # N, C, H, W, K, k, d, pad: weight gradients whose splits end inside an image, and kernels of more than 32 taps
    (3, 40, 37, 29, 70, 1, 1, 0),        # 1073-pixel planes: element copies, splits at odd pixels
    (2, 64, 60, 52, 130, 1, 1, 0),       # tensor maps: splits of whole pixel groups
    (1, 8, 90, 70, 24, 3, 1, 1),         # one image, gathered operand
    (1, 5, 64, 64, 16, 7, 2, 3),         # 49 taps
    (2, 3, 71, 53, 40, 11, 4, 2),        # 121 taps, stride 4
    (2, 6, 19, 23, 33, 9, 1, 4),         # 81 taps at stride 1: all three passes
    (1, 2, 40, 40, 70, 16, 3, 0),        # 256 taps: the largest kernel of this path
    (1, 2, 40, 40, 6, 17, 3, 0),         # one row more: the kernel for any size
    (1, 2, 20, 22, 5, 17, 1, 8),         # ... its three passes
    (1, 700, 1, 1, 40, 1, 1, 0),         # a single pixel
    (130, 100, 1, 1, 36, 1, 1, 0),       # fully connected: two row tiles, ragged reduction and columns
    (1, 32, 1, 1, 4, 1, 1, 0),           # ... one image, one k-block
    (5, 1024, 1, 1, 1000, 1, 1, 0),      # ... a classifier
    (5, 64, 1, 1, 6, 1, 1, 0),           # ... outputs whose rows are not 16-byte multiples
    (1, 512, 14, 14, 512, 1, 1, 0),      # few row tiles: column tiles of 32
    (1, 96, 14, 14, 200, 3, 1, 1),       # ... gathered operand
])
def test_convmm_split_reductions_and_large_kernels(F, ref64, shape):
    N, C, H, W, K, k, d, pad = shape
    case = make_case(abs(hash(shape)) % 99991, N, C, H, W, K, k, d, pad, True)
    check_against_oracle(ref64, F, *case, d, pad, 0.75)


@pytest.mark.parametrize("shape", [
    # N, C, H, K, k, d, pad: weight gradients split with rounding
    (2, 3, 16, 12, 7, 2, 3),             # 49 taps, 128 pixels
    (13, 3, 16, 18, 11, 4, 5),           # 121 taps
    (64, 136, 1, 184, 1, 1, 0),          # a fully connected layer
    (7, 60, 9, 33, 1, 1, 0),             # 567 pixels of unaligned planes
    (6, 3, 16, 112, 5, 4, 2),            # three k-blocks
    (5, 20, 13, 40, 3, 1, 1),            # 3x3
])
def test_weight_gradient_of_short_reductions(F, shape):
    import torch
    N, C, H, K, k, d, p = shape
    o = (H + 2 * p - k) // d + 1
    g = torch.Generator(device="cuda").manual_seed(8)
    x, gy = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(N, K, o, o, device="cuda", generator=g)
    cols = torch.nn.functional.unfold(x.double(), k, padding=p, stride=d)
    want = torch.einsum("nkp,ncp->kc", gy.double().view(N, K, -1), cols).view(K, C, k, k)
    gw, gb = torch.zeros(K, C, k, k, device="cuda"), torch.zeros(K, device="cuda")
    F.convmm_acc_grad(x, gy, gw, gb, d, d, p, p)
    # 2-norm: 0.76e-7 from parts of 11 rounded bits without lo * lo (normal values), and a chain's truncations of 2^-24 on average, at
    # most twelve of them at the size of the sum: 2.5e-7 holds both.  Truncated parts alone are 3.5e-7 off.
    assert float((gw.double() - want).norm() / want.norm()) <= 2.5e-7
    b = gy.double().sum((0, 2, 3))
    assert float((gb.double() - b).norm() / b.norm()) <= 2.0 ** -23        # a rounding or two of 32 bits


def test_weight_gradient_chains_stay_short(F):
    """37 images of 64 x 17 x 17 against 120 x 34 x 34, 4x4 stride 2: 335 k-blocks, split so that an accumulator takes no more of them
    than with whole images per tile."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(9)
    x, gy = torch.randn(37, 120, 34, 34, device="cuda", generator=g), torch.randn(37, 64, 17, 17, device="cuda", generator=g)
    cols = torch.nn.functional.unfold(x.double(), 4, padding=1, stride=2)
    want = torch.einsum("nkp,ncp->kc", gy.double().view(37, 64, -1), cols).view(64, 120, 4, 4)
    gw = torch.zeros(64, 120, 4, 4, device="cuda")
    F.convmm_acc_grad(x, gy, gw, None, 2, 2, 1, 1)
    # truncated operands 3.5e-7; an accumulator's n truncations of about 2^-24 / 1.4 at two thirds of the sum: 16 a tile of 10 or 19
    # k-blocks over three accumulators, n = 28 at most -> 8e-7 with half a factor for their growth; one of 38 has n = 52 -> 1.2e-6
    assert float((gw.double() - want).norm() / want.norm()) <= 1e-6


def test_fully_connected_gradient_of_2_24_outputs(F):
    """2^24 outputs: more than the filters of the convolution that stands in for the gradient of a fully connected layer may have taps."""
    import torch
    K, C = 1 << 24, 4
    gy, w = torch.zeros(1, K, 1, 1, device="cuda"), torch.zeros(K, C, 1, 1, device="cuda")
    at = torch.tensor([0, 5, 8191, K // 2 + 3, K - 1], device="cuda")
    gy[0, at, 0, 0] = torch.tensor([1.0, 2.0, -3.0, 4.0, 0.5], device="cuda")
    w[at] = torch.arange(20.0, device="cuda").view(5, 4, 1, 1)
    gx = F.convmm_grad_input(gy, w, 1, 1, 1, 1, 0, 0)
    assert torch.equal(gx.view(4), (gy[0, at, 0, 0].view(5, 1) * w[at].view(5, 4)).sum(0))


@pytest.mark.parametrize("shape", [(64, 8, 60), (3, 152, 4), (130, 64, 64), (64, 60, 8)])
def test_fully_connected_layers_of_one_or_two_k_blocks(F, shape):
    """Forward and input gradient keep the large products' accumulator apart from the small ones'."""
    import torch
    N, C, K = shape
    g = torch.Generator(device="cuda").manual_seed(10)
    x, w, gy = (torch.randn(*s, 1, 1, device="cuda", generator=g) for s in ((N, C), (K, C), (N, K)))
    y, gx = F.convmm_forward(x, w, None, 1, 1, 0, 0).view(N, K), F.convmm_grad_input(gy, w, 1, 1, 1, 1, 0, 0).view(N, C)
    xd, wd, gd = (t.double().flatten(1) for t in (x, w, gy))
    # truncated operands 3.5e-7; two chains of four and eight truncations, the longer one at 2^-10 of the sum: 2e-7
    for got, want in ((y, xd @ wd.t()), (gx, gd @ wd)):
        assert float((got.double() - want).norm() / want.norm()) <= 5.5e-7


@pytest.mark.parametrize("shape", [
    # N, C, K, H, W: clusters of four, two and eight CTAs a tile; reductions that do not divide by them; ragged tiles; two images in a tile
    (1, 512, 512, 14, 14), (1, 320, 40, 8, 8), (1, 332, 36, 5, 4), (2, 484, 100, 6, 6), (1, 768, 768, 14, 14), (1, 4096, 64, 4, 4), (1, 2052, 32, 1, 4),
    (3, 352, 200, 9, 4),
])
def test_pointwise_layers_of_few_tiles(shape):
    """Few tiles and long reductions: CTAs of a cluster share a tile.  Against fp64, with the bound of the truncating accumulation: products
    of 22 bits and chains of 12 additions a k-block of 32, at most KB k-blocks a CTA."""
    import torch
    from cunn_b200 import functional as F
    N, C, K, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(C + K)
    x, w = torch.randn(N, C, H, W, device="cuda", generator=g), torch.randn(K, C, 1, 1, device="cuda", generator=g)
    b, gy = torch.randn(K, device="cuda", generator=g), torch.randn(N, K, H, W, device="cuda", generator=g)
    wm = w.double().view(K, C)
    for what, got, a, t, bias in (("y", F.convmm_forward(x, w, b, 1, 1, 0, 0), wm, x, b), ("gx", F.convmm_grad_input(gy, w, H, W, 1, 1, 0, 0), wm.t(), gy, None)):
        want = torch.einsum("kc,nchw->nkhw", a, t.double())
        size = torch.einsum("kc,nchw->nkhw", a.abs(), t.double().abs())
        if bias is not None:
            want, size = want + bias.double().view(1, -1, 1, 1), size + bias.double().abs().view(1, -1, 1, 1)
        kb = -(-a.shape[1] // 32)
        assert bool(((got.double() - want).abs() <= (4 + 12 * kb) * 2.0 ** -23 * size).all()), what
        assert float((got.double() - want).norm() / want.norm()) <= 1e-6, what
    y = F.convmm_forward(x, w, b, 1, 1, 0, 0)
    assert torch.equal(y, F.convmm_forward(x, w, b, 1, 1, 0, 0))          # the same order of sums each time
    # infinities and NaN reach the outputs that read them and no others
    x[0, 1, 0, 0], x[-1, 0, -1, -1] = float("inf"), float("nan")
    bad = ~torch.isfinite(F.convmm_forward(x, w, b, 1, 1, 0, 0))
    hit = torch.zeros(N, 1, H, W, dtype=torch.bool, device="cuda")
    hit[0, 0, 0, 0] = hit[-1, 0, -1, -1] = True
    assert torch.equal(bad, hit.expand_as(bad))
