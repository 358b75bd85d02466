"""Input gradients of strided convolutions (and the forward pass of transposed ones) on the tensor-core kernel that takes them
apart into one GEMM per stride residue: sizes at which the phases, tiles and k-blocks end unevenly."""
import numpy as np
import pytest

from conftest import assert_parity, norm_err

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def F():
    from cunn_b200 import functional
    return functional


@pytest.mark.parametrize("shape", [
    # N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW
    (2, 128, 14, 14, 64, 3, 3, 2, 2, 1, 1, 1, 1),      # phases of 4, 2, 2 and 1 taps; one column tile of 128
    (3, 40, 15, 13, 24, 3, 3, 2, 2, 1, 1, 1, 1),       # odd map: phases of different sizes, ragged reduction and columns
    (1, 5, 9, 7, 3, 2, 2, 3, 3, 0, 0, 1, 1),           # kernel smaller than the stride: residues without taps
    (2, 70, 8, 8, 33, 1, 1, 2, 2, 0, 0, 1, 1),         # 1x1 stride 2: three of four phases are filled
    (2, 6, 30, 31, 10, 11, 11, 4, 4, 2, 2, 1, 1),      # sixteen phases of up to 3x3 taps
    (1, 3, 40, 37, 4, 5, 7, 5, 6, 3, 2, 1, 1),         # thirty phases: two launches
    (2, 8, 20, 20, 12, 3, 3, 2, 2, 2, 2, 2, 2),        # stride and dilation share a factor: only even residues have taps
    (2, 8, 21, 19, 12, 3, 3, 2, 3, 3, 3, 3, 2),        # stride and dilation without a common factor
    (2, 8, 6, 6, 12, 3, 3, 1, 1, 5, 5, 1, 1),          # stride 1, padding beyond the kernel
    (1, 4, 1, 3, 6, 3, 3, 2, 2, 1, 1, 1, 1),           # fewer rows than the stride
    (1, 5, 90, 70, 6, 1, 2, 40, 33, 0, 0, 1, 1),       # 1320 residues, two of them with taps
    (5, 130, 12, 12, 260, 3, 3, 2, 1, 1, 1, 1, 1),     # strides differ; two column tiles, 25 k-blocks
])
def test_strided_input_gradient(F, ref64, ref32, shape):
    N, C, H, W, K, kH, kW, dH, dW, pH, pW, dilH, dilW = shape
    rng = np.random.default_rng(abs(hash(shape)) % 99991)
    oH, oW = (H + 2 * pH - dilH * (kH - 1) - 1) // dH + 1, (W + 2 * pW - dilW * (kW - 1) - 1) // dW + 1
    gy, w = rng.standard_normal((N, K, oH, oW)).astype(np.float32), rng.uniform(-1, 1, (K, C, kH, kW)).astype(np.float32)
    want = ref64.dilconv_grad_input(gy, w, H, W, dH, dW, pH, pW, dilH, dilW)
    got = F.dilated_conv_grad_input(dev(gy), dev(w), H, W, dH, dW, pH, pW, dilH, dilW).cpu().numpy()
    port = ref32.dilconv_grad_input(gy, w, H, W, dH, dW, pH, pW, dilH, dilW)
    assert_parity("strided gx", got, want, 1e-4, port=port)
    # a k-block's chain truncates four times at the size of its sum (2^-23 each), the k-blocks are added with rounding (2^-24 each, at
    # most 56 of them), the split drops 2^-21 of a product: 4e-6 of the largest value holds all of it
    assert norm_err(got, want) <= 4e-6
    if dilH == dilW == 1:
        b = rng.uniform(-1, 1, C).astype(np.float32)
        adj = (H - ((oH - 1) * dH - 2 * pH + kH), W - ((oW - 1) * dW - 2 * pW + kW))
        y = F.full_conv_forward(dev(gy), dev(w), dev(b), dH, dW, pH, pW, 1, 1, *adj).cpu().numpy()
        bias = b[None, :, None, None]
        assert_parity("transposed y", y, want + bias, 1e-4, port=port + bias)
        assert norm_err(y, want + bias) <= 4e-6


def test_strided_input_gradient_not_finite(F):
    """Infinities and NaN reach exactly the pixels whose taps read them, with the sign that fp32 arithmetic gives."""
    import torch
    N, C, H, W, K = 1, 5, 11, 11, 7
    gy, w = torch.ones(N, K, 6, 6, device="cuda"), torch.full((K, C, 3, 3), 0.5, device="cuda")
    gy[0, 3, 2, 2] = float("inf")
    gy[0, 1, 4, 5] = float("nan")
    gx = F.convmm_grad_input(gy, w, H, W, 2, 2, 1, 1)
    want = torch.nn.functional.conv_transpose2d(gy.cpu().double(), w.cpu().double(), None, 2, 1)
    assert torch.equal(gx.cpu().double(), want) or torch.allclose(gx.cpu().double(), want, rtol=1e-6, equal_nan=True)


@pytest.mark.parametrize("shape", [
    # N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW: long kernels of up to 32 taps, all passes
    (2, 3, 5, 60, 7, 1, 32, 1, 1, 0, 5, 1, 1),         # a row of 32 taps
    (2, 3, 90, 4, 7, 32, 1, 1, 2, 3, 0, 2, 1),         # a dilated column of them, strided across
    (1, 4, 20, 80, 6, 1, 20, 2, 1, 0, 9, 1, 3),        # a dilated row, more than sixteen columns
])
def test_long_kernels(F, ref64, shape):
    N, C, H, W, K, kH, kW, dH, dW, pH, pW, dilH, dilW = shape
    rng = np.random.default_rng(abs(hash(shape)) % 99991)
    oH, oW = (H + 2 * pH - dilH * (kH - 1) - 1) // dH + 1, (W + 2 * pW - dilW * (kW - 1) - 1) // dW + 1
    x, gy = rng.standard_normal((N, C, H, W)).astype(np.float32), rng.standard_normal((N, K, oH, oW)).astype(np.float32)
    w, b = rng.uniform(-1, 1, (K, C, kH, kW)).astype(np.float32), rng.uniform(-1, 1, K).astype(np.float32)
    geo = (dH, dW, pH, pW, dilH, dilW)
    # the split drops up to 2^-20 of a product and the tensor core truncates its sums: 1e-5 of the largest value, as for the other kernels
    y = F.dilated_conv_forward(dev(x), dev(w), dev(b), *geo).cpu().numpy()
    assert norm_err(y, ref64.dilconv_forward(x, w, b, *geo)) <= 1e-5
    gx = F.dilated_conv_grad_input(dev(gy), dev(w), H, W, *geo).cpu().numpy()
    assert norm_err(gx, ref64.dilconv_grad_input(gy, w, H, W, *geo)) <= 1e-5
    gw, gb = np.zeros_like(w), np.zeros(K, np.float32)
    dgw, dgb = dev(gw), dev(gb)
    F.dilated_conv_acc_grad(dev(x), dev(gy), dgw, dgb, *geo, 0.75)
    want = ref64.dilconv_acc_grad(x, gy, gw.copy(), gb.copy(), *geo, 0.75)
    assert norm_err(dgw.cpu().numpy(), want[0]) <= 1e-5
    assert norm_err(dgb.cpu().numpy(), want[1]) <= 1e-5


NANS = [0x7fffffff, -1, 0x7fc00000, 0x7f800001]      # what CUDA arithmetic makes of inf - inf, its negative, the host's NaN, the smallest one


def with_bits(t, index, bits):
    import torch
    t = t.clone()
    t.view(torch.int32)[index] = bits
    return t


@pytest.mark.parametrize("bits", NANS)
@pytest.mark.parametrize("where", ["gy", "w"])
def test_strided_gradient_keeps_every_nan(F, where, bits):
    """A NaN of any bit pattern reaches the strided input gradient and the transposed forward pass, at the pixels that read it."""
    import torch
    rng = torch.Generator(device="cuda").manual_seed(3)
    gy, w = (torch.randn(*s, device="cuda", generator=rng) for s in ((2, 64, 7, 7), (64, 5, 3, 3)))
    if where == "gy":
        gy = with_bits(gy, (1, 40, 2, 3), bits)
    else:
        w = with_bits(w, (17, 2, 2, 1), bits)
    b = torch.randn(5, device="cuda", generator=rng)
    want = torch.nn.functional.conv_transpose2d(gy.cpu().double(), w.cpu().double(), None, 2, 1)
    assert int(torch.isnan(want).sum()) > 0 and not torch.isnan(want).all()
    gx = F.convmm_grad_input(gy, w, 13, 13, 2, 2, 1, 1).cpu().double()
    assert torch.equal(torch.isnan(gx), torch.isnan(want)) and torch.allclose(gx, want, rtol=1e-4, atol=1e-4, equal_nan=True)
    y = F.full_conv_forward(gy, w, b, 2, 2, 1, 1).cpu()
    assert torch.equal(torch.isnan(y), torch.isnan(want))


@pytest.mark.parametrize("bits", NANS + [0x7f800000])
@pytest.mark.parametrize("where", ["x", "w"])
def test_large_kernel_keeps_what_is_not_finite(F, where, bits):
    """7x7 forward and stride-1 input gradient: a sum that reads a NaN or an infinity is not finite, every other one is."""
    import torch
    rng = torch.Generator(device="cuda").manual_seed(4)
    x, w = (torch.randn(*s, device="cuda", generator=rng) for s in ((2, 3, 20, 21), (6, 3, 7, 7)))
    if where == "x":
        x = with_bits(x, (1, 2, 9, 8), bits)
    else:
        w = with_bits(w, (4, 1, 3, 6), bits)
    want = torch.nn.functional.conv2d(x.cpu().double(), w.cpu().double())
    y = F.convmm_forward(x, w, None, 1, 1, 0, 0).cpu()
    assert torch.equal(torch.isfinite(y), torch.isfinite(want)) and not torch.isfinite(y).all()
    # the same kernel's gradient with every output pixel's taps inside the map: no product that the definition lacks
    gy = torch.ones(2, 6, 14, 15, device="cuda")
    if where == "w":
        want = torch.nn.functional.conv_transpose2d(gy.cpu().double(), w.cpu().double())
        gx = F.convmm_grad_input(gy, w, 20, 21, 1, 1, 0, 0).cpu().double()
        assert torch.allclose(gx, want, rtol=1e-4, atol=1e-4, equal_nan=True)


def test_largest_finite_values_stay_finite(F):
    """Rounding the high part of a value next to the largest float must not make it infinite, in either pass."""
    import torch
    big = torch.finfo(torch.float32).max
    x, w = torch.zeros(1, 1, 12, 12, device="cuda"), torch.zeros(1, 1, 7, 7, device="cuda")
    x[0, 0, 5, 6], w[0, 0, 2, 3] = big, 0.5
    y = F.convmm_forward(x, w, None, 1, 1, 3, 3)
    assert y[0, 0, 6, 6].item() == pytest.approx(0.5 * big, rel=2 ** -20) and int((y != 0).sum()) == 1
    gx = F.convmm_grad_input(x, w, 24, 24, 2, 2, 3, 3)
    assert gx[0, 0, 9, 12].item() == pytest.approx(0.5 * big, rel=2 ** -20) and int((gx != 0).sum()) == 1


def test_diverged_gradient_of_a_long_reduction(F):
    """Every sum of a reduction of 73,728 products is infinite or NaN: all are taken again in fp32, outside any wait that has a limit."""
    import torch
    from cunn_b200 import device_status
    K, C, k = 2048, 33, 12
    gy = torch.full((1, K, 3, 3), float("inf"), device="cuda")
    w = torch.rand(K, C, k, k, device="cuda") + 0.5
    w[5, 7, 3, 4] = -1.0                                  # inf - inf for the pixels that read it
    gx = F.convmm_grad_input(gy, w, 16, 16, 2, 2, 0, 0)
    want = torch.full((1, C, 16, 16), float("inf"), device="cuda")
    want[0, 7, 3:9:2, 4:10:2] = float("nan")
    assert torch.allclose(gx, want, equal_nan=True) and device_status() == 0


@pytest.mark.parametrize("shape", [
    # N, C, H, W, K, k, d, pad: reductions and residues that the tensor-core kernel does not take
    (1, 1, 16, 16, 65540, 16, 1, 0),     # 256 taps of 65,540 filters: an index that cannot be divided by multiplication
    (2, 5, 40, 37, 6, 35, 2, 3),         # residues of 18 and 17 rows of taps
    (1, 9, 21, 19, 3, 17, 1, 17),        # stride 1, padding of the kernel size
    (2, 2, 300, 290, 4, 150, 130, 40),   # more residues than one launch lists, two rows of taps in some
    (2, 3, 64, 64, 50, 64, 64, 0),       # a residue per tap, two pixels each, on the fp32 side of the rule
    (3, 61, 196, 196, 90, 14, 14, 0),    # ... and on the tensor cores' side
])
def test_residues_in_fp32(F, shape):
    import torch
    N, C, H, W, K, k, d, p = shape
    oH, oW = (H + 2 * p - k) // d + 1, (W + 2 * p - k) // d + 1
    g = torch.Generator().manual_seed(6)
    gy, w, b = torch.randn(N, K, oH, oW, generator=g), torch.rand(K, C, k, k, generator=g) * 2 - 1, torch.rand(C, generator=g)
    adj = (H - ((oH - 1) * d - 2 * p + k), W - ((oW - 1) * d - 2 * p + k))
    want = torch.zeros(N, C, H + 2 * p + k, W + 2 * p + k, dtype=torch.double)
    for kh in range(k):
        for kw in range(k):
            want[:, :, kh:kh + (oH - 1) * d + 1:d, kw:kw + (oW - 1) * d + 1:d] += torch.einsum("nkhw,kc->nchw", gy.double(), w[:, :, kh, kw].double())
    want = want[:, :, p:p + H, p:p + W]
    gx = F.convmm_grad_input(dev(gy.numpy()), dev(w.numpy()), H, W, d, d, p, p).cpu().double()
    # a chain of n fp32 additions of products: n 2^-24 of the sum of magnitudes at most; sqrt(n) 2^-24 of the largest value is met in practice
    n = K * (-(-k // d)) ** 2
    assert norm_err(gx.numpy(), want.numpy()) <= 4 * n ** 0.5 * 2.0 ** -24 + 2e-7
    y = F.full_conv_forward(dev(gy.numpy()), dev(w.numpy()), dev(b.numpy()), d, d, p, p, 1, 1, *adj).cpu()
    assert torch.equal(y, (gx.float() + b.view(1, -1, 1, 1)))


@pytest.mark.parametrize("shape", [
    # N, C, K, H, k, d, pad: sums of 1 to 47 products (fp32), of 48 and more (tensor cores), and calls that have both
    (2, 9, 1, 13, 1, 2, 0), (2, 6, 47, 12, 1, 2, 0), (2, 6, 48, 12, 1, 2, 0), (1, 7, 5, 11, 1, 70, 0), (2, 35, 11, 14, 4, 2, 1), (2, 35, 12, 14, 4, 2, 1),
    (1, 40, 23, 15, 3, 2, 1), (1, 40, 24, 15, 3, 2, 1), (2, 33, 46, 15, 3, 2, 1), (4, 64, 16, 28, 3, 2, 1),
])
def test_short_sums_lose_no_bits(F, shape):
    """2-norm of the error of strided input gradients against that of a chain of fp32 FMAs, one product after the other."""
    import torch
    N, C, K, H, k, d, p = shape
    o = (H + 2 * p - k) // d + 1
    g = torch.Generator(device="cuda").manual_seed(K)
    gy, w = torch.randn(N, K, o, o, device="cuda", generator=g), torch.rand(K, C, k, k, device="cuda", generator=g) * 2 - 1
    span = (o - 1) * d + k
    # fma(a, b, c) by rounding the exact 64-bit product and sum: 24 + 24 bits fit, the sum rounds once more at 53
    chain = torch.zeros(N, C, max(span, H + 2 * p), max(span, H + 2 * p), device="cuda")
    exact = chain.double()
    for kh in range(k):
        for kw in range(k):
            at = (slice(None), slice(None), slice(kh, kh + (o - 1) * d + 1, d), slice(kw, kw + (o - 1) * d + 1, d))
            for i in range(K):
                term = gy[:, i:i + 1].double() * w[i, :, kh, kw].double().view(1, C, 1, 1)
                exact[at] += term
                chain[at] = (chain[at].double() + term).float()
    exact, chain = exact[:, :, p:p + H, p:p + H], chain[:, :, p:p + H, p:p + H]
    gx = F.convmm_grad_input(gy, w, H, H, d, d, p, p)
    err = lambda t: float((t.double() - exact).norm() / exact.norm())
    if K * (-(-k // d)) ** 2 < 48:
        assert torch.equal(gx, chain)
    # above the limit the tensor cores' error is the smaller one on average; a tenth covers the scatter of one draw
    assert err(gx) <= 1.1 * err(chain)


@pytest.mark.parametrize("shape", [
    # N, C, K, H, k, d, pad: sums of 64 to 9216 products on the tensor cores
    (2, 40, 64, 26, 1, 2, 0), (4, 128, 256, 28, 3, 2, 1), (1, 96, 1024, 15, 3, 2, 1), (1, 40, 1024, 14, 6, 2, 2), (8, 128, 256, 28, 4, 2, 1),
])
def test_long_sums_do_not_drift(F, shape):
    import torch
    N, C, K, H, k, d, p = shape
    o = (H + 2 * p - k) // d + 1
    g = torch.Generator(device="cuda").manual_seed(11)
    gy, w = torch.randn(N, K, o, o, device="cuda", generator=g), torch.rand(K, C, k, k, device="cuda", generator=g) * 2 - 1
    want = torch.nn.grad.conv2d_input((N, C, H, H), w.double(), gy.double(), d, p)
    gx = F.convmm_grad_input(gy, w, H, H, d, d, p, p)
    # 2-norm: 0.8e-7 from parts of 11 rounded bits without lo * lo and 1e-7 from a k-block's truncations at the size of its own sum, which do
    # not grow with the blocks' number b; its additions round a growing sum, 2^-24 / sqrt(12) of sqrt(i / b) each: 1.8e-8 sqrt(b / 2)
    blocks = -(-K * (-(-k // d)) ** 2 // 32)
    assert float((gx.double() - want).norm() / want.norm()) <= 1.7e-7 + 1.8e-8 * (blocks / 2) ** 0.5
