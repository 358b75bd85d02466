"""Convolutions on operands that are split once (conv_split.cu): all passes at the edges of tiles, blocks, groups and residues, the range of
their exponents, what is not finite, and calls whose scratch memory is too small."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import cunn_b200.functional as F
    from cunn_b200 import device_status
    yield F
    assert device_status() == 0


def out_size(size, k, d, p, dil):
    return (size + 2 * p - dil * (k - 1) - 1) // d + 1


def scratch(which, N, C, H, W, K, kH, kW, d, p, dil):
    from cunn_b200._lib import lib
    return lib.cunn_b200_conv_scratch(which, N, C, H, W, K, kH, kW, d, d, p, p, dil, dil)


def off(got, want):
    return float((got.double() - want).norm() / want.norm())


def bound(products, group=64):
    # 2-norm: 0.8e-7 from parts of 11 rounded bits without lo * lo; a block's chain truncates four times at up to the size of its own
    # sum, 2^-24 on average; its additions to fp32 registers round a growing sum, 1.8e-8 sqrt(b / 2) for b blocks
    return 0.8e-7 + 4 * 2.0 ** -24 + 1.8e-8 * (products / group / 2) ** 0.5


SHAPES = [
    # N, C, H, W, K, kH, kW, stride, pad, dilation, passes: forward, input gradient, parameter gradient
    (4, 144, 15, 15, 72, 5, 5, 1, 2, 1, "fg"),        # partial tiles and groups
    (3, 96, 17, 13, 200, 3, 3, 2, 1, 1, "fg"),       # two residues of odd sizes; 200 columns of a tile of 256
    (8, 130, 19, 23, 150, 3, 3, 2, 1, 1, "fg"),       # channels that are no multiple of eight
    (24, 130, 29, 23, 150, 3, 3, 1, 1, 1, "fgw"),     # ... and a part of a row tile
    (16, 64, 31, 29, 65, 3, 3, 1, 2, 2, "fg"),        # dilation; one column past a tile half
    (2, 256, 14, 14, 256, 3, 3, 1, 1, 1, "fg"),       # few tiles, cut into many parts
    (33, 130, 28, 28, 150, 2, 2, 2, 0, 1, "g"),       # one tap per residue
    (20, 37, 40, 40, 320, 4, 4, 2, 1, 1, "fgw"),      # two column tiles; a group of 37 channels
    (64, 128, 28, 28, 256, 3, 3, 1, 1, 1, "fgw"),     # whole tiles and cut ones
    (9, 80, 33, 35, 64, 3, 5, 1, 1, 1, "fgw"),        # a kernel that is not square
    (3, 176, 12, 50, 96, 1, 7, 1, 3, 1, "fg"),        # one row of taps, padding beyond it
    (40, 256, 14, 14, 100, 7, 7, 1, 3, 1, "fgw"),     # 49 taps
    (128, 1024, 7, 7, 512, 1, 1, 1, 0, 1, "fgw"),     # 1x1 on planes of an odd size
    (40, 512, 15, 15, 500, 1, 1, 1, 0, 1, "fg"),      # ... two column tiles, the second one ragged
    (32, 3, 150, 141, 48, 7, 7, 2, 3, 1, "fw"),       # few channels: row windows of 21 values, an odd map
    (64, 12, 60, 60, 64, 5, 5, 1, 2, 1, "fw"),        # ... of 60
    (20, 3, 150, 161, 40, 11, 11, 4, 5, 1, "f"),      # ... of 33, parts of a row tile
    (30, 3, 150, 161, 40, 11, 11, 2, 5, 1, "w"),      # ... in groups of 64 columns
    (9, 5, 90, 97, 130, 3, 3, 1, 1, 1, "f"),          # ... and two columns past a tile
    (12, 3, 40, 700, 64, 5, 5, 1, 2, 1, "f"),         # ... rows that share a block in twos
]


@pytest.mark.parametrize("shape", SHAPES)
def test_all_passes(F, shape):
    N, C, H, W, K, kH, kW, d, p, dil, passes = shape
    oH, oW = out_size(H, kH, d, p, dil), out_size(W, kW, d, p, dil)
    g = torch.Generator(device="cuda").manual_seed(20)
    x, gy = (torch.randn(*s, device="cuda", generator=g) for s in ((N, C, H, W), (N, K, oH, oW)))
    w, b = torch.rand(K, C, kH, kW, device="cuda", generator=g) * 2 - 1, torch.randn(K, device="cuda", generator=g)
    X, V, G = x.double(), w.double(), gy.double()
    geo = (d, d, p, p, dil, dil)
    assert all(scratch("fgw".index(n), N, C, H, W, K, kH, kW, d, p, dil) for n in passes)
    if "f" in passes:
        y = F.dilated_conv_forward(x, w, b, *geo)
        assert off(y, torch.nn.functional.conv2d(X, V, b.double(), d, p, dil)) <= bound(C * kH * kW)
    if "g" in passes:
        gx = F.dilated_conv_grad_input(gy, w, H, W, *geo, out=torch.full_like(x, 7.0))
        assert off(gx, torch.nn.grad.conv2d_input(X.shape, V, G, d, p, dil)) <= bound(K * kH * kW)
        if dil == 1 and kH == kW:
            adj = [s - ((o - 1) * d - 2 * p + kH) for s, o in ((H, oH), (W, oW))]
            q = torch.randn(C, device="cuda", generator=g)
            t = F.full_conv_forward(gy, w, q, d, d, p, p, 1, 1, *adj)
            assert torch.equal(t, gx + q.view(1, -1, 1, 1))
    if "w" in passes:
        gw, gb = torch.ones_like(w), torch.ones_like(b)
        F.dilated_conv_acc_grad(x, gy, gw, gb, *geo, 0.5)
        want = torch.nn.grad.conv2d_weight(X, V.shape, G, d, p, dil)
        assert off((gw.double() - 1) * 2, want) <= bound(N * oH * oW) + 2.0 ** -24 * 2 * (want.numel() ** 0.5) / float(want.norm())
        sums = G.sum((0, 2, 3))
        assert off((gb.double() - 1) * 2, sums) <= 2.0 ** -22
        again, gb2 = torch.ones_like(w), torch.ones_like(b)
        F.dilated_conv_acc_grad(x, gy, again, gb2, *geo, 0.5)
        assert torch.equal(again, gw) and torch.equal(gb2, gb)


@pytest.mark.parametrize("stride", [1, 2])
def test_exponents_of_any_range(F, stride):
    """Images of sizes 1e-26 to 1e26 against filters of 1e-8 to 1e8: every plane is as exact as if it were alone."""
    N, C, K, H = 40, 96, 72, 28
    o = out_size(H, 3, stride, 1, 1)
    g = torch.Generator(device="cuda").manual_seed(21)
    x, gy = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(N, K, o, o, device="cuda", generator=g)
    w = torch.rand(K, C, 3, 3, device="cuda", generator=g) * 2 - 1
    images = 10.0 ** torch.linspace(-26, 26, N, device="cuda").view(-1, 1, 1, 1)
    rows, cols = 10.0 ** torch.linspace(-8, 8, K, device="cuda").view(-1, 1, 1, 1), 10.0 ** torch.linspace(-8, 8, C, device="cuda").view(1, -1, 1, 1)
    assert scratch(0, N, C, H, H, K, 3, 3, stride, 1, 1) and scratch(1, N, C, H, H, K, 3, 3, stride, 1, 1)

    def planes_off(got, want):
        d = (got.double() - want).flatten(2).norm(dim=2) / want.flatten(2).norm(dim=2)
        return float(d.max())

    y = F.convmm_forward(x * images, w * rows, None, stride, stride, 1, 1)
    want = torch.nn.functional.conv2d((x * images).double(), (w * rows).double(), None, stride, 1)
    assert planes_off(y, want) <= 3 * bound(C * 9)              # a plane's norm scatters more than the tensor's
    gx = F.convmm_grad_input(gy * images, w * cols, H, H, stride, stride, 1, 1)
    want = torch.nn.grad.conv2d_input(x.shape, (w * cols).double(), (gy * images).double(), stride, 1)
    assert planes_off(gx, want) <= 3 * bound(K * 9)


def test_parameter_gradient_of_any_range(F):
    """Channels of sizes 1e-15 to 1e15 on both sides."""
    N, C, K, H = 32, 96, 72, 28
    g = torch.Generator(device="cuda").manual_seed(22)
    x, gy = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(N, K, H, H, device="cuda", generator=g)
    x *= 10.0 ** torch.linspace(-15, 15, C, device="cuda").view(1, -1, 1, 1)
    gy *= 10.0 ** torch.linspace(-15, 15, K, device="cuda").view(1, -1, 1, 1)
    assert scratch(2, N, C, H, H, K, 3, 3, 1, 1, 1)
    gw, gb = torch.zeros(K, C, 3, 3, device="cuda"), torch.zeros(K, device="cuda")
    F.convmm_acc_grad(x, gy, gw, gb, 1, 1, 1, 1)
    want = torch.nn.grad.conv2d_weight(x.double(), gw.shape, gy.double(), 1, 1)
    d = (gw.double() - want).flatten(2).norm(dim=2) / want.flatten(2).norm(dim=2)
    # nine sums each: the error of a sum of random signs against its own size
    assert float(d.median()) <= 2 * bound(N * H * H) and float(d.max()) <= 40 * bound(N * H * H)


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where", ["x", "w"])
def test_what_is_not_finite(F, where, value):
    """A sum that reads it is not finite, every other one is what it was; a strided input gradient has the sign of its infinities."""
    N, C, K, H = 96, 64, 64, 28
    assert scratch(0, N, C, H, H, K, 3, 3, 1, 1, 1) and scratch(1, N, C, H, H, K, 3, 3, 2, 1, 1)
    g = torch.Generator(device="cuda").manual_seed(23)
    x, gy = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(N, K, 14, 14, device="cuda", generator=g)
    w = torch.rand(K, C, 3, 3, device="cuda", generator=g) + 0.5
    if where == "x":
        x[3, 5, 7, 9] = gy[2, 6, 13, 0] = value
    else:
        w[9, 5, 2, 1] = value
    want = torch.nn.functional.conv2d(x.double(), w.double(), None, 1, 1)
    y = F.convmm_forward(x, w, None, 1, 1, 1, 1)
    ok = torch.isfinite(want) if where == "x" else torch.isfinite(want).all((0, 2, 3)).view(1, -1, 1, 1).expand_as(want)
    assert torch.isfinite(y[ok]).all() and not torch.isfinite(y[~torch.isfinite(want)]).any()
    assert off(y[ok], want[ok]) <= 2 * bound(C * 9)
    want = torch.nn.grad.conv2d_input(x.shape, w.double(), gy.double(), 2, 1)
    gx = F.convmm_grad_input(gy, w, H, H, 2, 2, 1, 1).double()
    assert not torch.isfinite(want).all() and torch.allclose(gx, want, rtol=1e-4, atol=1e-4, equal_nan=True)
    if where == "x":
        x, gy = (torch.randn(32, 128, H, H, device="cuda", generator=g) for _ in range(2))
        assert scratch(2, 32, 128, H, H, 128, 3, 3, 1, 1, 1)
        x[3, 5, 7, 9] = gy[2, 6, 13, 0] = value
        gw = torch.zeros(128, 128, 3, 3, device="cuda")
        F.convmm_acc_grad(x, gy, gw, None, 1, 1, 1, 1)
        read = torch.zeros(128, 128, 3, 3, dtype=torch.bool, device="cuda")
        read[6], read[:, 5] = True, True                 # the filter and the channel whose sums read a value that is not finite
        assert torch.isfinite(gw[~read]).all()
        assert not torch.isfinite(gw[6, :, :, 0:2]).any() and not torch.isfinite(gw[:, 5]).any()


def test_largest_values_stay_finite(F):
    big = torch.finfo(torch.float32).max
    x, w = torch.zeros(16, 64, 28, 28, device="cuda"), torch.zeros(64, 64, 3, 3, device="cuda")
    x[3, 5, 6, 7], w[11, 5, 1, 1] = big, 0.5
    assert scratch(0, 16, 64, 28, 28, 64, 3, 3, 1, 1, 1) and scratch(1, 16, 64, 28, 28, 64, 3, 3, 1, 1, 1)
    y, gx = F.convmm_forward(x, w, None, 1, 1, 1, 1), F.convmm_grad_input(x, w.transpose(0, 1).contiguous(), 28, 28, 1, 1, 1, 1)
    for t in (y, gx):
        assert t[3, 11, 6, 7].item() == pytest.approx(0.5 * big, rel=2 ** -20) and int((t != 0).sum()) == 1
    # many large products whose sum is a float
    x, w = torch.full((16, 64, 28, 28), 1e37, device="cuda"), torch.full((64, 64, 3, 3), 1e-2, device="cuda")
    y = F.convmm_forward(x, w, None, 1, 1, 0, 0)
    assert torch.allclose(y, torch.full_like(y, 64 * 9 * 1e35), rtol=1e-5)


def test_without_enough_scratch(F):
    """Less scratch than the pass takes, or none: the result of the kernels without it, to the bit."""
    from cunn_b200._lib import lib, check
    N, C, H, K = 8, 64, 28, 96
    g = torch.Generator(device="cuda").manual_seed(24)
    x, w = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(K, C, 3, 3, device="cuda", generator=g)
    geo = (N, C, H, H, K, 3, 3, 1, 1, 1, 1)
    need = lib.cunn_b200_conv_scratch(0, *geo, 1, 1)
    y0, y1, y2 = (torch.empty(N, K, H, H, device="cuda") for _ in range(3))
    ws, stream = torch.empty(need, dtype=torch.uint8, device="cuda"), torch.cuda.current_stream().cuda_stream
    check(lib.cunn_b200_convmm_forward(x.data_ptr(), w.data_ptr(), None, y0.data_ptr(), *geo, stream))
    check(lib.cunn_b200_conv_forward_scratch(x.data_ptr(), w.data_ptr(), None, y1.data_ptr(), *geo, 1, 1, ws.data_ptr(), need - 1, stream))
    check(lib.cunn_b200_conv_forward_scratch(x.data_ptr(), w.data_ptr(), None, y2.data_ptr(), *geo, 1, 1, None, 0, stream))
    assert torch.equal(y0, y1) and torch.equal(y0, y2)
    check(lib.cunn_b200_conv_forward_scratch(x.data_ptr(), w.data_ptr(), None, y1.data_ptr(), *geo, 1, 1, ws.data_ptr(), need, stream))
    assert not torch.equal(y0, y1) and off(y1, y0.double()) <= 2e-6


def test_capture_and_streams(F):
    """A graph keeps its own scratch: eager calls between its replays, and a second graph, do not touch it."""
    N, C, H, K = 8, 64, 28, 96
    g = torch.Generator(device="cuda").manual_seed(25)
    x, w = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(K, C, 3, 3, device="cuda", generator=g)
    want = F.convmm_forward(x, w, None, 1, 1, 1, 1)
    graphs, outs = [], []
    for scale in (1.0, 2.0):
        xs = x * scale
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs.append(F.convmm_forward(xs, w, None, 1, 1, 1, 1))
        graphs.append((graph, xs))
    streams = [torch.cuda.Stream() for _ in graphs]
    for _ in range(10):
        for (graph, _), s in zip(graphs, streams):
            with torch.cuda.stream(s):
                graph.replay()
        F.convmm_forward(x * 3, w, None, 1, 1, 1, 1)
    torch.cuda.synchronize()
    assert torch.equal(outs[0], want) and torch.equal(outs[1], want * 2)


def test_thnn_layer(F):
    """The THNN entry points take the same kernels, with scratch of their own."""
    from cunn_b200 import thnn
    N, C, H, K = 32, 128, 28, 128
    g = torch.Generator(device="cuda").manual_seed(26)
    x, gy = (torch.randn(N, C, H, H, device="cuda", generator=g) for _ in range(2))
    w, b = torch.randn(K, C, 3, 3, device="cuda", generator=g), torch.randn(K, device="cuda", generator=g)
    assert all(scratch(which, N, C, H, H, K, 3, 3, 1, 1, 1) for which in range(3))
    nnb = thnn.THNN()
    for _ in range(2):
        assert torch.equal(nnb.SpatialConvolutionMM_updateOutput(x, w.view(K, -1), b, 3, 3, 1, 1, 1, 1), F.convmm_forward(x, w, b, 1, 1, 1, 1))
        assert torch.equal(nnb.SpatialConvolutionMM_updateGradInput(x, gy, w.view(K, -1), 3, 3, 1, 1, 1, 1), F.convmm_grad_input(gy, w, H, H, 1, 1, 1, 1))
        got, want = [torch.zeros_like(w), torch.zeros_like(b)], [torch.zeros_like(w), torch.zeros_like(b)]
        nnb.SpatialConvolutionMM_accGradParameters(x, gy, got[0].view(K, -1), got[1], 3, 3, 1, 1, 1, 1, 0.5)
        F.convmm_acc_grad(x, gy, *want, 1, 1, 1, 1, 0.5)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    nnb.close()


# ---- values of very different sizes that share an exponent ------------------------------------------------------------------------
def wide_cases():
    """(name, shape, what is scaled): a group with one large value whose partner is zero, so that it adds nothing to any sum."""
    layer, strided = (32, 128, 28, 28, 128, 3, 3, 1, 1, 1), (20, 37, 40, 40, 320, 4, 4, 2, 1, 1)
    first, point = (32, 3, 150, 141, 48, 7, 7, 2, 3, 1), (64, 512, 15, 15, 256, 1, 1, 1, 0, 1)
    return [(what, shape) for shape in (layer, strided, first, point) for what in ("channel", "channels", "pixel", "weight")]


def gather_bound(products):
    """The gathering kernels' own error: operands of 22 bits without lo * lo 1.2e-7, chains that truncate at the size of the sum so far,
    2^-24 an addition and 1.8e-8 sqrt(n) for what they round."""
    return 1.2e-7 + 2.0 ** -24 * 40 + 1.8e-8 * products ** 0.5


@pytest.mark.parametrize("size", [1e5, 1e6, 1e9, 1e13, 1e25])
@pytest.mark.parametrize("what,shape", wide_cases())
def test_large_values_opposite_zeros(F, what, shape, size):
    """A channel, most channels, a pixel or a weight that is `size` times what shares its exponent, and adds nothing: the other values keep their bits."""
    N, C, H, W, K, kH, kW, d, p, dil = shape
    oH, oW = out_size(H, kH, d, p, dil), out_size(W, kW, d, p, dil)
    g = torch.Generator(device="cuda").manual_seed(30)
    x, gy = (torch.randn(*s, device="cuda", generator=g) for s in ((N, C, H, W), (N, K, oH, oW)))
    w = torch.rand(K, C, kH, kW, device="cuda", generator=g) * 2 - 1
    geo = (d, d, p, p, dil, dil)
    takes = [scratch(i, N, C, H, W, K, kH, kW, d, p, dil) for i in range(3)]
    assert any(takes)
    if takes[0]:
        xf, wf = x.clone(), w.clone()
        if what in ("channel", "channels"):
            n = slice(1, 2) if what == "channel" else slice(0, C * 4 // 5)
            xf[:, n] *= size
            wf[:, n] = 0
        elif what == "pixel":
            xf[3, 1, H // 2, W // 2] = size
            wf[:, 1] = 0
        else:
            wf[5, 1, kH // 2, 0] = size
            xf[:, 1] = 0
        want = torch.nn.functional.conv2d(xf.double(), wf.double(), None, d, p, dil)
        assert off(F.dilated_conv_forward(xf, wf, None, *geo), want) <= gather_bound(C * kH * kW)
    if takes[1]:
        gf, wf = gy.clone(), w.clone()
        if what in ("channel", "channels"):
            n = slice(1, 2) if what == "channel" else slice(0, K * 4 // 5)
            gf[:, n] *= size
            wf[n] = 0
        elif what == "pixel":
            gf[3, 1, oH // 2, oW // 2] = size
            wf[1] = 0
        else:
            wf[1, 5, kH // 2, 0] = size
            gf[:, 1] = 0
        want = torch.nn.grad.conv2d_input(x.shape, wf.double(), gf.double(), d, p, dil)
        assert off(F.dilated_conv_grad_input(gf, wf, H, W, *geo), want) <= gather_bound(K * kH * kW)
    if takes[2] and what == "pixel":
        # an outlier on one side, zeros where its sums read the other: every filter and channel for itself
        for outlier in ("gy", "x"):
            xw, gg, gw, gb = x.clone(), gy.clone(), torch.zeros_like(w), torch.zeros(K, device="cuda")
            if outlier == "gy":
                gg[3, 7, oH // 2, oW // 2] = size
                xw[3] = 0
            else:
                xw[3, 1, H // 2, W // 2] = size
                gg[3] = 0
            F.dilated_conv_acc_grad(xw, gg, gw, gb, *geo)
            want = torch.nn.grad.conv2d_weight(xw.double(), w.shape, gg.double(), d, p, dil)
            rows = (gw.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
            cols = (gw.double() - want).transpose(0, 1).flatten(1).norm(dim=1) / want.transpose(0, 1).flatten(1).norm(dim=1)
            assert max(float(rows.max()), float(cols.max())) <= 2 * gather_bound(N * oH * oW)


@pytest.mark.parametrize("kind", ["normal", "sparse", "gradient"])
def test_ordinary_values_stay_here(F, kind):
    """What a network's layers hold has values close to zero by chance: not a reason to leave the kernels of split operands."""
    from cunn_b200._lib import lib, check
    N, C, H, K = 64, 64, 28, 64
    g = torch.Generator(device="cuda").manual_seed(32)
    x, w = torch.randn(N, C, H, H, device="cuda", generator=g), torch.rand(K, C, 3, 3, device="cuda", generator=g) * 2 - 1
    if kind == "sparse":                                # a ReLU with few active units
        x = (x - torch.linspace(0, 4, C, device="cuda").view(1, -1, 1, 1)).relu()
    elif kind == "gradient":                            # behind a ReLU and a batch normalisation of a million values
        x = torch.where(torch.rand(x.shape, device="cuda", generator=g) < 0.5, x, x * 1e-3)
    geo = (N, C, H, H, K, 3, 3, 1, 1, 1, 1)
    stream = torch.cuda.current_stream().cuda_stream
    y, gx = F.convmm_forward(x, w, None, 1, 1, 1, 1), F.convmm_grad_input(x, w, H, H, 1, 1, 1, 1)
    y0, gx0 = torch.empty_like(y), torch.empty_like(gx)
    check(lib.cunn_b200_convmm_forward(x.data_ptr(), w.data_ptr(), None, y0.data_ptr(), *geo, stream))
    check(lib.cunn_b200_convmm_grad_input(x.data_ptr(), w.data_ptr(), gx0.data_ptr(), *geo, stream))
    assert scratch(0, *geo[:8], 1, 1) and not torch.equal(y, y0) and not torch.equal(gx, gx0)
    gws = [torch.zeros_like(w) for _ in range(2)]
    assert scratch(2, *geo[:8], 1, 1)
    F.convmm_acc_grad(x, x, gws[0], None, 1, 1, 1, 1)
    ws = torch.empty(lib.cunn_b200_convmm_acc_grad_workspace(*geo), dtype=torch.uint8, device="cuda")
    check(lib.cunn_b200_convmm_acc_grad(x.data_ptr(), x.data_ptr(), gws[1].data_ptr(), None, *geo, 1.0, ws.data_ptr(), ws.numel(), stream))
    assert not torch.equal(*gws)
    for got, want in ((y, y0), (gx, gx0), (gws[0], gws[1])):
        assert off(got, want.double()) <= 6e-6


@pytest.mark.parametrize("outlier", ["gy", "x"])
@pytest.mark.parametrize("size", [1e7, 1e12])
def test_large_images_opposite_zeros(F, outlier, size):
    """A parameter gradient of images of two sizes, the large ones opposite zeros and among every eight images in turn."""
    N, C, H, K, k = 20, 37, 40, 320, 4
    assert scratch(2, N, C, H, H, K, k, k, 2, 1, 1)
    g = torch.Generator(device="cuda").manual_seed(35)
    x, gy = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(N, K, 20, 20, device="cuda", generator=g)
    large = torch.arange(N, device="cuda") // 8 % 2 == 0
    a, b = (gy, x) if outlier == "gy" else (x, gy)
    a[large] *= size
    b[large] = 0
    gw = torch.zeros(K, C, k, k, device="cuda")
    F.convmm_acc_grad(x, gy, gw, None, 2, 2, 1, 1)
    want = torch.nn.grad.conv2d_weight(x.double(), gw.shape, gy.double(), 2, 1)
    rows = (gw.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
    assert float(rows.max()) <= 2 * gather_bound(N * 400)


def test_large_values_in_a_later_round(F):
    """Scratch holds 512 MB of split values: a later part of the batch is judged, and taken, for itself; what the call adds to, it adds once."""
    N, C, H, K = 44, 64, 240, 16
    assert scratch(0, N, C, H, H, K, 3, 3, 1, 1, 1) and N * C * H * H * 4 > 512 << 20
    g = torch.Generator(device="cuda").manual_seed(31)
    x, w = torch.randn(N, C, H, H, device="cuda", generator=g), torch.rand(K, C, 3, 3, device="cuda", generator=g) * 2 - 1
    w[:, 1] = 0
    plain = F.convmm_forward(x, w, None, 1, 1, 1, 1)
    x[N - 1, 1] = 1e13
    y = F.convmm_forward(x, w, None, 1, 1, 1, 1)
    assert torch.equal(y[:N // 2], plain[:N // 2])
    for i in (0, N - 1):
        assert off(y[i], torch.nn.functional.conv2d(x[i].double(), w.double(), None, 1, 1)) <= gather_bound(C * 9)
    del y, plain
    assert scratch(2, N, C, H, H, K, 3, 3, 1, 1, 1)
    gy = torch.randn(N, K, H, H, device="cuda", generator=g)
    gy[N - 1] = 0
    gw, gb = torch.ones(K, C, 3, 3, device="cuda"), torch.ones(K, device="cuda")
    F.convmm_acc_grad(x, gy, gw, gb, 1, 1, 1, 1)
    want = sum(torch.nn.grad.conv2d_weight(x[i:i + 4].double(), w.shape, gy[i:i + 4].double(), 1, 1) for i in range(0, N, 4))
    assert off(gw.double() - 1, want) <= 4e-6 and off(gb.double() - 1, gy.double().sum((0, 2, 3))) <= 1e-6


@pytest.mark.parametrize("front", ["functional", "thnn"])
def test_kernel_does_not_depend_on_earlier_calls(F, front):
    """The parameter gradient of a layer that is better off without scratch, before and after another layer has made the shared buffers grow."""
    from cunn_b200 import thnn
    N, C, H, K = 16, 1024, 7, 2048
    g = torch.Generator(device="cuda").manual_seed(33)
    x, gy = torch.randn(N, C, H, H, device="cuda", generator=g), torch.randn(N, K, H, H, device="cuda", generator=g)
    state = thnn.THNN()

    def grad(x, gy):
        w = torch.zeros(gy.shape[1], x.shape[1], 1, 1, device="cuda")
        if front == "thnn":
            state.SpatialConvolutionMM_accGradParameters(x, gy, w.view(w.shape[0], -1), None, 1, 1, 1, 1, 0, 0, 1.0)
        else:
            F.convmm_acc_grad(x, gy, w, None, 1, 1, 0, 0)
        return w

    first = grad(x, gy)
    big = torch.randn(64, 1024, 20, 20, device="cuda", generator=g)
    grad(big, torch.randn(64, 2048, 20, 20, device="cuda", generator=g))
    if front == "functional":
        F.workspace(64 << 20, x.device)
    assert torch.equal(grad(x, gy), first)
    state.close()


def test_thnn_scratch_of_many_streams(F):
    """More streams than buffers were once kept: calls do not wait for what other streams run, give the same results from several threads,
    and the memory is given back with the state."""
    import gc, threading, time
    from cunn_b200 import thnn
    N, C, H, K = 32, 128, 28, 128
    g = torch.Generator(device="cuda").manual_seed(34)
    xs = [torch.randn(N, C, H, H, device="cuda", generator=g) for _ in range(7)]
    w = torch.randn(K, C * 9, device="cuda", generator=g)
    want = [F.convmm_forward(x, w.view(K, C, 3, 3), None, 1, 1, 1, 1) for x in xs]
    streams, states, got = [torch.cuda.Stream() for _ in xs], [thnn.THNN() for _ in xs], [None] * len(xs)
    torch.cuda.synchronize()

    def call(i):
        with torch.cuda.stream(streams[i]):
            got[i] = states[i].SpatialConvolutionMM_updateOutput(xs[i], w, None, 3, 3, 1, 1, 1, 1)

    def everywhere(threads):
        jobs = [threading.Thread(target=call, args=(i,)) for i in range(1, len(xs))] if threads else []
        for t in jobs:
            t.start()
        for t in jobs:
            t.join()
        if not threads:
            for i in range(1, len(xs)):
                call(i)

    for threads in (False, False, True):
        everywhere(threads)
        torch.cuda.synchronize()
    for threads in (False, True):
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(400_000_000)                    # a fifth of a second
        begin = time.perf_counter()
        everywhere(threads)
        assert time.perf_counter() - begin < 0.1
        assert not streams[0].query()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
    gc.collect()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    for s in states:
        s.close()
    assert torch.cuda.mem_get_info()[0] - before >= (scratch(0, N, C, H, H, K, 3, 3, 1, 1, 1) >> 21) << 21
