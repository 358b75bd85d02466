"""Max pooling and batch normalisation: CUDA kernels (flat C ABI) against the CPU oracle and the committed
PyTorch-CPU fixtures.  Pooling indices must match exactly; values/forward 1e-5, gradients 1e-4."""
import numpy as np
import pytest

from conftest import golden, rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FWD_TOL = 1e-5
GRAD_TOL = 1e-4


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


@pytest.fixture(params=[1, 2], ids=["default-kernels", "grouped-kernels"])
def grouped_mode(request):
    """Batch norm has two kernel families: two launches (statistics, then normalise) and one launch that walks
    groups of channels so that the second read comes from L2.  Mode 2 routes every shape the latter applies to
    through it, forward and backward; mode 1 is the library's default choice."""
    from cunn_b200._lib import lib
    lib.cunn_b200_batchnorm_set_grouped(request.param)
    yield request.param
    lib.cunn_b200_batchnorm_set_grouped(1)


# ---------------------------------------------------------------- max pooling
@pytest.mark.parametrize("name", ["maxpool_3s2p1", "maxpool_ceil", "maxpool_ties", "maxpool_2s2"])
def test_maxpool_golden(F, ref64, name):
    g = golden(name)
    k, d, pad, ceil_mode = [int(v) for v in g["params"]]
    y, ind = F.maxpool_forward(dev(g["x"]), k, k, d, d, pad, pad, bool(ceil_mode))
    assert np.array_equal(host(y), g["y"])
    assert np.array_equal(host(ind), g["ind0"] + ref64.index_base)
    H, W = g["x"].shape[2:]
    gx = F.maxpool_backward(dev(g["gy"]), ind, H, W, k, k, d, d, pad, pad, bool(ceil_mode))
    assert rel_err(host(gx), g["gx"]) < 1e-5


@pytest.mark.parametrize("shape", [
    # N, C, H, W, k, d, pad, ceil, ties
    (2, 3, 112, 112, 3, 2, 1, False, False),   # fast path (geometry of the benchmarked pooling layer)
    (2, 5, 32, 48, 3, 2, 1, False, True),      # fast path with many ties
    (3, 2, 31, 40, 3, 2, 1, False, True),      # fast path, odd height
    (2, 3, 112, 112, 3, 2, 1, True, False),    # ceil mode changes the output size -> generic
    (2, 4, 17, 19, 3, 2, 1, True, True),
    (1, 3, 20, 20, 2, 2, 0, False, True),
    (2, 2, 15, 15, 3, 1, 1, False, True),
    (2, 2, 14, 14, 5, 3, 2, True, False),
    (1, 1, 3, 3, 3, 2, 1, False, False),
    (4, 8, 56, 56, 3, 2, 1, False, False),
])
def test_maxpool_shapes(F, ref64, shape):
    N, C, H, W, k, d, pad, ceil_mode, ties = shape
    rng = np.random.default_rng(abs(hash(shape)) % 99991)
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    if ties:
        x = np.round(x * 2) / 2
    ry, rind = ref64.maxpool_forward(x, k, k, d, d, pad, pad, ceil_mode)
    y, ind = F.maxpool_forward(dev(x), k, k, d, d, pad, pad, ceil_mode)
    assert tuple(y.shape) == ry.shape
    assert np.array_equal(host(y), ry)
    assert int((host(ind) != rind).sum()) == 0          # indices bit-exact
    gy = rng.standard_normal(ry.shape).astype(np.float32)
    gx = F.maxpool_backward(dev(gy), ind, H, W, k, k, d, d, pad, pad, ceil_mode)
    assert rel_err(host(gx), ref64.maxpool_backward(gy, rind, H, W, k, k, d, d, pad, pad)) < 1e-5  # fp32 sums of up to k*k gradients


def test_maxpool_nan_and_inf_windows(F, ref64):
    # NaN / -inf never win the strict compare; an all-NaN window stores index -1 + base and -FLT_MAX
    x = np.random.default_rng(3).standard_normal((1, 2, 16, 16)).astype(np.float32)
    x[0, 0, :5, :5] = np.nan
    x[0, 1, 4:9, 8:] = -np.inf
    x[0, 1, 0, 0] = np.inf
    for k, d, pad in ((3, 2, 1), (2, 2, 0)):
        ry, rind = ref64.maxpool_forward(x, k, k, d, d, pad, pad, False)
        y, ind = F.maxpool_forward(dev(x), k, k, d, d, pad, pad, False)
        assert np.array_equal(host(ind), rind)
        assert np.array_equal(host(y), ry)
    assert rind.min() >= -1 + ref64.index_base


def test_maxpool_rejects_bad_arguments(F):
    from cunn_b200 import CunnError
    x = torch.zeros((1, 1, 8, 8), device="cuda")
    with pytest.raises(CunnError, match="pad should be smaller than half of kernel size"):
        F.maxpool_forward(x, 2, 2, 2, 2, 2, 2, out=torch.zeros(1, device="cuda"),
                          indices=torch.zeros(1, dtype=torch.int64, device="cuda"))


def test_maxpool_full_size_properties(F):
    # the benchmarked geometry at reduced batch (N=32): the stored index must point at the stored value,
    # and backward must conserve the gradient mass: sum(gx) == sum(gy).
    torch.manual_seed(0)
    x = torch.randn((32, 64, 112, 112), device="cuda") * 2 + 0.5
    y, ind = F.maxpool_forward(x, 3, 3, 2, 2, 1, 1)
    from cunn_b200._lib import lib
    flat = x.view(32 * 64, -1)
    picked = torch.gather(flat, 1, (ind.view(32 * 64, -1) - 1))
    assert torch.equal(picked.view_as(y), y)
    gy = torch.randn_like(y)
    gx = F.maxpool_backward(gy, ind, 112, 112, 3, 3, 2, 2, 1, 1)
    assert abs(float(gx.double().sum()) - float(gy.double().sum())) < 1e-6 * float(gy.double().abs().sum())


# ---------------------------------------------------------------- batch normalisation
def bn_check(F, ref64, x, w, b, rm0, rv0, gy, momentum, eps, scale, gw0=None, gb0=None):
    C = x.shape[1]
    # training forward
    ry, rrm, rrv, rsm, rss = ref64.bn_forward(x, w, b, rm0, rv0, True, momentum, eps)
    rm, rv = dev(rm0), dev(rv0)
    y, sm, ss = F.batchnorm_forward(dev(x), None if w is None else dev(w), None if b is None else dev(b), rm, rv,
                                    True, momentum, eps)
    assert rel_err(host(y), ry) < FWD_TOL
    assert rel_err(host(sm), rsm) < FWD_TOL and rel_err(host(ss), rss) < FWD_TOL
    assert rel_err(host(rm), rrm) < FWD_TOL and rel_err(host(rv), rrv) < FWD_TOL
    # training backward (accumulating into non-zero gradWeight / gradBias with scale)
    gw0 = np.zeros(C, np.float32) if gw0 is None else gw0
    gb0 = np.zeros(C, np.float32) if gb0 is None else gb0
    rgx, rgw, rgb = ref64.bn_backward(x, gy, w, rrm, rrv, rsm, rss, True, scale, eps, gw=gw0, gb=gb0)
    gw, gb = dev(gw0), dev(gb0)
    gx = F.batchnorm_backward(dev(x), dev(gy), None if w is None else dev(w), rm, rv, sm, ss, True, scale, eps,
                              grad_weight=gw, grad_bias=gb)
    assert rel_err(host(gx), rgx) < GRAD_TOL
    assert rel_err(host(gw), rgw) < GRAD_TOL and rel_err(host(gb), rgb) < GRAD_TOL
    # inference forward / backward on the given running statistics
    ry, rm2, rv2, _, _ = ref64.bn_forward(x, w, b, rm0, rv0, False, momentum, eps)
    rm, rv = dev(rm0), dev(rv0)
    y, _, _ = F.batchnorm_forward(dev(x), None if w is None else dev(w), None if b is None else dev(b), rm, rv,
                                  False, momentum, eps)
    assert rel_err(host(y), ry) < FWD_TOL
    assert np.array_equal(host(rm), rm0) and np.array_equal(host(rv), rv0)   # untouched in inference
    rgx, rgw, rgb = ref64.bn_backward(x, gy, w, rm0, rv0, rsm, rss, False, scale, eps, gw=gw0, gb=gb0)
    gw, gb = dev(gw0), dev(gb0)
    gx = F.batchnorm_backward(dev(x), dev(gy), None if w is None else dev(w), rm, rv, sm, ss, False, scale, eps,
                              grad_weight=gw, grad_bias=gb)
    assert rel_err(host(gx), rgx) < GRAD_TOL
    assert rel_err(host(gw), rgw) < GRAD_TOL and rel_err(host(gb), rgb) < GRAD_TOL
    # gradInput only / parameters only (the reference lets any of the three be NULL)
    gx_only = F.batchnorm_backward(dev(x), dev(gy), None if w is None else dev(w), rm, rv, sm, ss, True, scale, eps)
    rgx_t, _, _ = ref64.bn_backward(x, gy, w, rrm, rrv, rsm, rss, True, scale, eps)
    assert rel_err(host(gx_only), rgx_t) < GRAD_TOL
    gw = dev(gw0)
    assert F.batchnorm_backward(dev(x), dev(gy), None if w is None else dev(w), rm, rv, sm, ss, True, scale, eps,
                                grad_weight=gw, want_gx=False) is None
    _, rgw_t, _ = ref64.bn_backward(x, gy, w, rrm, rrv, rsm, rss, True, scale, eps, gw=gw0, want_gx=False)
    assert rel_err(host(gw), rgw_t) < GRAD_TOL


@pytest.mark.parametrize("name", ["bn_affine", "bn_plain"])
def test_bn_golden(F, name):
    g = golden(name)
    affine = int(g["params"][0])
    w = dev(g["g"]) if affine else None
    b = dev(g["b"]) if affine else None
    mom, eps, scale = float(g["momentum"]), float(g["eps"]), float(g["scale"])
    rm, rv = dev(g["rm0"]), dev(g["rv0"])
    y, sm, ss = F.batchnorm_forward(dev(g["x"]), w, b, rm, rv, True, mom, eps)
    assert rel_err(host(y), g["y_train"]) < FWD_TOL
    assert rel_err(host(rm), g["rm_train"]) < FWD_TOL and rel_err(host(rv), g["rv_train"]) < FWD_TOL
    assert rel_err(host(sm), g["save_mean"]) < FWD_TOL and rel_err(host(ss), g["save_std"]) < FWD_TOL
    C = g["x"].shape[1]
    gw, gb = torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda")
    gx = F.batchnorm_backward(dev(g["x"]), dev(g["gy"]), w, rm, rv, sm, ss, True, scale, eps, grad_weight=gw, grad_bias=gb)
    assert rel_err(host(gx), g["gx_train"]) < GRAD_TOL
    if affine:
        assert rel_err(host(gw), g["gw_train"]) < GRAD_TOL and rel_err(host(gb), g["gb_train"]) < GRAD_TOL
    rm, rv = dev(g["rm0"]), dev(g["rv0"])
    y, _, _ = F.batchnorm_forward(dev(g["x"]), w, b, rm, rv, False, mom, eps)
    assert rel_err(host(y), g["y_eval"]) < FWD_TOL


@pytest.mark.parametrize("shape,affine", [
    ((4, 64, 112, 112), True),     # the benchmarked geometry, reduced batch
    ((7, 5, 9, 11), True),         # S not a multiple of 4 -> scalar path
    ((3, 16, 32, 32), False),      # H*W = 1024, the reference's extra case; no affine
    ((300, 3, 2, 2), True),        # more images than chunks
    ((2, 1024, 7, 7), True),
    ((6, 24, 14, 14), True),       # 196-element planes: a multiple of 16 bytes, yet on the flat elementwise kernels
    ((4, 8, 2, 3), True),          # 24 elements per channel
    ((16, 4100, 2, 2), True),      # more channels than ticket counters: the merge runs as a separate launch
    ((40, 2, 16, 16), True),       # 40 chunks per channel: more than one warp-lane round in the merge
    ((64, 6, 28, 28), True),       # grouped kernels: several channels per CTA share
    ((12, 37, 20, 20), False),     # grouped kernels: a channel count that does not divide into equal groups
    ((48, 3, 112, 112), True),     # grouped kernels: planes longer than a stage
])
def test_bn_shapes(F, ref64, shape, affine, grouped_mode):
    rng = np.random.default_rng(abs(hash(shape)) % 99991)
    C = shape[1]
    x = (0.5 + 2.0 * rng.standard_normal(shape)).astype(np.float32)
    w = rng.uniform(0, 1, C).astype(np.float32) if affine else None
    b = rng.uniform(-1, 1, C).astype(np.float32) if affine else None
    rm0 = rng.standard_normal(C).astype(np.float32)
    rv0 = rng.uniform(0.5, 2, C).astype(np.float32)
    gy = rng.standard_normal(shape).astype(np.float32)
    bn_check(F, ref64, x, w, b, rm0, rv0, gy, 0.1, 1e-5, 0.5,
             gw0=rng.standard_normal(C).astype(np.float32), gb0=rng.standard_normal(C).astype(np.float32))


def test_bn_large_mean_small_std(F, ref64, grouped_mode):
    # |mean| >> std: a plain sum-of-squares in fp32 would lose the variance; the shifted sums must not.
    rng = np.random.default_rng(11)
    x = (100.0 + 0.01 * rng.standard_normal((8, 4, 28, 28))).astype(np.float32)
    rm0, rv0 = np.zeros(4, np.float32), np.ones(4, np.float32)
    _, _, _, rsm, rss = ref64.bn_forward(x, None, None, rm0, rv0, True, 0.1, 1e-5)
    rm, rv = dev(rm0), dev(rv0)
    _, sm, ss = F.batchnorm_forward(dev(x), None, None, rm, rv, True, 0.1, 1e-5)
    assert rel_err(host(sm), rsm) < 1e-6
    assert rel_err(host(ss), rss) < 1e-4


def test_bn_single_element_and_zero_variance(F):
    # n = 1 gives NaN running_var (division by n - 1 = 0) and, with eps = 0, invstd = 0 — both are the
    # reference's behaviour (BatchNormalization.cu:188-200) and are kept.
    x = torch.full((1, 2, 1, 1), 3.0, device="cuda")
    rm, rv = torch.zeros(2, device="cuda"), torch.ones(2, device="cuda")
    y, sm, ss = F.batchnorm_forward(x, None, None, rm, rv, True, 0.1, 0.0)
    assert torch.all(ss == 0) and torch.all(y == 0) and torch.all(sm == 3.0)
    assert torch.all(torch.isnan(rv))


@pytest.mark.parametrize("shape", [(4, 8, 14, 14), (3, 5, 7, 9), (64, 6, 28, 28)])
def test_bn_relu_fused_equals_separate_calls(F, shape, grouped_mode):
    # the fused BN+ReLU pair must equal BatchNormalization followed by Threshold(0, 0), forward and backward
    g = torch.Generator(device="cuda").manual_seed(9)
    C = shape[1]
    x = torch.randn(shape, device="cuda", generator=g) * 2 + 0.3
    w, b = torch.rand(C, device="cuda", generator=g), torch.rand(C, device="cuda", generator=g) - 0.5
    gy = torch.randn(shape, device="cuda", generator=g)
    rm1, rv1, rm2, rv2 = (torch.zeros(C, device="cuda"), torch.ones(C, device="cuda"), torch.zeros(C, device="cuda"),
                          torch.ones(C, device="cuda"))
    z, sm, ss = F.batchnorm_forward(x, w, b, rm1, rv1, True)
    y_ref = F.threshold_forward(z)
    y, sm2, ss2 = F.batchnorm_relu_forward(x, w, b, rm2, rv2, True)
    assert torch.equal(y, y_ref) and torch.equal(sm, sm2) and torch.equal(ss, ss2) and torch.equal(rm1, rm2)
    gw1, gb1, gw2, gb2 = (torch.zeros(C, device="cuda") for _ in range(4))
    gx_ref = F.batchnorm_backward(x, F.threshold_backward(z, gy), w, rm1, rv1, sm, ss, True, grad_weight=gw1, grad_bias=gb1)
    gx = F.batchnorm_relu_backward(x, gy, w, b, rm2, rv2, sm2, ss2, True, grad_weight=gw2, grad_bias=gb2)
    assert torch.equal(gx, gx_ref) and torch.equal(gw1, gw2) and torch.equal(gb1, gb2)


def test_bn_full_size_properties(F):
    # the benchmarked geometry at reduced batch (N = 64; test_full_size_gpu.py runs the full 256):
    # with gamma = 1, beta = 0 the training output has zero mean and unit biased variance per channel, the
    # saved statistics are those of x, and the input gradient is orthogonal to 1 and to (x - mean).
    g = torch.Generator(device="cuda").manual_seed(8)
    N, C, HW = 64, 64, 112
    x = torch.randn((N, C, HW, HW), device="cuda", generator=g) * 2 + 0.5
    rm, rv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    y, sm, ss = F.batchnorm_forward(x, None, None, rm, rv, True, 0.1, 1e-5)
    xd = x.double()
    mean = xd.mean((0, 2, 3))
    var = xd.var((0, 2, 3), unbiased=False)
    assert float((sm.double() - mean).abs().max()) < 1e-5 * float(mean.abs().max())
    assert float((ss.double() - 1 / torch.sqrt(var + 1e-5)).abs().max()) < 1e-5
    yd = y.double()
    assert float(yd.mean((0, 2, 3)).abs().max()) < 1e-5
    assert float((yd.var((0, 2, 3), unbiased=False) - 1).abs().max()) < 1e-4
    n = N * HW * HW
    assert float((rv.double() - (0.9 + 0.1 * var * n / (n - 1))).abs().max()) < 1e-5 * float(var.max())
    gy = torch.randn((N, C, HW, HW), device="cuda", generator=g)
    gx = F.batchnorm_backward(x, gy, None, rm, rv, sm, ss, True)
    gxd = gx.double()
    scale = float(gxd.abs().sum((0, 2, 3)).max())
    assert float(gxd.sum((0, 2, 3)).abs().max()) < 1e-5 * scale
    assert float((gxd * (xd - mean.view(1, C, 1, 1))).sum((0, 2, 3)).abs().max()) < 1e-5 * scale * 2


@pytest.mark.parametrize("shape", [
    # N, C, H, W: planes of 1025 to 4000 elements (backward too), larger ones, few of them; slabs of 28 MB groups
    (96, 101, 60, 60),       # three groups of 34 channels, the last smaller: CTAs whose shares end inside a channel
    (130, 67, 64, 68),       # two groups
    (16, 70, 180, 172),      # backward on two launches
    (2, 17, 1024, 1000),     # two planes a channel
    (129, 9, 112, 112),      # less than 128 MB
])
@pytest.mark.parametrize("relu", [False, True])
def test_batchnorm_groups_of_channels(F, shape, relu):
    """Layers large enough for the kernels that walk groups of channels, against fp64."""
    import torch
    N, C, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.randn(shape, device="cuda", generator=g) * 2 + torch.arange(C, device="cuda").view(1, C, 1, 1) * 0.5
    w, b = torch.rand(C, device="cuda", generator=g) + 0.5, torch.randn(C, device="cuda", generator=g)
    gy = torch.randn(shape, device="cuda", generator=g)
    rm, rv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    gw, gb = torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda")
    forward = F.batchnorm_relu_forward if relu else F.batchnorm_forward
    y, mean, std = forward(x, w, b, rm, rv, True)
    if relu:
        gx = F.batchnorm_relu_backward(x, gy, w, b, rm, rv, mean, std, True, 1.0, 1e-5, gw, gb)
    else:
        gx = F.batchnorm_backward(x, gy, w, rm, rv, mean, std, True, 1.0, 1e-5, gw, gb)
    n, col = N * H * W, lambda t: t.double().view(1, C, 1, 1)
    m64 = x.double().mean((0, 2, 3))
    v64 = x.double().var((0, 2, 3), unbiased=False)
    # the mean is rounded to fp32; a sum of n fp32 values in chains, then fp64, is far closer than 1e-6 of the deviation
    assert float(((mean.double() - m64).abs() / (m64.abs() * 2.0 ** -24 + 1e-6 * v64.sqrt())).max()) <= 1
    assert torch.allclose(std.double(), (v64 + 1e-5).rsqrt(), rtol=1e-6, atol=0)
    assert torch.allclose(rv.double(), 0.9 + 0.1 * v64 * n / (n - 1), rtol=1e-6, atol=0)
    xh = (x.double() - col(m64)) * (col(v64) + 1e-5).rsqrt()
    t = xh * col(w) + col(b)
    keep = (t > 0) if relu else torch.ones_like(t, dtype=torch.bool)
    sure = t.abs() > 1e-4                                # beyond rounding from where the ReLU turns
    # three roundings of values up to |x| / std and 8
    bound = 4 * 2.0 ** -24 * (x.double().abs() * (col(v64) + 1e-5).rsqrt() * col(w) + 8)
    assert bool(((y.double() - torch.where(keep, t, 0.0)).abs() <= bound + (0 if not relu else 1e-6)).all())
    g64 = torch.where(y > 0, gy, torch.zeros_like(gy)).double() if relu else gy.double()
    gb64, gw64 = g64.sum((0, 2, 3)), (g64 * xh).sum((0, 2, 3))
    size = n ** 0.5
    assert float((gb.double() - gb64).abs().max()) <= 1e-5 * size and float((gw.double() - gw64).abs().max()) <= 1e-5 * size
    gx64 = (g64 - col(gb64) / n - xh * col(gw64) / n) * col(w) * (col(v64) + 1e-5).rsqrt()
    assert float(((gx.double() - gx64).abs() * sure).max()) <= 1e-5


@pytest.mark.parametrize("mean", [10.0, 100.0, 1000.0])
@pytest.mark.parametrize("shape", [(128, 96, 56, 56), (2, 17, 1024, 1000), (129, 9, 112, 112)])
def test_batchnorm_groups_shift_by_typical_values(F, shape, mean):
    """Channels whose first values are none of the others' size (a border of zeros): the squares about the shift stay small beside what they are
    summed to.  A CTA's shift is off by at most 32 / 1024 of the mean in the share with the border, where its fp32 chains of 256 squares round by
    2^-24 of them; the other shares' shift is within a tenth of the deviation."""
    import torch
    N, C, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(12)
    x = torch.randn(shape, device="cuda", generator=g) + mean
    x.view(N, C, -1)[0, :, :32] = 0
    rm, rv = torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda")
    _, m, _ = F.batchnorm_forward(x, None, None, rm, rv, True)
    n = N * H * W
    m64, v64 = x.double().mean((0, 2, 3)), x.double().var((0, 2, 3))
    share = 4096.0 * 16 / n                                    # of the channel's values that are in the share with the border, or more
    bound = 1e-6 + 2.0 ** -24 * 16 * share * (mean / 32) ** 2
    assert float(((rv.double() * 10 - v64) / v64).abs().max()) <= bound
    assert float(((m.double() - m64).abs() / (m64.abs() * 2.0 ** -24 + 1e-6 * v64.sqrt())).max()) <= 1


@pytest.mark.parametrize("shape", [(128, 96, 56, 56), (129, 9, 112, 112)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_batchnorm_groups_of_what_is_not_finite(F, shape, value):
    """An infinity is the mean's, wherever it is; the other channels are what they were.  A constant channel has no variance at all."""
    import torch
    N, C, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(13)
    x = torch.randn(shape, device="cuda", generator=g)
    x[:, 5] = 0.1
    want = F.batchnorm_forward(x, None, None, torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda"), True)
    assert float(want[1][5]) == float(torch.tensor(0.1))
    rv0 = torch.zeros(C, device="cuda")
    F.batchnorm_forward(x, None, None, torch.zeros(C, device="cuda"), rv0, True)
    assert float(rv0[5]) == 0
    for at in ((0, 2, 0, 3), (N // 2, 2, 5, 7), (N - 1, 2, H - 1, W - 1)):
        z = x.clone()
        z[at] = value
        y, m, s = F.batchnorm_forward(z, None, None, torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda"), True)
        assert m[2].isnan() if value != value else float(m[2]) == value
        others = [c for c in range(C) if c != 2]
        assert torch.equal(m[others], want[1][others]) and torch.equal(s[others], want[2][others]) and torch.equal(y[:, others], want[0][:, others])


@pytest.mark.parametrize("shape", [(128, 128, 56, 56), (2, 16, 1024, 1024)])
def test_batchnorm_groups_gradient_sums(F, shape):
    """The weight's gradient of layers on the one-launch backward kernel.  A chain of 42 fp32 multiply-adds is off by 2^-25.8 (42 / 2^0.5) of a
    term, 7.8e-8 of its own size sqrt(42); so are their sums, with a largest of 4 times that among the channels and twice for the products."""
    import torch
    N, C, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(3)
    x, gy = torch.randn(shape, device="cuda", generator=g) + 30, torch.randn(shape, device="cuda", generator=g) + 0.5
    w, rm, rv = torch.ones(C, device="cuda"), torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    _, mean, std = F.batchnorm_forward(x, w, None, rm, rv, True)
    gw, gb = torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda")
    F.batchnorm_backward(x, gy, w, rm, rv, mean, std, True, 1.0, 1e-5, gw, gb)
    col = lambda t: t.double().view(1, C, 1, 1)
    want = (gy.double() * (x.double() - col(mean)) * col(std)).sum((0, 2, 3))
    assert float((gw.double() - want).abs().max()) <= 6e-7 * (N * H * W) ** 0.5
