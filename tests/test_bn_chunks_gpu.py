"""Batch-norm sums taken warp by warp: chunks that end inside planes, more chunks than a warp's lanes, planes of odd sizes and
unaligned tensors, constant channels."""
import numpy as np
import pytest

from test_pool_bn_gpu import F, bn_check     # noqa: F401  (F is a fixture)

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (5, 3, 61, 47),          # 14335 elements per channel of an odd plane: chunks end anywhere
    (9, 1, 96, 100),         # one channel, 42 chunks: two rounds of the merging warp
    (1, 2, 1, 2047),         # one element short of a chunk and a half, odd
    (3, 7, 1, 1),            # three elements per channel
    (70, 4, 5, 4),           # five 16-byte items per plane: a warp spans seven planes
    (2, 130, 33, 31),        # more channels than one CTA's warps
    (33, 2, 64, 64),         # 66 chunks of whole items
])
def test_bn_chunk_edges(F, ref64, shape):     # noqa: F811
    rng = np.random.default_rng(abs(hash(shape)) % 99991)
    C = shape[1]
    x = (0.5 + 2.0 * rng.standard_normal(shape)).astype(np.float32)
    w, b = rng.uniform(0, 1, C).astype(np.float32), rng.uniform(-1, 1, C).astype(np.float32)
    rm0, rv0 = rng.standard_normal(C).astype(np.float32), rng.uniform(0.5, 2, C).astype(np.float32)
    bn_check(F, ref64, x, w, b, rm0, rv0, rng.standard_normal(shape).astype(np.float32), 0.1, 1e-5, 0.5,
             gw0=rng.standard_normal(C).astype(np.float32), gb0=rng.standard_normal(C).astype(np.float32))


def test_bn_unaligned_tensor_equals_aligned(F):     # noqa: F811
    x = torch.randn(4, 6, 20, 20, device="cuda")
    buf = torch.empty(x.numel() + 1, device="cuda")
    shifted = buf[1:].view(x.shape).copy_(x)
    stats = [(torch.zeros(6, device="cuda"), torch.ones(6, device="cuda")) for _ in range(2)]
    a, b = (F.batchnorm_forward(t, None, None, *s, True) for t, s in zip((x, shifted), stats))
    for p, q in zip(a, b):
        assert torch.allclose(p, q, rtol=2e-6, atol=2e-6)


@pytest.mark.parametrize("shape,value", [((3, 2, 10, 10), 0.1), ((8, 3, 64, 48), 1e4 / 3), ((1, 2, 5, 5), -7.3)])
def test_bn_constant_channel_has_no_variance(F, shape, value):     # noqa: F811
    x = torch.full(shape, value, device="cuda")
    rm, rv = torch.zeros(shape[1], device="cuda"), torch.ones(shape[1], device="cuda")
    y, sm, ss = F.batchnorm_forward(x, None, None, rm, rv, True, 0.1, 0.0)
    assert torch.equal(sm, torch.full_like(sm, value)) and torch.all(ss == 0) and torch.all(y == 0)


@pytest.mark.parametrize("shape", [(3, 4, 20, 20), (40, 3, 31, 29), (2, 5000, 5, 7), (9, 2, 96, 100)])
def test_bn_statistics_of_what_is_not_finite(F, shape):     # noqa: F811
    """The mean is a sum: infinite where one sign of infinity is among the values, wherever it stands, NaN for both or a NaN."""
    inf = float("inf")
    for first in (True, False):
        x = torch.randn(shape, device="cuda")
        at = (0, slice(None), 0, 0) if first else (shape[0] - 1, slice(None), shape[2] - 1, shape[3] - 1)
        bad = torch.zeros(shape[1], device="cuda")
        bad[0], bad[1], bad[2 % shape[1]] = inf, -inf, float("nan")
        x[at] += bad
        rm, rv = torch.zeros(shape[1], device="cuda"), torch.ones(shape[1], device="cuda")
        _, sm, ss = F.batchnorm_forward(x, None, None, rm, rv, True, 0.1, 1e-5)
        want = x.double().mean((0, 2, 3)).float()
        assert torch.allclose(sm, want, rtol=1e-5, atol=1e-6, equal_nan=True) and torch.allclose(rm, 0.1 * want, rtol=1e-5, atol=1e-6, equal_nan=True)
        assert torch.equal(torch.isnan(ss), ~torch.isfinite(want)) and torch.equal(torch.isnan(rv), ~torch.isfinite(want))


def test_bn_constant_channel_of_large_values(F):     # noqa: F811
    x = torch.full((2, 3, 16, 16), 5e36, device="cuda")
    rm, rv = torch.zeros(3, device="cuda"), torch.ones(3, device="cuda")
    y, sm, _ = F.batchnorm_forward(x, None, None, rm, rv, True, 0.1, 1e-5)
    assert torch.equal(sm, torch.full_like(sm, 5e36)) and torch.all(y == 0)
