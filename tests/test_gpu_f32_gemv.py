"""The fp32 decode kernel at the edges of its tiles and at magnitudes where its scaled products, or the sums of them, could leave the range."""
import math

import pytest
import torch

from antares_b200 import ops

pytestmark = pytest.mark.gpu


def _case(M, K, N, group, seed, mul=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, generator=g, device="cuda") * mul
    q = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device="cuda", dtype=torch.int32)
    s = torch.rand(K // group, N, generator=g, device="cuda") * 0.019 + 0.001
    return x, q, s


def _wide(q, s, group):
    nib = torch.stack([(q >> (4 * j)) & 15 for j in range(8)], dim=1).view(-1, q.shape[1]).double()
    return nib, s.double().repeat_interleave(group, 0)


@pytest.mark.parametrize("K,N,group", [(32, 4, 32), (128, 132, 128), (288, 256, 32), (4096, 4096, 128), (11008, 520, 128)])
@pytest.mark.parametrize("M", [1, 2, 3])
@pytest.mark.parametrize("mul", [1.0, 2.0 ** -120, 2.0 ** -100, 2.0 ** -97, 2.0 ** 100, 2.0 ** 102, 2.0 ** 121, 2.0 ** 122])
def test_f32_gemv_matches_64_bits(K, N, group, M, mul):
    x, q, s = _case(M, K, N, group, K + N + M, mul)
    if M == 3:
        x[1] = 0.0                                   # a row of zeros
        x[2, ::2] *= 2.0 ** -20                      # small values beside large ones
    y = ops.w4a16_gemv(x, q, s)
    nib, sw = _wide(q, s, group)
    want = x.double() @ ((nib - 8) * sw)
    _close(y, x, nib, sw, want)
    assert torch.equal(y, ops.w4a16_gemv(x, q, s))
    if K >= 1024:
        # as a whole: chains of at most 8 products a lane, then 32-k units a warp (at most 43 of them), 8 warps, 8 CTAs.  Rounding
        # errors of about 2^-25 of each partial sum, the sums growing like a random walk: sqrt(64 / 2) * 2^-25
        assert float((y.double() - want).norm()) <= 32 ** 0.5 * 2.0 ** -24 * float(want.norm())


def _close(y, x, nib, sw, want):
    # a product passes through at most 80 roundings (2^-24 of partial sums no larger than sum |x (q - 8)| s); 2^-149: the smallest step
    bound = 80 * 2.0 ** -24 * (x.double().abs() @ ((nib - 8).abs() * sw)) + x.shape[1] * 2.0 ** -149
    assert bool(((y.double() - want).abs() <= bound).all()), float(((y.double() - want).abs() / bound).max())


@pytest.mark.parametrize("K,M", [(1024, 1), (4096, 2)])
@pytest.mark.parametrize("big", [2.0 ** 14, 2.0 ** 60, 2.0 ** 101, 2.0 ** 126])
def test_f32_gemv_large_activation_that_meets_zero_weights(K, M, big):
    """One activation far above the others whose weights are all zero (nibble 8) has no part in the result, nor in its error."""
    x, q, s = _case(M, K, 256, 128, K, 2.0 ** -3)
    k = 77
    x[:, k] = big
    q[k // 8] = (q[k // 8] & ~(15 << (4 * (k % 8)))) | (8 << (4 * (k % 8)))
    nib, sw = _wide(q, s, 128)
    assert bool((nib[k] == 8).all())
    _close(ops.w4a16_gemv(x, q, s), x, nib, sw, x.double() @ ((nib - 8) * sw))


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
def test_f32_gemv_special_values(value):
    """One infinite activation against a weight of either sign, or against zero: what x * scale * (q - 8) gives."""
    x, q, s = _case(2, 4096, 256, 128, 5)
    x[0, 1003] = value
    y = ops.w4a16_gemv(x, q, s)
    nib, sw = _wide(q, s, 128)
    w = (nib - 8) * sw
    want = torch.full((256,), math.nan, device="cuda", dtype=torch.float64) if math.isnan(value) else value * w[1003]
    assert torch.equal(y[0].isnan(), want.isnan()) and torch.equal(y[0][~want.isnan()].double(), want[~want.isnan()])
    assert torch.isfinite(y[1]).all()


@pytest.mark.parametrize("value", [math.inf, math.nan])
def test_f32_gemv_scales_that_are_not_finite(value):
    """scale * (q - 8) is formed first: an infinite scale times a zero weight is not a number, and so is its column."""
    x, q, s = _case(1, 1024, 256, 128, 9)
    s[3, 10] = value
    y = ops.w4a16_gemv(x, q, s)
    nib, sw = _wide(q, s, 128)
    want = x.double() @ ((nib - 8) * sw)
    assert bool(want[0, 10].isnan()) and bool(y[0, 10].isnan()) and int(y.isfinite().sum()) == 255


@pytest.mark.parametrize("K,N", [(4096, 256), (11008, 4096)])
def test_f32_gemv_scales_from_the_kernel_before(K, N):
    """The scales of a call are the result of the one launched just before it, which lets its successor start early."""
    x, q, s = _case(1, K, N, 128, 11)
    x2, q2, _ = _case(1, 128, N, 128, 12)
    want = ops.w4a16_gemv(x, q, s).clone()
    torch.cuda.synchronize()
    ref = ops.w4a16_gemv(x2, q2, want.view(1, N))
    torch.cuda.synchronize()
    for _ in range(20):
        assert torch.equal(ops.w4a16_gemv(x2, q2, ops.w4a16_gemv(x, q, s).view(1, N)), ref)
