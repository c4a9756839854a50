"""The fp32 decode kernel: raw-nibble products at the edges of its tiles and at magnitudes where the scaling matters."""
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
@pytest.mark.parametrize("mul", [1.0, 2.0 ** -100, 2.0 ** 100])
def test_f32_gemv_matches_64_bits(K, N, group, M, mul):
    x, q, s = _case(M, K, N, group, K + N + M, mul)
    if M == 3:
        x[1] = 0.0                                   # a row of zeros
        x[2, ::2] *= 2.0 ** -20                      # small values beside large ones
    y = ops.w4a16_gemv(x, q, s)
    nib, sw = _wide(q, s, group)
    want = x.double() @ ((nib - 8) * sw)
    # chains of 16 products q * x and the zero-point's sum, one rounding (2^-24) per step of partial sums no larger than
    # sum |x| (q + 8) s; then at most 64 additions across units, warps and CTAs
    bound = (16 + 64) * 2.0 ** -24 * (x.double().abs() @ ((nib + 8) * sw))
    assert bool(((y.double() - want).abs() <= bound).all())
    assert torch.equal(y, ops.w4a16_gemv(x, q, s))


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
