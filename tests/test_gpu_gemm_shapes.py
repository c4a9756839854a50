"""The tensor-core GEMM of a prompt at the edges of its tiles, K splits and rings."""
import pytest
import torch

from antares_b200 import ops
from antares_b200._lib import call

pytestmark = pytest.mark.gpu


def _case(M, K, N, group, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, generator=g, device="cuda").half()
    q = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device="cuda", dtype=torch.int32)
    s = (torch.rand(K // group, N, generator=g, device="cuda") * 0.019 + 0.001).half()
    return x, q, s


def _nibbles(q):
    return torch.stack([((q >> (4 * j)) & 15) - 8 for j in range(8)], dim=1).view(-1, q.shape[1])


def _check(y, x, w):
    """One fp16 rounding of the result, and fp32 sums: at most K steps of 2^-23 of partial sums that grow like sqrt(K)."""
    want = x.double() @ w
    K = x.shape[1]
    bound = want.abs() * 2 ** -11 + (K ** 0.5) * 2 ** -23 * (x.double().abs() @ w.abs()) + 2 ** -25
    assert bool(((y.double() - want).abs() <= bound).all())


# rows: both sides of a tile of 192 and of the padding to 16; K: fewer units than a ring, splits of uneven length
@pytest.mark.parametrize("M", [1, 17, 32, 33, 128, 143, 176, 192, 193, 300, 385])
@pytest.mark.parametrize("K,N,group", [(64, 8, 64), (192, 264, 192), (256, 256, 128), (1024, 1000, 128), (4096, 4096, 128), (11008, 520, 128)])
def test_prompt_gemm(M, K, N, group):
    x, q, s = _case(M, K, N, group, M + K + N)
    y = torch.full((M + 1, N), 7.0, device="cuda").half()
    ops.w4a16_gemm(x, q, s, out=y[:M])
    w = (_nibbles(q).half() * s.repeat_interleave(group, 0)).double()  # RN_fp16(scale * (q - 8))
    _check(y[:M], x, w)
    assert bool((y[M] == 7).all())
    assert torch.equal(y[:M], ops.w4a16_gemm(x, q, s))
    assert ops.kernel_status() == 0


@pytest.mark.parametrize("M", [1, 17, 40, 128, 256, 300])
@pytest.mark.parametrize("K,F,group", [(64, 8, 64), (256, 128, 128), (1024, 200, 128), (512, 1384, 64), (4096, 11008, 128)])
def test_prompt_gemm_with_swiglu(M, K, F, group):
    x, q, s = _case(M, K, 2 * F, group, M + K + F)
    out = torch.full((M, F), 7.0, device="cuda").half()
    call("ab200_w4a16_gemm_silu", x.data_ptr(), q.data_ptr(), s.data_ptr(), out.data_ptr(), M, K, 2 * F, group, torch.cuda.current_stream().cuda_stream)
    w = (_nibbles(q).half() * s.repeat_interleave(group, 0)).double()
    y = x.double() @ w
    off = y.abs() * 2 ** -11 + (K ** 0.5) * 2 ** -23 * (x.double().abs() @ w.abs()) + 2 ** -25  # of the fp16 projections, as above
    g, u, dg, du = y[:, :F], y[:, F:], off[:, :F], off[:, F:]
    want = torch.nn.functional.silu(g) * u
    # silu's slope is at most 1.1; then one fp16 rounding and a few fp32 steps
    bound = 1.1 * dg * (u.abs() + du) + torch.nn.functional.silu(g).abs() * du + want.abs() * (2 ** -11 + 2 ** -20) + 2 ** -25
    assert bool(((out.double() - want).abs() <= bound).all())
    # the same as the projections on their own and silu(gate) * up after them: one tiling, one order of sums
    both, apart = ops.w4a16_gemm(x, q, s), torch.empty_like(out)
    call("ab200_silu_mul_rows", both.data_ptr(), apart.data_ptr(), M, F, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(apart, out)
    early = torch.empty_like(out)
    call("ab200_w4a16_gemm_early", x.data_ptr(), q.data_ptr(), s.data_ptr(), early.data_ptr(), M, K, 2 * F, group, 1, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(early, out)
    assert ops.kernel_status() == 0


def test_a_recorded_prompt_gemm_survives_larger_ones():
    """A graph holds pointers: nothing the library owns may move when a later call needs more."""
    x, q, s = _case(40, 4096, 512, 128, 1)
    ops.w4a16_gemm(x, q, s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ops.w4a16_gemm(x, q, s)
    graph.replay()
    torch.cuda.synchronize()
    want = y.clone()
    for M in (128, 451, 600):
        ops.w4a16_gemm(*_case(M, 4096, 4096, 128, M))
    torch.cuda.synchronize()
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


@pytest.mark.parametrize("rows,K,N", [(70, 4096, 4096), (300, 4096, 22016), (2000, 4096, 512)])
def test_early_gemm_behind_a_long_kernel(rows, K, N):
    """Started at the beginning of a kernel of up to some milliseconds (prompt attention over values that are not finite),
    whose result it takes: nothing it waits for may run out meanwhile, and it reads the finished result."""
    H = K // 128
    g = torch.Generator(device="cuda").manual_seed(rows)
    qkv = torch.randn(3, rows, H, 128, generator=g, device="cuda").half()
    qkv[2, 0, 0, 3] = float("inf")
    pos = torch.zeros(1, device="cuda", dtype=torch.int32)
    _, q, s = _case(1, K, N, 128, N)
    stream = torch.cuda.current_stream().cuda_stream
    ys = []
    for name, extra in (("ab200_w4a16_gemm_early", 0), ("ab200_w4a16_gemm", 0)):
        att, y = torch.zeros(rows, K, device="cuda").half(), torch.empty(rows, N, device="cuda").half()
        torch.cuda.synchronize()
        call("ab200_attention_prefill", qkv[0].data_ptr(), qkv[1].data_ptr(), qkv[2].data_ptr(), att.data_ptr(), pos.data_ptr(), rows, rows, H, 128, K, 0.09, stream)
        call(name, att.data_ptr(), q.data_ptr(), s.data_ptr(), y.data_ptr(), rows, K, N, 128, extra, stream)
        torch.cuda.synchronize()
        assert ops.kernel_status() == 0 and not att.isfinite().all()
        ys.append(y)
    assert torch.equal(ys[0].isnan(), ys[1].isnan()) and torch.equal(ys[0].nan_to_num(), ys[1].nan_to_num())
