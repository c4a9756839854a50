"""The native front end against the Python code behind it: same results where it takes the call, and whatever it does
not take (strides, types, subclasses, errors) ends as it does without it."""
import pytest
import torch

import autort
from antares_b200 import autort_api, ops

pytestmark = pytest.mark.gpu


class _Declines:
    """Stands in for the native front end: takes no call."""

    def __getattr__(self, name):
        return (lambda *a: object()) if name == "program" else (lambda *a: None)


@pytest.fixture
def python_only(monkeypatch):
    def switch(on):
        monkeypatch.setattr(ops, "fast", (lambda: _Declines()) if on else _REAL)
        monkeypatch.setattr(autort_api, "fast", (lambda: _Declines()) if on else _REAL)
    yield switch
    switch(False)


_REAL = ops.fast


class _Sub(torch.Tensor):
    pass


def _gen(seed=0):
    return torch.Generator(device="cuda").manual_seed(seed)


def _w4(K, N, dtype, g):
    q = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device="cuda", dtype=torch.int32)
    return q, (torch.rand(K // 128, N, generator=g, device="cuda") * 0.019 + 0.001).to(dtype)


def _both(python_only, call):
    """(value or exception) of the call with and without the native front end."""
    got = []
    for on in (False, True):
        python_only(on)
        try:
            got.append(call())
        except Exception as e:  # noqa: BLE001 - the kind and text are compared
            got.append(e)
    return got


def _same(python_only, call):
    a, b = _both(python_only, call)
    if isinstance(b, Exception):
        assert type(a) is type(b) and str(a) == str(b), (a, b)
    else:
        assert type(a) is type(b) and a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(256,), (1, 256), (3, 256), (2, 3, 256), (17, 256), (0, 256), (255,)])
def test_projection_forms(python_only, dtype, shape):
    g = _gen()
    q, s = _w4(256, 264, dtype if dtype != torch.bfloat16 else torch.float16, g)
    x = torch.randn(*shape, generator=g, device="cuda").to(dtype)
    for f in (ops.w4a16_matmul, ops.w4a16_gemv, ops.w4a16_gemm):
        _same(python_only, lambda: f(x, q, s))
    if x.dim() == 2 and shape[0] == 3:
        _same(python_only, lambda: ops.w4a16_matmul(x.t().contiguous().t(), q, s))  # not contiguous
        _same(python_only, lambda: ops.w4a16_matmul(x.as_subclass(_Sub), q, s))
        _same(python_only, lambda: ops.w4a16_matmul(x.cpu(), q, s))
        _same(python_only, lambda: ops.w4a16_matmul(x, q[:, :8], s))
        _same(python_only, lambda: ops.w4a16_matmul(x, q.float(), s))
        _same(python_only, lambda: ops.w4a16_matmul(torch.empty(3 * 256 + 1, dtype=dtype, device="cuda")[1:].view(3, 256), q, s))  # alignment
        y = torch.empty(3, 264, dtype=x.dtype, device="cuda")
        assert (ops.w4a16_matmul(x, q, s, out=y) is y) if dtype != torch.bfloat16 else True


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_row_and_element_operators(python_only, dtype):
    g = _gen(1)
    x = torch.randn(6, 4, 128, generator=g, device="cuda").to(dtype)
    w = torch.randn(128, generator=g, device="cuda").half()
    pos, freq = torch.arange(6, device="cuda", dtype=torch.int32), torch.rand(128, generator=g, device="cuda")
    flat = x.view(24, 128)
    strided = torch.randn(24, 256, generator=g, device="cuda").to(dtype)[:, ::2]
    for t in (x, flat, strided, flat.cpu(), flat[:0], flat.long(), torch.zeros(24 * 128 + 1, dtype=dtype, device="cuda")[1:].view(24, 128)):
        _same(python_only, lambda: ops.sigmoid(t))
        _same(python_only, lambda: ops.softmax(t))
        _same(python_only, lambda: ops.rmsnorm(t, w))
        _same(python_only, lambda: ops.rmsnorm(t, w, 1))
    _same(python_only, lambda: ops.rope(x, pos, freq))
    _same(python_only, lambda: ops.rope(x, pos.long(), freq))
    _same(python_only, lambda: ops.rope(flat, pos, freq))


@pytest.mark.parametrize("name,dtype", [("f32", torch.float32), ("f16", torch.float16)])
def test_sample_operators(python_only, name, dtype):
    g = _gen(2)
    o = autort.ops
    rms, rot, att = (getattr(o, k + name) for k in ("rmsnorm_", "rotary_", "attention_"))
    x, w = torch.randn(512, generator=g, device="cuda").to(dtype), torch.randn(512, generator=g, device="cuda").to(dtype)
    vs = (x.float() ** 2).sum()
    for v in (vs.view(1), vs, vs.double().view(1), torch.ones(2, device="cuda")):
        for inv in (1 / 512, 1):
            _same(python_only, lambda: rms(x, v, w, extra=[inv]))
    _same(python_only, lambda: rms(x.to(torch.float64), vs, w, extra=[1.0]))
    _same(python_only, lambda: rms(x, vs, w))
    h, freq = torch.randn(4, 2, 64, generator=g, device="cuda").to(dtype), torch.rand(128, generator=g, device="cuda")
    for pos in (0, 37, True, 2.0, 2 ** 31 - 1, 2 ** 40):
        _same(python_only, lambda: rot(h, freq, extra=[pos]))
    _same(python_only, lambda: rot(h.transpose(0, 1), freq, extra=[3]))
    _same(python_only, lambda: rot(h, freq.double(), extra=[3]))
    buf = torch.empty(4, 128, dtype=dtype, device="cuda")
    for on in (False, True):
        python_only(on)
        assert rot(h, freq, buf, extra=[5]) is buf and torch.equal(buf, rot(h, freq, extra=[5]))
    q, kv = torch.randn(4, 128, generator=g, device="cuda").to(dtype), torch.randn(2, 40, 4, 128, generator=g, device="cuda").to(dtype)
    scale = torch.tensor([0.09], device="cuda")
    for k, v in ((kv[0], kv[1]), (kv[0][:1], kv[1][:1]), (kv[0][:0], kv[1][:0]), (kv[0].float().double(), kv[1])):
        for f in (scale, scale.cpu(), scale.double(), scale.view(())):
            _same(python_only, lambda: att(q, k, v, f))
    wide = torch.randn(40, 8, 128, generator=g, device="cuda").to(dtype)
    _same(python_only, lambda: att(q, wide[:, :4], wide[:, 4:], scale))


def test_exported_programs(python_only):
    g = _gen(3)
    mm = autort.export(ir=autort_api.W4A16_IR_SAMPLE, inputs=["input0=float16[S:512]", "qweight=int32[L:64, N:512]", "scales=float16[G:4, N:512]"], name="fast_mm")
    soft = autort.export(ir="t0[N] >=! x[N, C]; t1[N] +=! (x[N, C] - t0[N]).call(`exp`); y[N, C] = (x[N, C] - t0[N]).call(`exp`) / t1[N]",
                         inputs=["x=float16[N:64, C:512]"], name="fast_soft")
    elt = autort.export(ir="z[N, M] = x[N, M] * 2.0 + y[N, M]", inputs=["x=float16[N:64, M:512]", "y=float32[N:64, M:512]"], name="fast_elt")
    rows = autort.export(ir="s[N] +=! x[N, C] * g[C]; y[N, C] = x[N, C] - s[N]", inputs=["x=float16[N:64, C:512]", "g=float16[C:512]"], name="fast_rows")
    q, s = _w4(512, 512, torch.float16, g)
    x = torch.randn(64, 512, generator=g, device="cuda").half()
    for _ in range(2):  # the first call of a shape and the ones after it
        for K, N in ((512, 512), (256, 512), (256, 264), (128, 8), (384, 16), (512, 128), (512, 256), (512, 384), (128, 512), (256, 128)):
            a, b, c = x[0, :K].contiguous(), q[:K // 8, :N], s[:K // 128, :N]
            _same(python_only, lambda: mm(a, b, c))
            _same(python_only, lambda: mm(a, b.contiguous(), c.contiguous()))
        for n, c in ((64, 512), (3, 512), (64, 504), (1, 8), (65, 8)):
            t = x[:n, :c].contiguous() if n <= 64 else torch.zeros(n, c, device="cuda").half()
            _same(python_only, lambda: soft(t))
            _same(python_only, lambda: elt(t, t.float()))
            _same(python_only, lambda: elt(t, t))
            _same(python_only, lambda: elt(t, t.float().t().contiguous().t()))
            _same(python_only, lambda: rows(t, x[0, :c].contiguous()))
            _same(python_only, lambda: rows(t, x[0, :c - 1].contiguous()))
            _same(python_only, lambda: rows(t))
            _same(python_only, lambda: soft(t.cpu()))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        y = mm(x[0], q, s)
    side.synchronize()
    assert torch.equal(y, mm(x[0], q, s))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        z = mm(x[0], q, s)
    z.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(z, y)


def test_exported_operators_of_any_shape(monkeypatch):
    """After the first call, which has the native boundary accept the text, no call of any shape takes the Python route - and what
    that route refuses for its shapes still is refused."""
    seen = []
    forward = autort_api.NativeModules.forward
    monkeypatch.setattr(autort_api.NativeModules, "forward", lambda self, t, *a: seen.append([tuple(x.shape) for x in t]) or forward(self, t, *a))
    g = _gen(4)
    mm = autort.export(ir=autort_api.W4A16_IR_SAMPLE, inputs=["input0=float16[M:40, S:512]", "qweight=int32[L:64, N:512]", "scales=float16[G:8, N:512]"], name="any_mm")
    sig = autort.export(ir="y[N] = 1 - 1 / (1 + x[N].call(strs.exp))", inputs=["x=float32[N:4096]"], name="any_sig")
    soft = autort.export(ir="t0[N] >=! x[N, C]; t1[N] +=! (x[N, C] - t0[N]).call(`exp`); y[N, C] = (x[N, C] - t0[N]).call(`exp`) / t1[N]",
                         inputs=["x=float32[N:64, C:512]"], name="any_soft")
    for _ in range(2):
        for i in range(20):
            K, N, M = 128 * (1 + i % 4), 8 * (3 * i + 1), 1 + 2 * i
            q, s = _w4(K, N, torch.float16, g)
            x = torch.randn(M, K, generator=g, device="cuda").half()
            assert torch.equal(mm(x, q, s), ops.w4a16_matmul(x, q, s))
            v = torch.randn(100 * i + 1, generator=g, device="cuda")
            assert torch.equal(sig(v), ops.sigmoid(v))
            v = torch.randn(i + 1, 8 * (i + 1), generator=g, device="cuda")
            assert torch.equal(soft(v), ops.softmax(v))
    assert len(seen) == 3  # one first call each
    # groups of 64 where the text says 128: the same refusal through either route
    q, s = _w4(512, 512, torch.float16, g)
    x, s64 = torch.randn(2, 512, generator=g, device="cuda").half(), s.repeat(2, 1)
    assert s64.shape == (8, 512)
    with pytest.raises(Exception, match="W4A16 shapes disagree"):
        mm(x, q, s64)
    with pytest.raises(Exception):
        mm(x[:, :384].contiguous(), q, s)
