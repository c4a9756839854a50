"""What this framework is timed on: the work its users have it do, through its public entry points.

  listed()         the cases, from one exported operator call to a 2000-token prompt through the 7B model
  draw(rng)        one more case of the same kinds and ranges
  prepare(case, s) what a user's program holds before the call: weights in the checkpoint's layout, the exported
                   operators, the loaded decoder, and this call's inputs (from the seed s)
  run(state)       one pass; returns the path's outputs
  work(case)       bytes and operations one pass cannot do without
  tolerance(case)  how far another correct implementation of the same precision may be off
  exact(case, s)   what run() returns for the inputs of seed s, in plain torch and 64 bits

The model is the framework's own benchmark model, Llama-2-7B's architecture with int4 linears (group 128), random
weights: zero-mean nibbles and scales that keep activations in range, as a trained checkpoint has them.
"""
import math

import numpy as np
import torch

import autort
from antares_b200 import autort_api, ops
from antares_b200.llama import LlamaConfig, LlamaInt4Decoder, make_inv_freq, synth_prompt

DIM, FFN, HEADS, HEAD, VOCAB, GROUP = 4096, 11008, 32, 128, 32000, 128
# the decode projections of the 7B model, (K, N): V|Q|K, O, gate|up, down
PROJECTIONS = {"vqk": (DIM, 3 * DIM), "o": (DIM, DIM), "gate_up": (DIM, 2 * FFN), "down": (FFN, DIM)}
CACHE_ROWS = 256      # cache rows of the operator-by-operator sample
MAX_SEQ = 2304        # cache rows of the loaded decoder

LAYERNORM_IR = ("s[N] +=! x[N, C]; q[N] +=! x[N, C] * x[N, C]; "
                "y[N, C] = (x[N, C] - s[N] / C.val()) * (q[N] / C.val() - s[N] / C.val() * s[N] / C.val() + 1e-5).call(`rsqrt`) * g[C] + b[C]")
GELU_IR = "z[N] = 0.5 * y[N] * (1.0 + (0.7978845608 * (y[N] + 0.044715 * y[N] * y[N] * y[N])).call(`tanh`))"
SOFTMAX_IR = ("t0[N] >=! x[N, C]; t1[N] +=! (x[N, C] - t0[N]).call(`exp`); y[N, C] = (x[N, C] - t0[N]).call(`exp`) / t1[N]")
SIGMOID_IR = "y[N] = 1 - 1 / (1 + x[N].call(strs.exp))"


def listed():
    return [
        # one exported W4A16 operator call on one activation row: the smallest thing a caller of autort.ops does
        {"name": "export_f16_4096x4096", "kind": "export", "K": DIM, "N": DIM, "dtype": "float16"},
        # one decode step's four projections, one request
        {"name": "projections_m1", "kind": "projections", "M": 1},
        # the same for a few requests decoded together (an odd number of them), and for a full decode batch
        {"name": "projections_m6", "kind": "projections", "M": 6},
        {"name": "projections_m16", "kind": "projections", "M": 16},
        # a prompt's projection on the tensor cores
        {"name": "gemm_2048x4096x11008", "kind": "gemm", "M": 2048, "K": DIM, "N": FFN},
        # the int4 sample's own program: one decoder layer operator by operator, float32 activations and scales
        {"name": "sample_layer_f32", "kind": "sample_layer", "dtype": "float32", "pos": 37},
        # the element-wise and reduction operators at their benchmark shapes
        {"name": "elementwise_2048", "kind": "elementwise", "rows": 2048, "n": 4096000, "soft_rows": 32, "soft_cols": 4096},
        # operators a user writes as IR text: layernorm with weight and bias, then tanh-GELU
        {"name": "custom_ir_2048x4096", "kind": "custom_ir", "rows": 2048, "cols": 4096, "dtype": "float16"},
        # a request of the benchmark's size: 128 prompt tokens in one pass, then decode steps
        {"name": "chat_128_32", "kind": "chat", "layers": 32, "prompt": 128, "steps": 32, "page_rows": 0},
        # a longer context on a paged cache, odd sizes, a quarter of the depth
        {"name": "chat_paged_451_24", "kind": "chat", "layers": 8, "prompt": 451, "steps": 24, "page_rows": 16},
        # time to the first token: the benchmark's prompt, and a long ragged one
        {"name": "prefill_128", "kind": "prefill", "layers": 32, "prompt": 128, "page_rows": 0},
        {"name": "prefill_2000", "kind": "prefill", "layers": 32, "prompt": 2000, "page_rows": 0},
    ]


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["export", "projections", "projections", "gemm", "sample_layer", "elementwise", "custom_ir", "chat", "chat", "prefill", "prefill"])
    if kind == "export":
        return {"kind": kind, "K": GROUP * _log_int(rng, 8, FFN // GROUP), "N": 8 * _log_int(rng, 128, 2 * FFN // 8), "dtype": rng.choice(["float16", "float32"])}
    if kind == "projections":
        return {"kind": kind, "M": _log_int(rng, 1, 16), "of": ",".join(sorted(rng.sample(sorted(PROJECTIONS), rng.randrange(1, 4))))}
    if kind == "gemm":
        K, N = rng.choice(sorted(PROJECTIONS.values()))
        return {"kind": kind, "M": _log_int(rng, 17, 2048), "K": K, "N": N}
    if kind == "sample_layer":
        return {"kind": kind, "dtype": rng.choice(["float32", "float16"]), "pos": rng.randrange(CACHE_ROWS)}
    if kind == "elementwise":
        return {"kind": kind, "rows": _log_int(rng, 1, 4096), "n": _log_int(rng, 1000, 8192000), "soft_rows": _log_int(rng, 1, 2048),
                "soft_cols": 8 * _log_int(rng, 16, 1024)}
    if kind == "custom_ir":
        return {"kind": kind, "rows": _log_int(rng, 16, 4096), "cols": _log_int(rng, 256, 4200), "dtype": rng.choice(["float16", "float32"])}
    if kind == "chat":
        return {"kind": kind, "layers": 32, "prompt": _log_int(rng, 1, 1024), "steps": rng.randrange(4, 33), "page_rows": 0} if rng.random() < 0.6 else \
            {"kind": kind, "layers": 8, "prompt": _log_int(rng, 1, 1024), "steps": rng.randrange(4, 33), "page_rows": 16}
    return {"kind": kind, "layers": 32, "prompt": _log_int(rng, 2, 2000), "page_rows": 0}


def _projections(case):
    return [shape for name, shape in PROJECTIONS.items() if name in case.get("of", ",".join(PROJECTIONS)).split(",")]


# ---- inputs ------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.float16):
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


def _weights(g, K, N, dtype=torch.float16, scale_mul=1.0, centered=False):
    """Packed nibbles int32 [K/8, N] and scales [K/128, N] in the checkpoint's layout; nibbles uniform in 0..15
    (centered: every 0 becomes an 8, so q - 8 has zero mean), scales uniform in [0.001, 0.02] times scale_mul."""
    q = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device="cuda", dtype=torch.int32)
    if centered:
        for j in range(8):
            q |= (((q >> (4 * j)) & 15) == 0).to(torch.int32) << (4 * j + 3)
    s = ((torch.rand(K // GROUP, N, generator=g, device="cuda") * 0.019 + 0.001) * scale_mul).to(dtype)
    return q, s


class _Checkpoint:
    """The loaded model's weights, as LlamaInt4Decoder(weights=...) wants them: host arrays, layer by layer."""

    def __init__(self, cfg):
        self.cfg = cfg

    def layer(self, l):
        g = _gen(7000 + l)
        w = {}
        for key, K, N in (("vqk", DIM, 3 * DIM), ("o", DIM, DIM), ("gate", DIM, FFN), ("up", DIM, FFN), ("down", FFN, DIM)):
            q, s = _weights(g, K, N, scale_mul=0.25, centered=True)
            w[key + "_q"], w[key + "_s"] = q.cpu().numpy(), s.cpu().numpy()
        for key in ("att_norm", "ffn_norm"):
            w[key] = (1 + 0.1 * _randn(g, DIM, dtype=torch.float32)).half().cpu().numpy()
        return w

    def globals(self):
        g = _gen(6999)
        table = lambda: (0.02 * _randn(g, VOCAB, DIM, dtype=torch.float32)).half().cpu().numpy()  # noqa: E731
        return {"embed": table(), "lm_head": table(), "final_norm": (1 + 0.1 * _randn(g, DIM, dtype=torch.float32)).half().cpu().numpy()}


_loaded = {}


def _decoder(layers, page_rows):
    """A serving program loads the model once and keeps it: one decoder per depth and cache kind."""
    key = (layers, page_rows)
    if key not in _loaded:
        cfg = LlamaConfig(n_layers=layers, max_seq=MAX_SEQ)
        dec = LlamaInt4Decoder(cfg, torch.device("cuda:0"), max_tokens=MAX_SEQ, weights=_Checkpoint(cfg), kv_page_rows=page_rows)
        dec.capture(1)
        _loaded[key] = dec
    return _loaded[key]


def _w4_export(dtype, rows=0):
    x = "input0=%s[%sS:%d]" % (dtype, "M:%d, " % rows if rows else "", FFN)
    return autort.export(ir=autort_api.W4A16_IR_SAMPLE, inputs=[x, "qweight=int32[L:%d, N:%d]" % (FFN // 8, 2 * FFN), "scales=%s[G:%d, N:%d]" % (dtype, FFN // GROUP, 2 * FFN)],
                         config="~N~:[256,8,32],~S~:[64,8]", name="matmul_dequat_" + dtype)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "export":
        dt = getattr(torch, case["dtype"])
        st["op"] = _w4_export(case["dtype"])
        st["x"] = _randn(g, case["K"], dtype=dt)
        st["q"], st["s"] = _weights(g, case["K"], case["N"], dt)
    elif kind == "projections":
        st["calls"] = [(_randn(g, case["M"], K),) + _weights(g, K, N) for K, N in _projections(case)]
    elif kind == "gemm":
        st["calls"] = [(_randn(g, case["M"], case["K"]),) + _weights(g, case["K"], case["N"])]
    elif kind == "sample_layer":
        dt = getattr(torch, case["dtype"])
        st.update(dtype=case["dtype"], pos=case["pos"], mm=_w4_export(case["dtype"]), x=_randn(g, DIM, dtype=dt),
                  kc=_randn(g, CACHE_ROWS, DIM, dtype=dt), vc=_randn(g, CACHE_ROWS, DIM, dtype=dt),
                  att_norm=(1 + 0.1 * _randn(g, DIM, dtype=torch.float32)).to(dt), ffn_norm=(1 + 0.1 * _randn(g, DIM, dtype=torch.float32)).to(dt),
                  inv_freq=torch.from_numpy(make_inv_freq(HEAD, 10000.0)).cuda(), att_f=torch.tensor([1 / math.sqrt(HEAD)], device="cuda"))
        for key, K, N in (("vqk", DIM, 3 * DIM), ("o", DIM, DIM), ("gate", DIM, FFN), ("up", DIM, FFN), ("down", FFN, DIM)):
            st[key] = _weights(g, K, N, dt, scale_mul=0.25, centered=True)
    elif kind == "elementwise":
        rows = case["rows"]
        st.update(sigmoid=autort.export(ir=SIGMOID_IR, inputs=["x=float32[N:8192000]"], name="sigmoid_f32"),
                  softmax=autort.export(ir=SOFTMAX_IR, inputs=["x=float16[N:2048, C:8192]"], name="softmax_f16"),
                  data=_randn(g, case["n"], dtype=torch.float32), hidden=_randn(g, rows, DIM),
                  weight=(1 + 0.1 * _randn(g, DIM, dtype=torch.float32)).half(), heads=_randn(g, rows, HEADS, HEAD),
                  pos=torch.arange(rows, device="cuda", dtype=torch.int32), inv_freq=torch.from_numpy(make_inv_freq(HEAD, 10000.0)).cuda(),
                  scores=3 * _randn(g, case["soft_rows"], case["soft_cols"]))
    elif kind == "custom_ir":
        dt, cols = case["dtype"], case["cols"]
        tdt = getattr(torch, dt)
        st.update(norm=autort.export(ir=LAYERNORM_IR, inputs=["x=%s[N:4096, C:4200]" % dt, "g=%s[C:4200]" % dt, "b=%s[C:4200]" % dt], name="layernorm_" + dt),
                  gelu=autort.export(ir=GELU_IR, inputs=["y=%s[N:17203200]" % dt], name="gelu_" + dt),
                  x=_randn(g, case["rows"], cols, dtype=torch.float32).mul_(2).add_(0.5).to(tdt),
                  g=(1 + 0.1 * _randn(g, cols, dtype=torch.float32)).to(tdt), b=(0.1 * _randn(g, cols, dtype=torch.float32)).to(tdt))
    else:
        dec = _decoder(case["layers"], case["page_rows"])
        toks = synth_prompt(dec.cfg, case["prompt"] + case.get("steps", 0), int(seed))
        st.update(dec=dec, prompt=toks[:case["prompt"]], forced=[int(t) for t in toks[case["prompt"]:]], rows=len(toks))
    return st


# ---- one pass ----------------------------------------------------------------------------------------------

def _sample_layer(st):
    """One decoder layer as the int4 sample chains it: fused V|Q|K, rotary into the cache, attention, O, SwiGLU."""
    o = autort.ops
    f32 = st["dtype"] == "float32"
    rms, rot, att = (o.rmsnorm_f32, o.rotary_f32, o.attention_f32) if f32 else (o.rmsnorm_f16, o.rotary_f16, o.attention_f16)
    x, pos, mm = st["x"], st["pos"], st["mm"]
    norm = lambda v, w: rms(v, (v.float() * v.float()).sum().view(1), w, extra=[1.0 / DIM])  # noqa: E731
    vqk = mm(norm(x, st["att_norm"]), *st["vqk"])
    v, q, k = vqk[:DIM], vqk[DIM:2 * DIM], vqk[2 * DIM:]
    q_rot = torch.empty(HEADS, HEAD, dtype=x.dtype, device=x.device)
    rot(q.view(HEADS, 2, -1), st["inv_freq"], q_rot, extra=[pos])
    rot(k.view(HEADS, 2, -1), st["inv_freq"], st["kc"][pos].view(HEADS, HEAD), extra=[pos])
    st["vc"][pos].copy_(v)
    kc, vc = (st[c].view(CACHE_ROWS, HEADS, HEAD).narrow(0, 0, pos + 1) for c in ("kc", "vc"))
    x = x + mm(att(q_rot, kc, vc, st["att_f"]).view(DIM), *st["o"])
    h = norm(x, st["ffn_norm"])
    h = torch.nn.functional.silu(mm(h, *st["gate"])) * mm(h, *st["up"])
    return [x + mm(h, *st["down"]), st["kc"], st["vc"]]


def run(st):
    kind = st["kind"]
    if kind == "export":
        return st["op"](st["x"], st["q"], st["s"])
    if kind in ("projections", "gemm"):
        return [ops.w4a16_matmul(x, q, s) for x, q, s in st["calls"]]
    if kind == "sample_layer":
        return _sample_layer(st)
    if kind == "elementwise":
        return [st["sigmoid"](st["data"]), ops.rmsnorm(st["hidden"], st["weight"]), ops.rope(st["heads"], st["pos"], st["inv_freq"]), st["softmax"](st["scores"])]
    if kind == "custom_ir":
        y = st["norm"](st["x"], st["g"], st["b"])
        return [y, st["gelu"](y.view(-1))]
    # the decoder: the prompt in one pass, then one call per token with the caller's token ids; the logits after the
    # prompt and after the last step, and the cache rows written
    dec = st["dec"]
    dec.prefill(st["prompt"])
    out = {"k_cache": dec.k_cache[:, :st["rows"]], "v_cache": dec.v_cache[:, :st["rows"]]}
    if kind == "chat":
        out["first_logits"] = dec.logits.clone()
        for t in st["forced"]:
            dec.step(t)
    out["logits"] = dec.logits
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------

def _linear(M, K, N, elt=2):
    return {"bytes": K * N / 2 + (K // GROUP) * N * elt + M * K * elt + M * N * elt, "flops": 2.0 * M * K * N}


def _sum(parts):
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def _forward(layers, tokens, context):
    """`tokens` tokens through the model at once, the last of them at position context - 1; logits of the last one."""
    before = context - tokens
    attended = tokens * before + tokens * (tokens + 1) / 2
    # activations need not leave the chip inside a pass: the weights and the cache rows have to move, the embeddings come in
    layer = {"bytes": sum(K * N / 2 + (K // GROUP) * N * 2 for K, N in PROJECTIONS.values()) + 2 * context * DIM * 2,
             "flops": sum(2.0 * tokens * K * N for K, N in PROJECTIONS.values()) + 4.0 * attended * DIM}
    return {"bytes": layers * layer["bytes"] + VOCAB * DIM * 2 + tokens * DIM * 2, "flops": layers * layer["flops"] + 2.0 * VOCAB * DIM}


def work(case):
    kind = case["kind"]
    if kind == "export":
        return _linear(1, case["K"], case["N"], 4 if case["dtype"] == "float32" else 2)
    if kind == "projections":
        return _sum([_linear(case["M"], K, N) for K, N in _projections(case)])
    if kind == "gemm":
        return _linear(case["M"], case["K"], case["N"])
    if kind == "sample_layer":
        e = 4 if case["dtype"] == "float32" else 2
        return _sum([_linear(1, K, N, e) for K, N in PROJECTIONS.values()] + [{"bytes": 2 * (case["pos"] + 1) * DIM * e, "flops": 4.0 * (case["pos"] + 1) * DIM}])
    if kind == "elementwise":
        r = case["rows"] * DIM * 2
        return {"bytes": float(8 * case["n"] + 4 * r + 4 * case["soft_rows"] * case["soft_cols"]), "flops": float(4 * case["n"] + 5 * r + 4 * case["soft_rows"] * case["soft_cols"])}
    if kind == "custom_ir":
        n, e = case["rows"] * case["cols"], 4 if case["dtype"] == "float32" else 2
        return {"bytes": float(4 * n * e), "flops": 20.0 * n}
    parts = [_forward(case["layers"], case["prompt"], case["prompt"])]
    parts += [_forward(case["layers"], 1, case["prompt"] + 1 + i) for i in range(case.get("steps", 0))]
    return _sum(parts)


def tolerance(case):
    # About four times what two correct implementations of the same precision were seen to differ by.  One fp16 row: 1.2e-3
    # off a 64-bit sum (products chained in fp16); several rows: 2.8e-4 (the group scale factored out of the sum, or
    # multiplied into the weight and rounded).  float32: 3e-7.  The decoder: 7e-3 to 8e-3 between the prompt in one pass and
    # token by token, and between two projection kernels: 32 layers multiply each rounding.
    kind = case["kind"]
    f32 = case.get("dtype") == "float32"
    if kind in ("export", "projections", "gemm"):
        return {"rel": 2e-6, "max": 2e-5} if f32 else {"rel": 4e-3, "max": 2e-2} if case.get("M", 1) == 1 else {"rel": 1.1e-3, "max": 5e-3}
    if kind == "sample_layer":
        return {"rel": 2e-6, "max": 2e-5} if f32 else {"rel": 5e-3, "max": 2e-2}
    if kind == "elementwise":
        return {"rel": 8e-4, "max": 3e-3}
    if kind == "custom_ir":
        return {"rel": 2e-6, "max": 2e-5} if f32 else {"rel": 8e-4, "max": 3e-3}
    return {"rel": 0.03, "max": 0.2}


# ---- the same results in 64 bits ---------------------------------------------------------------------------

def _dequant(q, s):
    """Weights [K, N] in 64 bits from packed nibbles [K/8, N] and group scales [K/128, N], nothing rounded on the way."""
    w = torch.stack([((q >> (4 * j)) & 15) - 8 for j in range(8)], dim=1).view(-1, q.shape[1]).double()
    return w.view(s.shape[0], GROUP, -1).mul_(s.double()[:, None]).view(w.shape)


def _rms64(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.double()


def _rope64(x, pos, inv_freq):
    """x [T, H, D] rotated by halves at the positions pos [T]; angles as float32 products, which is what defines them."""
    ang = (pos.float()[:, None] * inv_freq[None]).double()[:, None]
    half = x.shape[-1] // 2
    return x * ang.cos() + torch.cat([-x[..., half:], x[..., :half]], -1) * ang.sin()


def _attend64(q, k, v, first):
    """Rows of q [T, H, D] at positions first, first + 1, ... over the cache rows k, v [S, H, D] up to their own."""
    later = torch.arange(k.shape[0], device="cuda")[None] > torch.arange(first, first + q.shape[0], device="cuda")[:, None]
    heads = []
    for h in range(q.shape[1]):
        heads.append(torch.softmax((q[:, h] @ k[:, h].T / math.sqrt(q.shape[2])).masked_fill_(later, -math.inf), -1) @ v[:, h])
    return torch.stack(heads, 1)


def _model64(case, seed):
    cfg = LlamaConfig(n_layers=case["layers"], max_seq=MAX_SEQ)
    ckpt, n = _Checkpoint(cfg), case["prompt"]
    toks = torch.from_numpy(synth_prompt(cfg, n + case.get("steps", 0), int(seed))).cuda().long()
    inv_freq, pos = torch.from_numpy(make_inv_freq(HEAD, 10000.0)).cuda(), torch.arange(len(toks), device="cuda")
    on = lambda w, *keys: [torch.from_numpy(w[k]).cuda() for k in keys]  # noqa: E731
    embed, head, final = on(ckpt.globals(), "embed", "lm_head", "final_norm")
    x, ks, vs = embed[toks].double(), [], []
    for l in range(case["layers"]):
        w = ckpt.layer(l)
        mm = lambda a, key: a @ _dequant(*on(w, key + "_q", key + "_s"))  # noqa: E731
        v, q, k = mm(_rms64(x, *on(w, "att_norm")), "vqk").view(-1, 3, HEADS, HEAD).unbind(1)
        q, k = _rope64(q, pos, inv_freq), _rope64(k, pos, inv_freq)
        x = x + mm(_attend64(q, k, v, 0).reshape(-1, DIM), "o")
        ks.append(k.reshape(-1, DIM))
        vs.append(v.reshape(-1, DIM))
        h = _rms64(x, *on(w, "ffn_norm"))
        x = x + mm(torch.nn.functional.silu(mm(h, "gate")) * mm(h, "up"), "down")
    logits = lambda row: _rms64(row, final) @ head.double().T  # noqa: E731
    out = {"k_cache": torch.stack(ks), "v_cache": torch.stack(vs)}
    if case["kind"] == "chat":
        out["first_logits"] = logits(x[n - 1])
    out["logits"] = logits(x[-1])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("chat", "prefill"):
        return _model64(case, seed)
    st = prepare(case, seed)
    if kind == "export":
        return st["x"].double() @ _dequant(st["q"], st["s"])
    if kind in ("projections", "gemm"):
        return [x.double() @ _dequant(q, s) for x, q, s in st["calls"]]
    if kind == "sample_layer":
        at, x, pos = torch.tensor([st["pos"]], device="cuda"), st["x"].double(), st["pos"]
        v, q, k = (_rms64(x, st["att_norm"]) @ _dequant(*st["vqk"])).view(3, 1, HEADS, HEAD)
        kc, vc = st["kc"].double(), st["vc"].double()
        q, kc[pos], vc[pos] = _rope64(q, at, st["inv_freq"]), _rope64(k, at, st["inv_freq"]).view(DIM), v.view(DIM)
        cache = [c[:pos + 1].view(-1, HEADS, HEAD) for c in (kc, vc)]
        x = x + _attend64(q, *cache, pos).view(DIM) @ _dequant(*st["o"])
        h = _rms64(x, st["ffn_norm"])
        return [x + (torch.nn.functional.silu(h @ _dequant(*st["gate"])) * (h @ _dequant(*st["up"]))) @ _dequant(*st["down"]), kc, vc]
    if kind == "elementwise":
        return [torch.sigmoid(st["data"].double()), _rms64(st["hidden"].double(), st["weight"]),
                _rope64(st["heads"].double(), st["pos"], st["inv_freq"]), torch.softmax(st["scores"].double(), -1)]
    y = torch.nn.functional.layer_norm(st["x"].double(), (case["cols"],), st["g"].double(), st["b"].double(), 1e-5)
    return [y, torch.nn.functional.gelu(y.view(-1), approximate="tanh")]
