"""The interpreter kernels against numpy: program shapes (which side of an operation is compound, how deep the
stack gets), ragged sizes, alignments and in-place results."""
import numpy as np
import pytest
import torch

import autort
from antares_b200 import ir, ops
from vm_ref import eval_program_numpy, eval_row_program_numpy

pytestmark = pytest.mark.gpu

EXPRESSIONS = [
    "x[N]", "-x[N]", "2.0", "x[N] - y[N]", "1.5 - x[N]", "x[N] / (1.5 + y[N] * y[N])", "(x[N] + 1.0) / (y[N] * y[N] + 2.0)",
    "(x[N] - y[N]) - (y[N] - 3.0)", "(x[N] + y[N]) * ((x[N] - y[N]) / ((x[N] * x[N] + 1.0) - (0.5 - (y[N] * y[N] + 2.0) * (x[N] - 1.0))))",
    "x[N].call(`max`, [y[N] - 0.25])", "(x[N] * 0.1).call(`exp`) - (0.5 - y[N].call(`tanh`)) * (x[N] - (y[N] + x[N] * (y[N] - 2.0)))",
    "2.0 / ((x[N] - y[N]).call(`abs`) + 1.0)", "(2.0).call(`pow`, [x[N]])",
]


@pytest.mark.parametrize("expr", EXPRESSIONS)
@pytest.mark.parametrize("n", [1, 7, 8, 1023, 1024, 1025, 100003])
def test_elementwise_program_shapes(expr, n):
    if "[N]" not in expr:
        expr = "x[N] * 0.0 + " + expr
    _, _, used, prog, consts = ir.compile_elementwise("z[N] = " + expr, ["x", "y"])
    rng = np.random.default_rng(n)
    host = {"x": rng.standard_normal(n + 1).astype(np.float32), "y": rng.standard_normal(n + 1).astype(np.float16)}
    for off in (0, 1):  # 1: pointers that are not 16-byte aligned
        arrays = [host[u][off:off + n] for u in used]
        ins = [torch.from_numpy(host[u]).cuda()[off:off + n] for u in used]
        want = np.broadcast_to(eval_program_numpy(prog, consts, arrays), (n,))
        got = ops.eltwise_program(prog, consts, ins, out_dtype=torch.float32).cpu().numpy()
        # up to 12 operations of 2 ulp each on values that may cancel: 24 * 2^-24 of the largest intermediate (< 64)
        np.testing.assert_allclose(got, want, rtol=4e-6, atol=24 * 2 ** -24 * 8)
    x = torch.from_numpy(host["x"][:n]).cuda()
    if used == ["x"]:
        want = ops.eltwise_program(prog, consts, [x])
        assert torch.equal(ops.eltwise_program(prog, consts, [x], out=x), want)  # in place


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 7), (5, 255), (2, 256), (4, 264), (3, 2047), (2, 2048), (3, 2056), (2, 4200), (3000, 33), (2072, 33), (2073, 33), (4100, 32), (1036, 128), (1037, 127), (518, 256), (519, 256)])
@pytest.mark.parametrize("dtype", ["float16", "float32"])
def test_row_programs_at_odd_sizes(rows, cols, dtype):
    text = "m[N] >=! x[N, C]; k[N] <=! x[N, C] * g[C]; s[N] +=! (x[N, C] - m[N]).call(`exp`) * (g[C] + (x[N, C] - k[N]) / (2.0 + g[C])); " \
           "o[N, C] = (x[N, C] - m[N]) / (s[N] + C.val()) + (k[N] - g[C]) * (x[N, C] - w[N, C])"
    dt = getattr(torch, dtype)
    fn = autort.export(ir=text, inputs=["x=%s[N:4200, C:4200]" % dtype, "w=%s[N:4200, C:4200]" % dtype, "g=%s[C:4200]" % dtype], name="rows_" + dtype)
    g = torch.Generator(device="cuda").manual_seed(rows * cols)
    x, w = (torch.randn(rows, cols, generator=g, device="cuda").to(dt) for _ in range(2))
    c = torch.randn(cols, generator=g, device="cuda").abs().to(dt)
    rp = fn.match.params
    by_name = {"x": x, "w": w, "g": c}
    want = eval_row_program_numpy(rp, [by_name[n].cpu().numpy() for n in rp["mats"]], [by_name[n].cpu().numpy() for n in rp["cols"]])
    got = fn(x, w, c).float().cpu().numpy()
    # fp32 sums of up to 4200 terms in another order, then one rounding to the result's type
    tol = 2 ** -11 + 2e-5 if dtype == "float16" else 2e-5
    np.testing.assert_allclose(got, want, rtol=tol, atol=tol * max(1e-3, np.abs(want).max()))
    flat = torch.zeros(rows * cols + 1, dtype=dt, device="cuda")[1:].view(rows, cols)  # unaligned input
    flat.copy_(x)
    np.testing.assert_allclose(fn(flat, w, c).float().cpu().numpy(), want, rtol=tol, atol=tol * max(1e-3, np.abs(want).max()))


@pytest.mark.parametrize("depth", [3, 5, 6])
@pytest.mark.parametrize("cols", [1000, 1025, 2050])
def test_row_programs_with_deep_expressions(depth, cols):
    """The operand stack is shared memory, up to 48 KiB of it in the widest block."""
    expr = "x[N, C] + %d.0" % (depth + 1)
    for i in range(depth, 0, -1):
        expr = "(x[N, C] + %d.0) * (%s)" % (i, expr)
    text = "s[N] +=! x[N, C]; y[N, C] = %s - s[N]" % expr
    fn = autort.export(ir=text, inputs=["x=float32[N:8, C:4096]"], name="deep_%d" % depth)
    x = torch.randn(3, cols, generator=torch.Generator(device="cuda").manual_seed(cols), device="cuda")
    rp = fn.match.params
    want = eval_row_program_numpy(rp, [x.cpu().numpy()], [])
    # sums of up to 2050 terms in another order, products of up to 7 factors of 2^-24 each
    np.testing.assert_allclose(fn(x).cpu().numpy(), want, rtol=2e-5, atol=2e-5 * np.abs(want).max())
