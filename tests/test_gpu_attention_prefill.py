"""Causal attention of a prompt's rows over the cache against the same softmax in 64 bits."""
import math

import numpy as np
import pytest
import torch

from antares_b200._lib import call
from antares_b200 import ops

pytestmark = pytest.mark.gpu
H, D = 48, 128  # with 48 heads the tensor-core kernel takes over at 40 rows


def _run(q, k, v, pos0, scale, table=None, page_rows=0, max_seq=None, in_place=False):
    rows, max_seq = q.shape[0], max_seq or k.shape[0]
    q = q.clone() if in_place else q
    out = q if in_place else torch.full_like(q, 7.0)
    pos = torch.tensor([pos0], dtype=torch.int32, device="cuda")
    args = [q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), pos.data_ptr(), rows, max_seq, H, D, k.stride(0), scale]
    if table is None:
        call("ab200_attention_prefill", *args, torch.cuda.current_stream().cuda_stream)
    else:
        call("ab200_attention_prefill_paged", *args, table.data_ptr(), page_rows, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    return out


def _expected(q, k, v, pos0, scale):
    q, k, v = q.double(), k.double().view(-1, H, D), v.double().view(-1, H, D)
    out = torch.zeros_like(q)
    for r in range(q.shape[0]):
        S = max(0, min(pos0 + 1 + r, k.shape[0]))
        if S:
            p = torch.softmax(torch.einsum("hd,shd->hs", q[r], k[:S]) * scale, -1)
            out[r] = torch.einsum("hs,shd->hd", p, v[:S])
    return out


def _inputs(rows, max_seq, seed, sharp=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    return (sharp * mk(rows, H, D)).half(), mk(max_seq, H * D).half(), mk(max_seq, H * D).half()


def _close(got, want, v, score=0.0):
    # half an fp16 step of the result, and fp32 sums of at most 2048 products of p <= 1 with v, weighted by sum p = 1; a score
    # of size `score` is an fp32 sum of 128 products, off by up to 2^-21 of it, which p carries on to 2 max|v|
    bound = want.abs() * 2 ** -11 * 1.01 + (2 ** -20 + 2 ** -20 * score) * v.abs().max().double() + 2 ** -25
    assert bool(((got.double() - want).abs() <= bound).all()), float(((got.double() - want).abs() / bound).max())


# edges of the query tile (128) and the key tile (64), both sides of the row rule (39 / 40), one row, prompts behind a filled cache
@pytest.mark.parametrize("rows,pos0,max_seq", [(1, 0, 64), (8, 3, 64), (16, 0, 16), (39, 0, 64), (40, 0, 64), (41, 0, 64), (41, 22, 63), (41, 900, 941), (63, 0, 64), (64, 1, 65), (65, 0, 80), (127, 0, 200),
                                               (128, 0, 128), (129, 0, 129), (200, 300, 512), (451, 0, 451), (30, 1000, 1030)])
@pytest.mark.parametrize("sharp", [1.0, 24.0])  # 24: scores spread over hundreds, the running maximum moves often
def test_prefill_attention(rows, pos0, max_seq, sharp):
    q, k, v = _inputs(rows, max_seq, rows + pos0, sharp)
    scale = 1 / math.sqrt(D)
    want = _expected(q, k, v, pos0, scale)
    score = float(torch.einsum("rhd,shd->rhs", q.double(), k.double().view(-1, H, D)).abs().max()) * scale
    _close(_run(q, k, v, pos0, scale), want, v, score)
    page = 4
    n = (max_seq + page - 1) // page
    table = torch.from_numpy(np.random.default_rng(1).permutation(n).astype(np.int32)).cuda()
    kp, vp = torch.full((n * page, H * D), math.nan, device="cuda").half(), torch.full((n * page, H * D), math.nan, device="cuda").half()
    s = torch.arange(max_seq, device="cuda")
    phys = table[s // page].long() * page + s % page
    kp[phys], vp[phys] = k, v
    _close(_run(q, kp, vp, pos0, scale, table, page, max_seq), want, v, score)


@pytest.mark.parametrize("rows", [5, 70, 200])
def test_rows_beyond_the_cache_and_below_it(rows):
    """Rows at negative positions attend to nothing (0), rows past the cache's end to all of it."""
    q, k, v = _inputs(rows, 48, rows)
    for pos0 in (-3, 20):
        got, want = _run(q, k, v, pos0, 0.1), _expected(q, k, v, pos0, 0.1)
        _close(got, want, v)
    assert not _run(q, k, v, -rows, 0.1).any()


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("at", [0, 5, 63, 100, 130])
def test_values_that_are_not_finite_reach_only_the_rows_that_attend(value, at):
    """A key's V row reaches the query rows from its own position on, cache rows never written reach none."""
    rows = 140
    q, k, v = _inputs(rows, 256, at)
    k[rows:], v[rows:] = math.nan, math.nan
    v[at, D + 3] = value
    got, want = _run(q, k, v, 0, 0.09), _expected(q, k, v, 0, 0.09)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    fine = want.isfinite()
    _close(got[fine], want[fine], v[:rows][v[:rows].isfinite()])
    assert torch.equal(fine[:at], torch.ones_like(fine[:at]))


@pytest.mark.parametrize("rows", [5, 70, 300])
@pytest.mark.parametrize("value", [1.0, math.inf, math.nan])
def test_result_over_the_queries(rows, value):
    """`out` may be `q`: a row's query is read before its result is stored, whichever code computes it."""
    q, k, v = _inputs(rows, 320, rows)
    v[3, 5] = value
    got = _run(q, k, v, 0, 0.09, in_place=True)
    want = _run(q, k, v, 0, 0.09)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~got.isnan()], want[~want.isnan()])
    _close(got[want.isfinite()], _expected(q, k, v, 0, 0.09)[want.isfinite()], v[:rows][v[:rows].isfinite()])
    # the page table form, and every row in a tile whose values are not finite
    table = torch.arange(80, device="cuda", dtype=torch.int32)
    paged = _run(q, k, v, 0, 0.09, table, 4, 320, in_place=True)
    assert torch.equal(paged.isnan(), want.isnan()) and torch.equal(paged[~want.isnan()], want[~want.isnan()])


@pytest.mark.parametrize("heads,rows", [(1, 406), (1, 407), (2, 279), (2, 280), (8, 127), (8, 128), (32, 52), (32, 53)])
def test_both_sides_of_the_rule(monkeypatch, heads, rows):
    """Which kernel serves a prompt depends on heads and rows; the result does not."""
    monkeypatch.setitem(globals(), "H", heads)
    q, k, v = _inputs(rows, rows + 7, heads)
    for pos0 in (0, 7):
        _close(_run(q, k, v, pos0, 0.09), _expected(q, k, v, pos0, 0.09), v)
