"""Prompt portions in true 32-bit attention (the tiled kernel): against the plain kernel's formulas in 64 bits at the ends of its tiles
(32 rows of tokens and heads, 64 keys), with windows, sinks, ragged requests beside single tokens, odd head and page sizes, and values
of later tokens that are not finite."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [
    # q heads, kv heads, head size, page size, window, sink, (new tokens, tokens before) per request
    (12, 2, 128, 64, 0, False, ((1, 40), (1, 0), (43, 0), (33, 200))),
    (5, 5, 64, 16, 0, True, ((32, 0), (65, 31))),
    (6, 2, 24, 7, 20, False, ((1, 300), (64, 300), (97, 5))),
    (16, 1, 100, 32, 64, True, ((2, 254), (40, 64))),
    (3, 3, 128, 128, 1, False, ((63, 129),)),
]


@pytest.mark.parametrize("q_heads,kv_heads,dim,page,window,with_sink,requests", CASES)
def test_portions_against_64_bits(q_heads, kv_heads, dim, page, window, with_sink, requests):
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import attention_dispatch, ops
    from llm_inference_b200.parts.context import CacheView

    rng = np.random.default_rng(q_heads * dim + window)
    runs, starts = [r for r, _ in requests], [s for _, s in requests]
    lengths = [r + s for r, s in requests]
    need = [-(-n // page) for n in lengths]
    order = rng.permutation(sum(need) + 2)
    tables, at = np.zeros((len(runs), max(need)), dtype=np.int32), 0
    for row, count in zip(tables, need):
        row[:count] = order[at : at + count]
        at += count
    keys, values = (rng.normal(size=(sum(need) + 2, kv_heads, page, dim)).astype(np.float32) for _ in range(2))
    q = (3.0 * rng.normal(size=(sum(runs), q_heads, dim))).astype(np.float32)
    sink = rng.normal(size=q_heads).astype(np.float32)
    last = len(runs) - 1  # the last token of the last request has values that are not finite: nobody before it sees them
    where = lengths[last] - 1
    values[tables[last][where // page], :, where % page] = np.nan
    scale, share = dim**-0.5, q_heads // kv_heads
    want, row = np.zeros((sum(runs), q_heads, dim)), 0
    for i, (run, start) in enumerate(requests):
        flat = [a[tables[i][: need[i]]].transpose(0, 2, 1, 3).reshape(-1, kv_heads, dim)[: lengths[i]].astype(np.float64) for a in (keys, values)]
        for t in range(run):
            pos = start + t
            lo = max(0, pos - window + 1) if window else 0
            for h in range(q_heads):
                s = flat[0][lo : pos + 1, h // share] @ q[row, h].astype(np.float64) * scale
                top = max(s.max(), sink[h]) if with_sink else s.max()
                p = np.exp(s - top)
                want[row, h] = (p @ flat[1][lo : pos + 1, h // share]) / (p.sum() + (np.exp(sink[h] - top) if with_sink else 0.0))
            row += 1
    ctx = make_ctx([p for r, s in requests for p in range(s, s + r)], [i for i, r in enumerate(runs) for _ in range(r)], starts, runs)
    ctx.num_decode_seqs = sum(1 for r in runs if r == 1)
    view = CacheView(0, True, torch.from_numpy(keys).cuda(), torch.from_numpy(values).cuda(), torch.from_numpy(tables).cuda(), len(order), tables.shape[1], page, window)
    shape = ops.ScoreShape(sink=torch.from_numpy(sink).cuda()) if with_sink else ops.NO_SHAPE
    rows = torch.from_numpy(q.reshape(sum(runs), -1)).cuda()
    assert ops.portion_attention_f32_takes(ctx, view, rows, q_heads, kv_heads, dim, -1, shape)
    out = torch.full_like(rows, 7.0)
    attention_dispatch.attend(ctx, view, rows, out, q_heads, kv_heads, dim, scale, shape=shape)
    assert int(ctx.err.item()) == 0
    got = out.double().cpu().numpy().reshape(want.shape)
    assert np.isnan(got[-1]).all() and np.isnan(want[-1]).all()
    # 32-bit: a score is a sum of dim products of size up to ten, its error enters the weights as it is
    np.testing.assert_allclose(got[:-1], want[:-1], atol=3e-5, rtol=3e-5)


def test_a_bad_page_is_flagged_and_not_read():
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops
    from llm_inference_b200.parts.context import CacheView

    ctx = make_ctx(list(range(70)), [0] * 70, [0], [70])
    arena = torch.randn(3, 1, 64, 16, device="cuda")
    q = torch.randn(70, 16, device="cuda")
    view = CacheView(0, True, arena, arena, torch.tensor([[1, 9]], dtype=torch.int32, device="cuda"), 3, 2, 64, 0)
    out = ops.portion_attention_f32(ctx, view, q, torch.empty_like(q), 1, 1, 16, 0.25, first_seq=0)
    assert int(ctx.err.item()) == 1 and torch.isfinite(out).all()


def attend_one_request(q, keys, values, heads, dim, decode=0):
    """One request's tokens, all new, one kv head a query head; rows of keys and values in pages of 32."""
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops
    from llm_inference_b200.parts.context import CacheView

    n, page = q.shape[0], 32
    pages = -(-n // page)
    arenas = [torch.zeros(pages, heads, page, dim, device="cuda") for _ in range(2)]
    for arena, rows in zip(arenas, (keys, values)):
        padded = torch.zeros(pages * page, heads, dim, device="cuda")
        padded[:n] = rows
        arena.copy_(padded.view(pages, page, heads, dim).transpose(1, 2))
    ctx = make_ctx(list(range(n)), [0] * n, [0], [n])
    view = CacheView(0, True, *arenas, torch.arange(pages, dtype=torch.int32, device="cuda")[None], pages, pages, page, 0)
    rows = q.reshape(n, -1).contiguous()
    out = ops.portion_attention_f32(ctx, view, rows, torch.full_like(rows, 7.0), heads, heads, dim, dim**-0.5, first_seq=0)
    assert int(ctx.err.item()) == 0
    return out.view(n, heads, dim)


@pytest.mark.parametrize("operand", ["q", "k"])
@pytest.mark.parametrize("at", [0, 16, 17, 48, 90])
@pytest.mark.parametrize("dim", [64, 128])
def test_a_score_that_is_nan_reaches_its_row(operand, at, dim):
    """Also where it is the only one that a row has of its sixteen keys (tokens 0, 16 and 48), or all of a row's scores are."""
    torch.manual_seed(at)
    n, heads = 100, 2
    operands = dict(q=torch.randn(n, heads, dim, device="cuda"), k=torch.randn(n, heads, dim, device="cuda"), v=torch.randn(n, heads, dim, device="cuda"))
    clean = attend_one_request(*operands.values(), heads, dim)
    operands[operand][at, 1, 3] = float("nan")
    got = attend_one_request(*operands.values(), heads, dim)
    reached = torch.zeros(n, heads, dtype=torch.bool, device="cuda")
    reached[at : at + 1 if operand == "q" else n, 1] = True
    assert torch.isnan(got[reached]).all()
    assert torch.equal(got[~reached], clean[~reached])


@pytest.mark.parametrize("operand,value", [("q", "inf"), ("k", "inf"), ("k", "-inf"), ("v", "inf"), ("v", "-inf"), ("v", "3.4e38"), ("k", "3.4e38"), ("k", "-3.4e38")])
@pytest.mark.parametrize("at", [0, 16, 31, 75])
@pytest.mark.parametrize("dim", [24, 128])
def test_infinite_and_very_large_numbers(operand, value, at, dim):
    """As 32-bit products and sums have them: signs of infinities, keys that an infinite score takes out, numbers next to the largest."""
    torch.manual_seed(at + dim)
    n, heads = 90, 2
    operands = dict(q=0.3 * torch.randn(n, heads, dim, device="cuda"), k=torch.randn(n, heads, dim, device="cuda"), v=torch.randn(n, heads, dim, device="cuda"))
    clean = attend_one_request(*operands.values(), heads, dim)
    operands[operand][at, 1, 5] = float(value)
    q, k, v = (x.double().transpose(0, 1) for x in operands.values())
    scores = (q @ k.transpose(1, 2)).float().double() * dim**-0.5  # very large sums overflow 32 bits
    want = torch.zeros(n, heads, dim, dtype=torch.float64, device="cuda")
    for t in range(n):
        seen = scores[:, t, : t + 1]
        weights = torch.where(seen == -float("inf"), 0.0, torch.exp(seen - seen.max(-1, keepdim=True).values))
        total = weights.sum(-1, keepdim=True)
        want[t] = (weights[..., None] * v[:, : t + 1]).sum(1) * torch.where(total > 0, 1 / total, 0.0)
    got = attend_one_request(*operands.values(), heads, dim).double()
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    finite = torch.isfinite(want)
    close = 3e-5 + 3e-5 * want[finite].abs()  # as for the portions above
    assert ((got[finite] - want[finite]).abs() <= close).all()
    assert torch.equal(got[:at], clean[:at].double())


@pytest.mark.parametrize("q_heads,kv_heads,dim,window,with_sink", [(12, 2, 128, 0, False), (3, 3, 64, 20, True), (16, 1, 100, 0, True), (4, 2, 24, 70, False)])
def test_both_forms_give_the_same_bits(q_heads, kv_heads, dim, window, with_sink):
    """The form for few keys a block is chosen by the whole step; a row must not depend on that."""
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops
    from llm_inference_b200.parts.context import CacheView

    torch.manual_seed(dim)
    runs, starts, page = [5, 64, 33, 130, 1, 70], [3, 0, 40, 200, 300, 0], 16
    pages = -(-max(r + s for r, s in zip(runs, starts)) // page)
    table = torch.randperm(len(runs) * pages, device="cuda").int().view(len(runs), pages)
    keys, values = (torch.randn(len(runs) * pages, kv_heads, page, dim, device="cuda") for _ in range(2))
    keys[7, :, 3], values[11, :, 5, 2], values[12, :, 9] = float("inf"), float("-inf"), torch.finfo(torch.float32).max
    shape = ops.ScoreShape(sink=torch.randn(q_heads, device="cuda")) if with_sink else ops.NO_SHAPE
    view = CacheView(0, True, keys, values, table, len(runs) * pages, pages, page, window)
    q = torch.randn(sum(runs), q_heads * dim, device="cuda")
    outs = []
    for form in ("few", "many"):
        ctx = make_ctx([p for r, s in zip(runs, starts) for p in range(s, s + r)], [i for i, r in enumerate(runs) for _ in range(r)], starts, runs, {"portion_keys": form})
        outs.append(ops.portion_attention_f32(ctx, view, q, torch.full_like(q, 7.0), q_heads, kv_heads, dim, dim**-0.5, first_seq=0, shape=shape))
        assert int(ctx.err.item()) == 0
    assert torch.equal(outs[0].nan_to_num(nan=1e30), outs[1].nan_to_num(nan=1e30)) and torch.isfinite(outs[0]).any()


def test_infinities_of_both_signs_and_nan_in_one_column():
    """Values that are not finite, told apart: NaN beats all, infinities of both signs are NaN, one sign stays, other columns are as they were."""
    torch.manual_seed(3)
    n, dim = 80, 64
    q, k, v = (0.3 * torch.randn(n, 1, dim, device="cuda") for _ in range(3))
    clean = attend_one_request(q, k, v, 1, dim)
    inf, nan = float("inf"), float("nan")
    v[5, 0, 1], v[40, 0, 2], v[7, 0, 3], v[41, 0, 3], v[9, 0, 4], v[9, 0, 4] = inf, -inf, inf, -inf, inf, nan
    got = attend_one_request(q, k, v, 1, dim)
    assert (got[5:, 0, 1] == inf).all() and (got[40:, 0, 2] == -inf).all() and (got[7:41, 0, 3] == inf).all()
    assert torch.isnan(got[41:, 0, 3]).all() and torch.isnan(got[9:, 0, 4]).all()
    assert torch.equal(got[:5], clean[:5]) and torch.isfinite(got[5:, 0, 5:]).all()
