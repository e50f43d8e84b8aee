"""Recurrent rules over prompt portions chunk by chunk: what is not finite in a token's operands reaches that token and later ones of
its request, never an earlier one of its chunk and never another request."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from test_state_chunks import device_context

pytestmark = pytest.mark.gpu

HEADS, DIM, RUNS = 2, 64, (41, 70)


def outputs(rule, operands, n):
    from llm_inference_b200.parts import ops

    shapes = ((HEADS, DIM, DIM), (HEADS, DIM), (HEADS,)) if rule == "memory" else ((HEADS, DIM, DIM),)
    runner, cache, ctx = device_context(RUNS, (1, 0), shapes, {"delta_portions": "chunks"})
    for array in cache.states[0]:
        array.fill_(0.125)
    state, out = cache.states[0][0], torch.full((n, HEADS * DIM), 7.0, device="cuda")
    sizes = (HEADS, DIM, DIM)
    if rule == "channel":
        ops.delta_recurrence(ctx, *(operands[x] for x in ("q", "k", "v", "beta", "decay")), state, out, HEADS, HEADS, DIM, DIM)
    elif rule == "head":
        kq = (operands["q"] * operands["k"]).view(n, HEADS, DIM).sum(-1).contiguous()
        ops.delta_head_recurrence(ctx, *(operands[x] for x in ("q", "k", "v", "beta")), operands["decay"][:, :HEADS].log().contiguous(), kq, state, out, HEADS, HEADS, DIM, DIM)
    elif rule == "general":
        ops.delta_general_recurrence(ctx, *(operands[x] for x in ("q", "k", "v", "decay")), operands["k"] * 0.5, operands["k"], state, out, *sizes)
    elif rule == "wkv":
        ops.wkv_recurrence(ctx, *(operands[x] for x in ("q", "k", "v", "beta", "decay")), state, out, *sizes)
    else:
        wide = HEADS * DIM
        proj = torch.cat([operands[x] for x in ("q", "k", "v", "decay")] + [operands["beta"]] * 2, 1).contiguous()
        zero = torch.zeros(HEADS, device="cuda")
        ops.mlstm(ctx, proj, (0, wide, 2 * wide, 3 * wide, 4 * wide, 4 * wide + HEADS), zero, zero, 9.0, cache.states[0], HEADS, DIM, DIM,
                  torch.ones(wide, device="cuda"), 1e-6, out)
    runner.check()
    return out


@pytest.mark.parametrize("rule", ["channel", "head", "general", "wkv", "memory"])
@pytest.mark.parametrize("operand,value", [("v", float("nan")), ("v", float("inf")), ("k", float("nan")), ("q", float("nan"))])
@pytest.mark.parametrize("at", [40, 41 + 30, 41 + 66])  # the last of its request and chunk; inside a whole chunk; inside a request's last chunk
def test_earlier_tokens_keep_their_bits(rule, operand, value, at):
    n = sum(RUNS)
    torch.manual_seed(at)
    unit = torch.nn.functional.normalize(torch.randn(2, n, HEADS, DIM, device="cuda"), dim=-1).reshape(2, n, -1)
    operands = dict(q=unit[0].contiguous(), k=unit[1].contiguous(), v=torch.randn(n, HEADS * DIM, device="cuda"),
                    beta=torch.rand(n, HEADS, device="cuda"), decay=0.6 + 0.4 * torch.rand(n, HEADS * DIM, device="cuda"))
    clean = outputs(rule, operands, n)
    spoilt = dict(operands)
    spoilt[operand] = operands[operand].clone()
    spoilt[operand][at] = value
    got = outputs(rule, spoilt, n)
    assert (rule, operand) == ("wkv", "k") or not torch.isfinite(got[at]).all()  # wkv reads out in front of the token's update
    own = range(RUNS[0]) if at < RUNS[0] else range(RUNS[0], n)
    others = [t for t in range(n) if t < at or t not in own]
    assert torch.isfinite(clean).all() and torch.equal(got[others], clean[others])


@pytest.mark.parametrize("rule", ["channel", "head", "general", "wkv", "memory"])
@pytest.mark.parametrize("operand", ["v", "k", "q"])
@pytest.mark.parametrize("value", [torch.finfo(torch.float32).max, -3.397e38])
@pytest.mark.parametrize("at", [41 + 5, 41 + 30, 41 + 66])
def test_the_largest_numbers_leave_earlier_tokens_alone(rule, operand, value, at):
    """They are finite: a zero in a triangle of pairs takes them out, although bfloat16 rounds them to infinity."""
    n = sum(RUNS)
    torch.manual_seed(at)
    unit = torch.nn.functional.normalize(torch.randn(2, n, HEADS, DIM, device="cuda"), dim=-1).reshape(2, n, -1)
    operands = dict(q=unit[0].contiguous(), k=unit[1].contiguous(), v=torch.randn(n, HEADS * DIM, device="cuda"),
                    beta=torch.rand(n, HEADS, device="cuda"), decay=0.6 + 0.4 * torch.rand(n, HEADS * DIM, device="cuda"))
    clean = outputs(rule, operands, n)
    operands[operand] = operands[operand].clone()
    operands[operand][at] = value
    got = outputs(rule, operands, n)
    own = range(RUNS[0], n)
    others = [t for t in range(n) if t < at or t not in own]
    assert torch.isfinite(clean).all() and torch.equal(got[others], clean[others])
