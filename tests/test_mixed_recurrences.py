"""Recurrent rules in steps that hold decoded tokens beside prompt portions: the portions run 32 tokens at a time, the single tokens in
front of them take one step of the recurrence, to the bit what either gives by itself."""

from __future__ import annotations

import pytest
import torch

from test_state_chunks import device_context

pytestmark = pytest.mark.gpu

HEADS, DIM = 3, 64
RULES = ["channel", "head", "general", "wkv", "memory"]


def run(rule, operands, slots, runs, options):
    """(outputs, state slots) of one step; ``operands`` hold the step's tokens."""
    from llm_inference_b200.parts import ops

    n = sum(runs)
    shapes = ((HEADS, DIM, DIM), (HEADS, DIM), (HEADS,)) if rule == "memory" else ((HEADS, DIM, DIM),)
    runner, cache, ctx = device_context(runs, slots, shapes, options)
    ctx.num_decode_seqs = next((i for i, r in enumerate(runs) if r > 1), len(runs))
    states = cache.states[0]
    torch.manual_seed(2)
    for array in states:
        array.normal_()
    o = {name: rows.contiguous() for name, rows in operands.items()}
    out = torch.full((n, HEADS * DIM), float("nan"), device="cuda")
    calls = ctx.lib.calls
    if rule == "channel":
        ops.delta_recurrence(ctx, o["q"], o["k"], o["v"], o["beta"], o["decay"], states[0], out, HEADS, HEADS, DIM, DIM)
    elif rule == "head":
        kq = (o["q"] * o["k"]).view(n, HEADS, DIM).sum(-1).contiguous()
        ops.delta_head_recurrence(ctx, o["q"], o["k"], o["v"], o["beta"], o["decay"][:, :HEADS].log().contiguous(), kq, states[0], out, HEADS, HEADS, DIM, DIM)
    elif rule == "general":
        ops.delta_general_recurrence(ctx, o["q"], o["k"], o["v"], o["decay"], o["k"] * 0.5, o["k"], states[0], out, HEADS, DIM, DIM)
    elif rule == "wkv":
        ops.wkv_recurrence(ctx, o["q"], o["k"], o["v"], o["beta"], o["decay"], states[0], out, HEADS, DIM, DIM)
    else:
        wide = HEADS * DIM
        proj = torch.cat([o[x] for x in ("q", "k", "v", "decay")] + [o["beta"]] * 2, 1).contiguous()
        zero = torch.zeros(HEADS, device="cuda")
        ops.mlstm(ctx, proj, (0, wide, 2 * wide, 3 * wide, 4 * wide, 4 * wide + HEADS), zero, zero, 9.0, states, HEADS, DIM, DIM,
                  torch.ones(wide, device="cuda"), 1e-6, out)
    runner.check()
    return out, [array.clone() for array in states], ctx.lib.calls - calls


@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("runs", [(1, 1, 1, 150), (1, 33, 1, 64), (1, 1)])
def test_single_tokens_beside_portions(rule, runs):
    n, slots = sum(runs), [3, 0, 4, 1][: len(runs)]
    torch.manual_seed(n)
    unit = torch.nn.functional.normalize(torch.randn(2, n, HEADS, DIM, device="cuda"), dim=-1).reshape(2, n, -1)
    operands = dict(q=unit[0], k=unit[1], v=torch.randn(n, HEADS * DIM, device="cuda"), beta=torch.rand(n, HEADS, device="cuda"),
                    decay=0.6 + 0.4 * torch.rand(n, HEADS * DIM, device="cuda"))
    lead = next((i for i, r in enumerate(runs) if r > 1), 0)  # a step of single tokens only goes as it is told
    out, states, _ = run(rule, operands, slots, runs, {"delta_portions": "chunks"})
    front, front_states, _ = run(rule, {k: v[:lead] for k, v in operands.items()}, slots[:lead], runs[:lead], {"delta_portions": "tokens"}) if lead else (None, None, 0)
    back, back_states, _ = run(rule, {k: v[lead:] for k, v in operands.items()}, slots[lead:], runs[lead:], {"delta_portions": "chunks"})
    if lead and rule != "memory":  # the memory's single tokens work their gates out in another kernel when they are alone
        assert torch.equal(out[:lead], front)
    elif lead:
        torch.testing.assert_close(out[:lead], front, atol=2e-5, rtol=2e-5)
    assert torch.equal(out[lead:], back)
    for array, own, other in zip(states, front_states or back_states, back_states):
        if lead and rule != "memory":
            assert torch.equal(array[slots[:lead]], own[slots[:lead]])
        assert torch.equal(array[slots[lead:]], other[slots[lead:]])
        untouched = [s for s in range(array.shape[0]) if s not in slots]
        assert torch.equal(array[untouched], other[untouched])


@pytest.mark.parametrize("rule", RULES)
def test_decoded_tokens_do_not_depend_on_the_portion_beside_them(rule):
    """The same single tokens beside a portion that runs token by token and beside one that runs in chunks."""
    torch.manual_seed(7)
    n = 2 + 400
    unit = torch.nn.functional.normalize(torch.randn(2, n, HEADS, DIM, device="cuda"), dim=-1).reshape(2, n, -1)
    operands = dict(q=unit[0], k=unit[1], v=torch.randn(n, HEADS * DIM, device="cuda"), beta=torch.rand(n, HEADS, device="cuda"),
                    decay=0.6 + 0.4 * torch.rand(n, HEADS * DIM, device="cuda"))
    short, _, calls = run(rule, {k: v[: 2 + 9] for k, v in operands.items()}, [3, 0, 1], (1, 1, 9), {})
    long, _, more = run(rule, operands, [3, 0, 1], (1, 1, 400), {})
    assert more > calls  # the long portion took the chunked form
    assert torch.equal(short[:2], long[:2])
