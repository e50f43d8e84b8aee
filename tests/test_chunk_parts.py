"""Chunked recurrences whose scratch does not hold all heads: the heads go in parts through the same scratch, with the same bits, also where
the last part is smaller and where q/k heads are shared; a step that would need too many parts goes token by token."""

from __future__ import annotations

import pytest
import torch

from test_mixed_recurrences import DIM, HEADS, RULES, run

pytestmark = pytest.mark.gpu


def operands(n):
    torch.manual_seed(n)
    unit = torch.nn.functional.normalize(torch.randn(2, n, HEADS, DIM, device="cuda"), dim=-1).reshape(2, n, -1)
    return dict(q=unit[0], k=unit[1], v=torch.randn(n, HEADS * DIM, device="cuda"), beta=torch.rand(n, HEADS, device="cuda"),
                decay=0.6 + 0.4 * torch.rand(n, HEADS * DIM, device="cuda"))


@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("heads_at_once,parts", [(3, 1), (2, 2), (1, 3)])
def test_parts_of_the_heads(rule, heads_at_once, parts, monkeypatch):
    from llm_inference_b200.csrc.library import kernels
    from llm_inference_b200.parts import ops

    runs, slots = (1, 300, 290), [2, 0, 1]
    given = operands(sum(runs))
    out, states, launches = run(rule, given, slots, runs, {})
    number = dict(channel=0, head=0, general=1, wkv=2, memory=3)[rule]
    floats = int(kernels().lib.b200_state_chunks_scratch(number, sum(runs), 2, heads_at_once, heads_at_once, DIM, DIM))
    monkeypatch.setattr(ops, "CHUNK_SCRATCH_BYTES", 4 * floats)
    got, after, more = run(rule, given, slots, runs, {})
    assert more == launches + 3 * (parts - 1)
    assert torch.equal(got, out)
    assert all(torch.equal(a, b) for a, b in zip(after, states))
    monkeypatch.setattr(ops, "CHUNK_PARTS", 1)
    tokens = run(rule, given, slots, runs, {"delta_portions": "tokens"})[0]
    assert torch.equal(run(rule, given, slots, runs, {})[0], out if parts == 1 else tokens)


def test_q_and_k_heads_shared_across_parts(monkeypatch):
    """Six heads on two q/k heads, four at a time: a part's border inside a group of heads."""
    from llm_inference_b200.parts import ops
    from test_state_chunks import device_context

    heads, kvh, n = 6, 2, 200
    torch.manual_seed(1)
    q, k = (torch.nn.functional.normalize(torch.randn(n, kvh, DIM, device="cuda"), dim=-1).reshape(n, -1) for _ in range(2))
    v, beta, decay = torch.randn(n, heads * DIM, device="cuda"), torch.rand(n, heads, device="cuda"), 0.6 + 0.4 * torch.rand(n, heads * DIM, device="cuda")
    outs = []
    for limit in (1 << 30, None):
        runner, cache, ctx = device_context((n,), (0,), ((heads, DIM, DIM),), {})
        if limit is None:
            limit = 4 * int(ctx.lib.lib.b200_state_chunks_scratch(0, n, 1, 4, 4, DIM, DIM))
        monkeypatch.setattr(ops, "CHUNK_SCRATCH_BYTES", limit)
        cache.states[0][0].fill_(0.25)
        out = torch.full((n, heads * DIM), float("nan"), device="cuda")
        ops.delta_recurrence(ctx, q, k, v, beta, decay, cache.states[0][0], out, heads, kvh, DIM, DIM)
        runner.check()
        outs.append((out, cache.states[0][0].clone()))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
