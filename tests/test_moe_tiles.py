"""Where routed experts go over from short tiles to tall ones: just below and above the line, tall tiles a quarter full among them,
both forms give the same bits (mma.sync for the same tall tiles, tcgen05) and agree with the plain kernels."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,top,width,ff", [(319, 32, 4, 1536, 1120), (320, 32, 4, 1536, 1120), (834, 16, 2, 2048, 512), (835, 16, 2, 2048, 512),
                                                         (1001, 8, 3, 1000, 904)])
def test_tall_and_short_tiles_agree(tokens, experts, top, width, ff):
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops

    torch.manual_seed(tokens)
    h = torch.randn(tokens, width, device="cuda", dtype=torch.bfloat16)
    w_gate_up = torch.randn(experts, 2 * ff, width, device="cuda", dtype=torch.bfloat16) * width**-0.5
    w_down = torch.randn(experts, width, ff, device="cuda", dtype=torch.bfloat16) * ff**-0.5
    ids = torch.rand(tokens, experts, device="cuda").topk(top, 1).indices.to(torch.int32).contiguous()
    ids[: tokens // 2, 0] = 0  # one expert with far more slots than the others
    results, tall = {}, {}
    for choice in ("auto", "mma", "plain"):
        ctx = make_ctx(list(range(tokens)), [0] * tokens, options={"moe": choice})
        ctx.buffer = lambda name, shape, dtype=None, per_token=True, ws=ctx.workspace: ws.get(name, shape, dtype or torch.bfloat16, per_token=per_token)
        results[choice] = ops.moe_experts(ctx, h, ids, w_gate_up, w_down, 7.0, torch.empty(tokens * top, width, device="cuda"))
        assert int(ctx.err.item()) == 0
        tall[choice] = "moe_sorted_rows:torch.bfloat16" in ctx.workspace._flat  # what only the tcgen05 form asks for
    assert tall == dict(auto=tokens in (320, 835, 1001), mma=False, plain=False)
    assert torch.equal(results["auto"], results["mma"])
    # bfloat16 activations between the products: two roundings of 2^-9 apart at most
    torch.testing.assert_close(results["auto"], results["plain"], atol=2e-2, rtol=2e-2)
