"""Attention over cached latents of prompt portions with expanded keys and values (tcgen05): beside the absorbed form on mma.sync and the
plain kernel, for ragged portions behind earlier tokens and beside single tokens, with and without a rotated part, sinks, gates per
head and per element, queries from a latent of their own, portions that end on and off a tile of 128."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

def step_of(part, runs, starts, page_size=16):
    """A runner, a cache with pages for every position and the context of one step."""
    from types import SimpleNamespace

    from llm_inference_b200.cache import PagedCache
    from llm_inference_b200.engine.runner import ModelRunner, StepEntry

    device, dtype = torch.device("cuda:0"), torch.bfloat16
    cache = PagedCache({0: part.cache_spec()}, dtype=dtype, device=device, page_size=page_size, max_num_sequences=8, max_model_length=512, step_tokens=256, num_pages=128)
    runner = ModelRunner(SimpleNamespace(device=device, dtype=dtype), cache, max_batch_tokens=512)
    for i, (run, start) in enumerate(zip(runs, starts)):
        cache.open(i + 1)
        cache.manager.ensure(i + 1, start + run)
    ctx = runner._build_context([StepEntry(i + 1, [0] * run) for i, run in enumerate(runs)], list(starts), [])
    return runner, cache, ctx


FORMS = {
    "rotated, sink, gate per head": dict(rot_dim=64, sink=True, gate=True, rank=512),
    "no position, latent queries": dict(rot_dim=0, sink=False, gate=False, rank=256, q_rank=96),
    "rotated, gate per element": dict(rot_dim=64, sink=False, gate=True, gate_per="element", rank=96, q_rank=40),
}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("runs,starts", [((128,), (0,)), ((1, 1, 129, 66), (77, 0, 3, 127)), ((200, 64), (0, 192))])
def test_expanded_portions_agree_with_the_latent_space(form, runs, starts):
    from llm_inference_b200.parts import PartSpec, build_part, ops
    from llm_inference_b200.weights import random_weights

    sizes = dict(FORMS[form])
    heads, hidden, rot = 3, 72, sizes["rot_dim"]
    position = PartSpec("rotary", dict(head_dim=rot, theta=1e4, rotary_dims=rot, interleaved=True)) if rot else None
    part = build_part("mixer", PartSpec("latent_attention", dict(prefix="", hidden_size=hidden, heads=heads, dim=128, vdim=128, scale=0.3 * (128 + rot) ** -0.5,
                                                                 eps=1e-5, position=position, **sizes)))
    torch.manual_seed(len(runs))
    part.load(random_weights(part.tensor_specs(), seed=3, std=0.2), torch.bfloat16, torch.device("cuda:0"))
    h = torch.randn(sum(runs), hidden, device="cuda").bfloat16()
    results = {}
    for choice in ("auto", "flash", "plain"):
        runner, cache, ctx = step_of(part, runs, starts)
        assert ctx.num_decode_seqs == sum(1 for r in runs if r == 1)
        view = cache.view(0, True, runner._tables)
        torch.manual_seed(5)
        view.keys.normal_(0.0, 0.7)
        ctx.options = {"attention": choice}
        results[choice] = part.forward(ctx, view, h).double().clone()
        rows = ops.latent_expansion(ctx, view, h.dtype, heads, 128, rot, 128, sizes["rank"])[1]
        assert (rows > 0) == (choice == "auto")  # the tcgen05 form is what is compared with the two others
        runner.check()
    scale = results["plain"].abs().max()
    off = {name: ((results[name] - results["plain"]).norm() / results["plain"].norm()).item() for name in ("auto", "flash")}
    # bfloat16 keys and values (or queries and weighted latents): a few roundings of 2^-9 on the way, in either form.
    assert off["auto"] < max(1.5 * off["flash"], 6e-3), off
    assert (results["auto"] - results["plain"]).abs().max() < 3e-2 * scale


def test_what_is_not_finite_in_one_request_stays_there():
    from llm_inference_b200.parts import PartSpec, build_part
    from llm_inference_b200.weights import random_weights

    part = build_part("mixer", PartSpec("latent_attention", dict(prefix="", hidden_size=64, heads=2, dim=128, rot_dim=0, vdim=128, rank=64, scale=0.1, eps=1e-5)))
    part.load(random_weights(part.tensor_specs(), seed=3, std=0.2), torch.bfloat16, torch.device("cuda:0"))
    h = torch.randn(200, 64, device="cuda").bfloat16()
    outs = []
    for bad in (False, True):
        runner, cache, ctx = step_of(part, [100, 100], [0, 0])
        rows = h.clone()
        if bad:
            rows[100:] = float("nan")
        outs.append(part.forward(ctx, cache.view(0, True, runner._tables), rows).clone())
        runner.check()
    assert torch.equal(outs[0][:100], outs[1][:100]) and torch.isnan(outs[1][100:]).all()
