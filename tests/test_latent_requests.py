"""Latent attention of steps whose requests differ in length: long portions expand their keys and values whatever stands beside them, short
ones where that takes less than their walks in the latent space, in whatever order the requests come."""

from __future__ import annotations

import pytest
import torch

from test_latent_portions import FORMS, step_of


@pytest.mark.parametrize("requests,new,keys,heads,expand", [
    (1, 2, 500, 12, True), (1, 47, 16000, 12, True), (20, 2, 500, 12, False), (20, 16, 4000, 12, True), (20, 2, 4000, 16, False), (20, 32, 4000, 16, True),
    (60, 2, 500, 12, False), (60, 16, 500, 12, False), (60, 2, 4000, 12, False), (60, 16, 4000, 12, False), (8, 2, 1000, 16, True), (1, 8, 8, 12, False),
])
def test_short_portions_expand_where_that_was_measured_to_take_less(requests, new, keys, heads, expand):
    from llm_inference_b200.parts import ops

    lengths = [new] * requests, [keys + new] * requests
    assert (ops.latent_expand_from(*lengths, heads, 148) == 2) == expand
    # Long portions beside them change nothing; without short ones there is nothing to decide.
    beside = lengths[0] + [2000], lengths[1] + [2000]
    assert ops.latent_expand_from(*beside, heads, 148) == ops.latent_expand_from(*lengths, heads, 148)
    assert ops.latent_expand_from([48, 2000], [48, 2000], heads, 148) == ops.LATENT_EXPAND_FROM


def built(form):
    from llm_inference_b200.parts import PartSpec, build_part
    from llm_inference_b200.weights import random_weights

    sizes = dict(FORMS[form])
    rot = sizes["rot_dim"]
    position = PartSpec("rotary", dict(head_dim=rot, theta=1e4, rotary_dims=rot, interleaved=True)) if rot else None
    part = build_part("mixer", PartSpec("latent_attention", dict(prefix="", hidden_size=72, heads=3, dim=128, vdim=128, scale=0.3 * (128 + rot) ** -0.5, eps=1e-5,
                                                                 position=position, **sizes)))
    part.load(random_weights(part.tensor_specs(), seed=3, std=0.2), torch.bfloat16, torch.device("cuda:0"))
    return part


def forward(part, runs, starts, h, choice="auto"):
    """The layer's output and what the step decided: fewest new tokens, key rows, rows in the latent space."""
    from llm_inference_b200.parts import ops

    runner, cache, ctx = step_of(part, runs, starts)
    view = cache.view(0, True, runner._tables)
    torch.manual_seed(5)
    view.keys.normal_(0.0, 0.7)
    ctx.options = {"attention": choice}
    for name in ("attn", "latent_out"):  # what earlier steps left in shared scratch must not show
        ctx.workspace.get(name, (1 << 18,), torch.bfloat16, per_token=False).fill_(float("nan"))
    out = part.forward(ctx, view, h).clone()
    runner.check()
    return out, ops.latent_expansion(ctx, view, torch.bfloat16, part.heads, part.dim, part.rot_dim, part.vdim, part.rank)


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("fewest", [2, 48])
@pytest.mark.parametrize("runs,starts", [((1, 200, 20, 48, 47), (5, 0, 100, 60, 3)), ((2, 140), (300, 0)), ((140, 2), (0, 300)), ((1, 1, 47, 3), (9, 0, 0, 40))])
def test_requests_of_either_kind_in_any_order(form, fewest, runs, starts, monkeypatch):
    from llm_inference_b200.parts import ops

    monkeypatch.setattr(ops, "latent_expand_from", lambda *lengths: fewest)
    part = built(form)
    torch.manual_seed(len(runs))
    h = torch.randn(sum(runs), 72, device="cuda").bfloat16()
    got, decided = forward(part, runs, starts, h)
    long = [r >= fewest for r in runs]
    rows = sum(-(-(r + s) // 128) * 128 for r, s, own in zip(runs, starts, long) if own)
    absorbed = sum(runs[: 1 + max((i for i, own in enumerate(long) if not own), default=-1)])
    assert decided == ((fewest, rows, absorbed) if rows else (0, 0, sum(runs)))
    want = forward(part, runs, starts, h, "plain")[0].double()
    assert torch.isfinite(got).all()
    at = 0
    for run in runs:  # bfloat16 keys and values, or queries and weighted latents: a few roundings of 2^-9
        own = slice(at, at + run)
        assert ((got[own].double() - want[own]).norm() / want[own].norm()).item() < 8e-3
        at += run


@pytest.mark.gpu
def test_too_much_scratch_and_other_options_stay_in_the_latent_space(monkeypatch):
    from llm_inference_b200.parts import ops

    part = built("rotated, sink, gate per head")
    h = torch.randn(200, 72, device="cuda").bfloat16()
    expanded, decided = forward(part, (200,), (0,), h)
    latent, nothing = forward(part, (200,), (0,), h, "flash")
    assert decided == (48, 256, 0) and nothing == (0, 0, 200) and not torch.equal(expanded, latent)
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", 256 * 3 * 256 * 2 - 1)
    got, decided = forward(part, (200,), (0,), h)
    assert decided == nothing and torch.equal(got, latent)
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", 256 * 3 * 256 * 2)
    got, decided = forward(part, (200,), (0,), h)
    assert decided == (48, 256, 0) and torch.equal(got, expanded)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["rotated, sink, gate per head", "no position, latent queries"])
def test_neighbours_change_no_bits_of_a_long_portion(form):
    """Beside another long one and beside two short ones, with the same number of rows in every product."""
    part = built(form)
    torch.manual_seed(0)
    rows = torch.randn(150, 72, device="cuda").bfloat16()
    beside, _ = forward(part, (100, 50), (0, 10), rows)
    split, _ = forward(part, (100, 25, 25), (0, 10, 0), rows)  # the 50 become two short requests
    assert torch.equal(beside[:100], split[:100])


@pytest.mark.gpu
@pytest.mark.parametrize("change,dtype,kept", [({}, torch.bfloat16, True), ({}, torch.float32, False), ({"window": 40}, torch.bfloat16, False),
                                               ({"dim": 96}, torch.bfloat16, False), ({"rank": 68}, torch.bfloat16, False)])
def test_the_expanding_matrix_is_held_only_where_it_can_be_used(change, dtype, kept):
    from llm_inference_b200.parts import PartSpec, build_part
    from llm_inference_b200.weights import random_weights

    sizes = dict(dict(prefix="", hidden_size=64, heads=2, dim=128, rot_dim=0, vdim=128, rank=64, scale=0.1, eps=1e-5), **change)
    part = build_part("mixer", PartSpec("latent_attention", sizes))
    part.load(random_weights(part.tensor_specs(), seed=3, std=0.2), dtype, torch.device("cuda:0"))
    assert (part.w_expand is not None) == kept
