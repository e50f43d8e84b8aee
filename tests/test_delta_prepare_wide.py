"""The delta rules' convolution, unit vectors, betas and decays over steps long enough for four tokens a block: ragged requests whose
first tokens reach into their slots, a step that ends inside a block of four, heads of up to 128, of up to 256 and of more channels that are no
whole number of a warp's."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from test_state_chunks import device_context, on_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dk,dv,runs", [(12, 12, 128, 128, (301,)), (4, 2, 64, 36, (1, 2, 3, 300, 1)), (3, 1, 20, 8, (4, 297)),
                                                       (2, 2, 132, 8, (298,)), (3, 1, 256, 16, (2, 5, 297)), (2, 1, 260, 8, (1, 299)), (2, 2, 1028, 8, (3, 298))])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("per_head", [False, True])
def test_against_64_bits(heads, kv_heads, dk, dv, runs, dtype, per_head):
    from llm_inference_b200.parts import ops

    n, taps, span = sum(runs), 4, 1 if per_head else dk
    channels = 2 * kv_heads * dk + heads * dv
    rng = np.random.default_rng(dk)
    rounded = lambda a: torch.from_numpy(a.astype(np.float32)).to(dtype)
    width = channels + heads + (-(channels + heads) % 8)
    proj, decay_in = rounded(rng.normal(size=(n, width))), rounded(rng.normal(size=(n, heads * span + (-heads * span) % 4)))
    slots = list(range(len(runs)))[::-1]
    held = rounded(rng.normal(size=(len(runs), taps - 1, channels)))
    weights, a_log, dt_bias = (rng.normal(size=s).astype(np.float32) for s in ((channels, taps), (heads,), (heads * span,)))
    runner, cache, ctx = device_context(runs, slots, ((1,),), {})
    ctx.token_seq = torch.tensor(np.repeat(np.arange(len(runs)), runs).tolist(), dtype=torch.int32, device="cuda")
    conv = torch.zeros(len(runs), taps - 1, channels, dtype=dtype, device="cuda")
    conv[slots] = held.cuda()
    outs = [torch.full((n, w), float("nan"), device="cuda") for w in (kv_heads * dk, kv_heads * dk, heads * dv, heads, heads * span)]
    kq = torch.full((n, kv_heads), float("nan"), device="cuda") if per_head else None
    ops.delta_prepare(ctx, proj.cuda(), decay_in.cuda(), on_device(weights), conv, torch.from_numpy(a_log).cuda(), torch.from_numpy(dt_bias).cuda(),
                      heads, kv_heads, dk, dv, *outs, kq)
    runner.check()
    x, z, at = proj.double().numpy(), decay_in.double().numpy()[:, : heads * span], 0
    sigmoid = lambda v: 1 / (1 + np.exp(-v))
    y = np.zeros((n, channels))
    for i, run in enumerate(runs):
        rows = np.concatenate([held[i].double().numpy(), x[at : at + run, :channels]])
        y[at : at + run] = sum(rows[j : j + run] * weights[:, j].astype(np.float64) for j in range(taps))
        assert torch.equal(conv[slots[i]].cpu().double(), torch.from_numpy(rows[-(taps - 1) :]))
        at += run
    y *= sigmoid(y)
    q, k = (y[:, j * kv_heads * dk : (j + 1) * kv_heads * dk].reshape(n, kv_heads, dk) for j in range(2))
    q, k = (v / np.sqrt((v * v).sum(-1, keepdims=True) + 1e-6) for v in (q, k))
    q = q * dk**-0.5
    log_decay = -np.exp(a_log.astype(np.float64))[:, None] * np.log1p(np.exp(z + dt_bias.astype(np.float64))).reshape(n, heads, span)
    want = [q, k, y[:, 2 * kv_heads * dk :], sigmoid(x[:, channels : channels + heads]), log_decay if per_head else np.exp(log_decay)]
    for got, wanted in zip(outs, want):  # 32-bit sums of at most 128 products of order one
        np.testing.assert_allclose(got.double().cpu().numpy(), wanted.reshape(n, -1), atol=1e-5, rtol=1e-5)
    if per_head:
        np.testing.assert_allclose(kq.double().cpu().numpy(), (q * k).sum(-1), atol=1e-5, rtol=1e-5)
