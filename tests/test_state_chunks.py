"""Recurrent rules over prompt portions chunk by chunk and token by token, against the recurrences themselves in 64 bits, at the
sizes where a chunk, a tile of the state or a wide copy ends: portions around multiples of 32 tokens, key and value sizes that are
multiples of nothing, decays from one down to zero, states that come in."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from test_parts import context_for

pytestmark = pytest.mark.gpu

# All arithmetic is 32-bit: a sum of n products carries about sqrt(n) roundings of 6e-8, and a state here adds up at most a few hundred
# unit-sized terms.
CLOSE = dict(atol=2e-5, rtol=2e-5)


def device_context(runs, slots, state_shapes, options):
    from llm_inference_b200.parts import StateSpec

    runner, cache, ctx = context_for({0: StateSpec(state_shapes, (torch.float32,) * len(state_shapes))}, torch.float32, [1] * len(runs))
    ctx.options = options
    as_device = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    ctx.num_tokens, ctx.num_seqs, ctx.max_q_len = sum(runs), len(runs), max(runs)
    ctx.seq_q_start, ctx.seq_q_len = as_device(np.concatenate([[0], np.cumsum(runs)[:-1]]).tolist()), as_device(list(runs))
    ctx.seq_slot = as_device(list(slots))
    return runner, cache, ctx


def on_device(array):
    return torch.from_numpy(np.ascontiguousarray(array.reshape(array.shape[0], -1))).cuda()


DELTA_SIZES = [
    (2, 1, 128, 128, (113, 32, 1)),
    (3, 3, 64, 16, (31, 65)),
    (2, 2, 33, 17, (64, 33)),
    (1, 1, 256, 40, (127,)),
    (2, 2, 72, 130, (96, 95, 97)),
]


@pytest.mark.parametrize("heads,kv_heads,dk,dv,runs", DELTA_SIZES)
@pytest.mark.parametrize("portions", ["chunks", "tokens"])
@pytest.mark.parametrize("per_head", [False, True])
def test_delta_rules(heads, kv_heads, dk, dv, runs, portions, per_head):
    from llm_inference_b200.parts import ops

    n = sum(runs)
    rng = np.random.default_rng(dk + dv)
    unit = lambda x: x / np.linalg.norm(x, axis=-1, keepdims=True)
    q, k = unit(rng.normal(size=(n, kv_heads, dk))), unit(rng.normal(size=(n, kv_heads, dk)))
    k[5:20] = k[5]  # keys that repeat, with beta near one: the triangular system at its stiffest
    v, beta = rng.normal(size=(n, heads, dv)), rng.uniform(0.9, 1.0, (n, heads))
    logs = -np.exp(rng.normal(-4, 3, (n, heads, 1 if per_head else dk)))
    logs[3::29] = 0.0
    logs[17::41, 0] = -400.0  # a memory that ends at once
    start = rng.normal(size=(len(runs), heads, dk, dv))
    q, k, v, beta, logs, start = (a.astype(np.float32) for a in (q, k, v, beta, logs, start))
    decay = logs if per_head else np.exp(logs)
    factors = np.broadcast_to(np.exp(logs.astype(np.float64)) if per_head else decay.astype(np.float64), (n, heads, dk))
    states, want, at = start.astype(np.float64), np.zeros((n, heads, dv)), 0
    share = heads // kv_heads
    for s, run in enumerate(runs):
        for t in range(at, at + run):
            key, query = (x[t].repeat(share, axis=0).astype(np.float64) for x in (k, q))
            S = states[s] * factors[t][..., None]
            u = beta[t].astype(np.float64)[:, None] * (v[t] - np.einsum("hkv,hk->hv", S, key))
            states[s] = S + key[..., None] * u[:, None]
            want[t] = np.einsum("hkv,hk->hv", states[s], query)
        at += run
    slots = [4, 0, 2][: len(runs)]
    runner, cache, ctx = device_context(runs, slots, ((heads, dk, dv),), {"delta_portions": portions})
    state = cache.states[0][0]
    untouched = state.clone().normal_()
    state.copy_(untouched)
    state[slots] = torch.from_numpy(start).cuda()
    out = torch.full((n, heads * dv), float("nan"), device="cuda")
    device = [on_device(a) for a in (q, k, v, beta, decay)]
    if per_head:
        ops.delta_head_recurrence(ctx, *device, on_device((q * k).sum(-1)), state, out, heads, kv_heads, dk, dv)
    else:
        ops.delta_recurrence(ctx, *device, state, out, heads, kv_heads, dk, dv)
    runner.check()
    np.testing.assert_allclose(out.double().cpu().numpy().reshape(want.shape), want, **CLOSE)
    np.testing.assert_allclose(state[slots].double().cpu().numpy(), states, **CLOSE)
    others = [slot for slot in range(state.shape[0]) if slot not in slots]
    assert torch.equal(state[others], untouched[others])


LINEAR_SIZES = [
    (2, 64, 64, (81, 32, 1)),
    (3, 33, 17, (31, 65)),
    (1, 128, 70, (127,)),
    (2, 16, 130, (96, 95, 97)),
]


@pytest.mark.parametrize("heads,dk,dv,runs", LINEAR_SIZES)
@pytest.mark.parametrize("portions", ["chunks", "tokens"])
@pytest.mark.parametrize("general", [False, True])
def test_rules_in_which_the_values_enter_as_they_are(heads, dk, dv, runs, portions, general):
    from llm_inference_b200.parts import ops

    n = sum(runs)
    rng = np.random.default_rng(dk + dv)
    r, k, v = (rng.normal(size=(n, heads, width)) for width in (dk, dk, dv))
    k[5:20] = k[5]
    w = np.exp(-np.exp(rng.normal(-3, 2, (n, heads, dk))))
    w[3::29], w[17::41, 0] = 1.0, 0.0
    start, bonus = rng.normal(size=(len(runs), heads, dk, dv)), rng.normal(size=(n, heads))
    u = k / np.linalg.norm(k, axis=-1, keepdims=True)
    if general:  # decays of this rule are bounded from below
        w = np.maximum(w, 0.545)
    au = u * rng.uniform(0.0, 1.0, (n, heads, dk))
    r, k, v, w, start, bonus, u, au = (a.astype(np.float32) for a in (r, k, v, w, start, bonus, u, au))
    states, want, at = start.astype(np.float64), np.zeros((n, heads, dv)), 0
    for s, run in enumerate(runs):
        for t in range(at, at + run):
            R, K, V, D, U, A = (x[t].astype(np.float64) for x in (r, k, v, w, u, au))
            old = states[s]
            added = K[..., None] * V[:, None]
            if general:
                states[s] = D[..., None] * old - A[..., None] * np.einsum("hkv,hk->hv", old, U)[:, None] + added
                want[t] = np.einsum("hkv,hk->hv", states[s], R)
            else:
                want[t] = np.einsum("hkv,hk->hv", old, R) + bonus[t][:, None] * V
                states[s] = D[..., None] * old + added
        at += run
    slots = [4, 0, 2][: len(runs)]
    runner, cache, ctx = device_context(runs, slots, ((heads, dk, dv),), {"delta_portions": portions})
    state = cache.states[0][0]
    untouched = state.clone().normal_()
    state.copy_(untouched)
    state[slots] = torch.from_numpy(start).cuda()
    out = torch.full((n, heads * dv), float("nan"), device="cuda")
    if general:
        ops.delta_general_recurrence(ctx, *(on_device(a) for a in (r, k, v, w, au, u)), state, out, heads, dk, dv)
    else:
        ops.wkv_recurrence(ctx, *(on_device(a) for a in (r, k, v, bonus, w)), state, out, heads, dk, dv)
    runner.check()
    # States and read-outs here are sums of a few hundred products of order one over dk channels: errors go with the whole's size.
    for got, wanted in ((out.double().cpu().numpy().reshape(want.shape), want), (state[slots].double().cpu().numpy(), states)):
        np.testing.assert_allclose(got, wanted, rtol=2e-5, atol=2e-6 * np.sqrt(np.mean(wanted**2)) * np.sqrt(dk) + 2e-5)
    others = [slot for slot in range(state.shape[0]) if slot not in slots]
    assert torch.equal(state[others], untouched[others])


MEMORY_SIZES = [
    (2, 128, 128, (97, 32, 1)),
    (3, 33, 17, (31, 65)),
    (1, 64, 70, (127,)),
    (2, 16, 130, (96, 95, 98)),
]


@pytest.mark.parametrize("heads,dk,dv,runs", MEMORY_SIZES)
@pytest.mark.parametrize("portions", ["chunks", "tokens"])
def test_the_matrix_memory(heads, dk, dv, runs, portions):
    """Given projections over portions that continue states: gates from nearly shut to wide open, the state, its normaliser and the
    running maximum read back, the states of other requests untouched."""
    from llm_inference_b200.parts import ops

    n, cap, eps = sum(runs), 9.0, 1e-6
    rng = np.random.default_rng(dk + dv)
    widths = [heads * dk, heads * dk, heads * dv, heads * dv, heads, heads]
    columns = tuple(int(c) for c in np.cumsum([0] + widths[:-1]))
    proj = rng.normal(size=(n, sum(widths)))
    proj[:, columns[4] : columns[5]] *= 6.0
    proj[:, columns[5] :] = proj[:, columns[5] :] * 6.0 + 3.0
    bias = rng.normal(size=(2, heads))
    norm = 1.0 + rng.normal(0, 0.2, heads * dv)
    start = [rng.normal(size=(len(runs), heads, dk, dv)), rng.normal(size=(len(runs), heads, dk)), rng.normal(size=(len(runs), heads))]
    proj, bias, norm, *start = (a.astype(np.float32) for a in (proj, bias, norm, *start))
    q, k, v, gate, i_log, f_log = (proj[:, c : c + w].astype(np.float64) for c, w in zip(columns, widths))
    q, k, v = q.reshape(n, heads, dk) * dk**-0.5, k.reshape(n, heads, dk), v.reshape(n, heads, dv)
    i_log = cap * np.tanh((i_log + bias[0]) / cap)
    f_log = -np.logaddexp(0.0, -cap * np.tanh((f_log + bias[1]) / cap))
    S, N, M = (a.astype(np.float64) for a in start)
    want, weak, at = np.zeros((n, heads, dv)), np.zeros((n, heads)), 0
    for s, run in enumerate(runs):
        for t in range(at, at + run):
            top = np.maximum(f_log[t] + M[s], i_log[t])
            keep, put = np.exp(f_log[t] + M[s] - top), np.exp(i_log[t] - top)
            M[s] = top
            S[s] = keep[:, None, None] * S[s] + put[:, None, None] * k[t][..., None] * v[t][:, None]
            N[s] = keep[:, None] * N[s] + put[:, None] * k[t]
            want[t] = np.einsum("hkv,hk->hv", S[s], q[t])
            # What a head's norm leaves of rounding: its read-out's size against the terms it was summed from.
            weak[t] = np.linalg.norm(S[s], axis=(1, 2)) * np.linalg.norm(q[t], axis=-1) / np.linalg.norm(want[t], axis=-1)
            want[t] /= np.maximum(np.abs((N[s] * q[t]).sum(-1)), np.exp(-top))[:, None]
        at += run
    want = want / np.sqrt((want**2).mean(-1, keepdims=True) + eps)
    want = want * norm.reshape(heads, dv) / (1.0 + np.exp(-gate.reshape(n, heads, dv)))
    slots = [4, 0, 2][: len(runs)]
    runner, cache, ctx = device_context(runs, slots, ((heads, dk, dv), (heads, dk), (heads,)), {"delta_portions": portions})
    state = cache.states[0]
    untouched = [array.normal_().clone() for array in state]
    for array, own in zip(state, start):
        array[slots] = torch.from_numpy(own).cuda()
    out = torch.full((n, heads * dv), float("nan"), device="cuda")
    device = [torch.from_numpy(a).cuda() for a in (proj, bias, norm)]
    ops.mlstm(ctx, device[0], columns, device[1][0], device[1][1], cap, state, heads, dk, dv, device[2], eps, out)
    runner.check()
    got = out.double().cpu().numpy().reshape(want.shape)
    assert np.all(np.abs(got - want).max(-1) <= 2e-5 * (1.0 + weak) * (1.0 + np.abs(want).max(-1)))
    for array, wanted in zip(state, (S, N, M)):
        np.testing.assert_allclose(array[slots].double().cpu().numpy(), wanted, rtol=2e-5, atol=2e-5)
    others = [slot for slot in range(state[0].shape[0]) if slot not in slots]
    for array, before in zip(state, untouched):
        assert torch.equal(array[others], before[others])


def test_portions_whose_scratch_would_be_too_large_go_token_by_token(monkeypatch):
    from llm_inference_b200.parts import ops

    heads, dk, dv, n = 2, 64, 64, 160
    torch.manual_seed(3)
    r, k, w, v, bonus = (torch.rand(n, heads * width, device="cuda") for width in (dk, dk, dk, dv, 1))

    def run(choice):
        runner, cache, ctx = device_context((n,), (1,), ((heads, dk, dv),), {"delta_portions": choice})
        cache.states[0][0].zero_()
        out = torch.empty(n, heads * dv, device="cuda")
        ops.wkv_recurrence(ctx, r, k, v, bonus, w, cache.states[0][0], out, heads, dk, dv)
        runner.check()
        return out

    tokens, chunks = run("tokens"), run("chunks")
    assert torch.equal(run("auto"), chunks) and not torch.equal(chunks, tokens)
    monkeypatch.setattr(ops, "CHUNK_SCRATCH_BYTES", 1 << 10)
    assert torch.equal(run("auto"), tokens)
