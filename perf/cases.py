"""Work that users of the engine have it do, one case at a time: whole decode steps, and single layers of the designs it runs.

A case is a layer of one of the architectures (the Qwen2.5 shapes and the six designs, at the layer sizes that ``bench.py``
uses) fed a step's tokens, or a whole decode step of a model. ``prepare`` builds the part or model from seeded weights and
lays the step out, ``run`` is one pass, ``exact`` is the same computation in 64 bits without the engine.

The weights that steer decays are drawn as such models start out (slow and fast channels side by side), and so are those of a
whole model that add into its stream; everything else as the engine's own random weights: N(0, 0.02), norm scales around one.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from llm_inference_b200.cache import PagedCache
from llm_inference_b200.cli.presets import PRESETS
from llm_inference_b200.config import parse_config
from llm_inference_b200.csrc.library import kernels
from llm_inference_b200.engine.runner import ModelRunner, StepEntry
from llm_inference_b200 import models  # noqa: F401  (registers the architectures)
from llm_inference_b200.parts import PartSpec, build_part
from llm_inference_b200.parts.context import CacheView, HostBatch, StepContext, Workspace
from llm_inference_b200.parts.model import Model

DEVICE = "cuda:0"
PAGE = 64
# Layer sizes by width: heads of 128, key/value heads, width of a dense feed-forward.
SIZES = {1536: (12, 2, 8960), 2048: (16, 4, 5632), 5120: (40, 8, 13824)}
DECAY_RANK = 64
TAPS = 4
EXPERTS, TOP, GROUPS, KEPT_GROUPS, ROUTE_SCALE, CLAMP = 32, 4, 4, 2, 2.0, 7.0
RANK, ROTATED = 512, 64
GATE_CAP = 10.0
EPS = 1e-5
STEP_MODEL = "qwen2.5-1.5b"
STEPS_BEFORE = 4  # decode steps that a request has behind it when the timed one runs (the first ones of an engine are not replayed)

RECURRENT = ("channel_delta", "head_delta", "wkv", "general_delta", "matrix_memory")


def listed() -> list[dict]:
    return [
        # A chat with one user: one decoded token after a prompt of 2,048, the whole Qwen2.5-1.5B. Latency counts.
        dict(name="decode_step_1", kind="decode_step", requests=1, context=2040),
        # A loaded server of the same model: 64 requests, one token each.
        dict(name="decode_step_64", kind="decode_step", requests=64, context=1000),
        # The attention layer of Qwen2.5-14B in a continuous-batching step: 63 decoding requests beside a prompt portion of 512.
        dict(name="serving_mix_attention", kind="attention", width=5120, tokens=512, requests=1, before=1100, decoding=63, dtype="bfloat16"),
        # The feed-forward of Qwen2.5-1.5B on a prompt of 2,048 tokens.
        dict(name="feed_forward_2048", kind="swiglu", width=1536, tokens=2048, dtype="bfloat16"),
        # The true 32-bit path (replay of a recorded prompt): attention layer of the 1.5B shape.
        dict(name="attention_float32", kind="attention", width=1536, tokens=500, requests=1, before=0, decoding=0, dtype="float32"),
        # Gunedra: attention over cached latents, a prompt of 2,048 tokens.
        dict(name="latent_attention_2048", kind="latent_attention", width=1536, tokens=2048, requests=1, before=0),
        # Gunedra: delta rule with a decay per channel, the same prompt.
        dict(name="channel_delta_2048", kind="channel_delta", width=1536, tokens=2048, requests=1, continued=False),
        # Tosipel: delta rule with one decay per head, the same prompt.
        dict(name="head_delta_2048", kind="head_delta", width=1536, tokens=2048, requests=1, continued=False),
        # Tunadra: the recurrent mixer, three prompts of different lengths in one step.
        dict(name="wkv_ragged", kind="wkv", width=1536, tokens=1999, requests=3, continued=False),
        # Lerorax: the generalized delta rule, a prompt of 2,048 tokens.
        dict(name="general_delta_2048", kind="general_delta", width=1536, tokens=2048, requests=1, continued=False),
        # Dugalix: the matrix memory, a prompt portion of 512 in the middle of a prompt.
        dict(name="matrix_memory_portion", kind="matrix_memory", width=1536, tokens=512, requests=1, continued=True),
        # Tunadra: routed experts on a prompt whose length is a multiple of nothing.
        dict(name="routed_experts_1777", kind="routed_experts", width=1536, tokens=1777),
    ]


def draw(rng) -> dict:
    """Another case of the same ranges: prompt portions of 100 to 2,048 tokens, decode steps of 1 to 64 requests."""

    def spread(low: int, high: int) -> int:
        return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))

    kind = rng.choice(("decode_step", "attention", "swiglu", "latent_attention", "routed_experts") + RECURRENT)
    if kind == "decode_step":
        requests = spread(1, 64)
        return dict(kind=kind, requests=requests, context=spread(100, min(2040, 64000 // requests)))
    tokens = spread(100, 2048)
    width = rng.choice((1536, 2048))
    if kind == "swiglu":
        dtype = rng.choice(("bfloat16", "float32"))
        return dict(kind=kind, width=width, tokens=min(tokens, 500) if dtype == "float32" else tokens, dtype=dtype)
    if kind == "routed_experts":
        return dict(kind=kind, width=width, tokens=tokens)
    requests = rng.choice((1, 1, 2, 5))
    if kind == "attention":
        if rng.random() < 0.3:
            return dict(kind=kind, width=1536, tokens=min(tokens, 500), requests=requests, before=0, decoding=0, dtype="float32")
        return dict(kind=kind, width=rng.choice((1536, 2048, 5120)), tokens=min(tokens, 512), requests=requests, before=rng.randint(0, 1500),
                    decoding=spread(1, 63), dtype="bfloat16")
    if kind == "latent_attention":
        return dict(kind=kind, width=width, tokens=tokens, requests=requests, before=rng.choice((0, rng.randint(1, 1000))))
    return dict(kind=kind, width=width, tokens=tokens, requests=requests, continued=rng.random() < 0.5)


# --- what a case consists of ---------------------------------------------------------------------


def split(total: int, parts: int) -> list[int]:
    """``total`` tokens over ``parts`` requests of different lengths."""
    shares = [1.0 + 0.7 * math.cos(2.3 * i) for i in range(parts)]
    lengths = [max(1, int(total * s / sum(shares))) for s in shares]
    lengths[0] += total - sum(lengths)
    return lengths


def layout(case: dict) -> tuple[list[int], list[int]]:
    """(new tokens, tokens before them) of each request of the step, single decoded tokens first."""
    if case["kind"] == "attention":
        portions = split(case["tokens"], case["requests"])
        behind = [200 + (case["before"] + 600 + 613 * i) % 3400 for i in range(case["decoding"])]
        return [1] * case["decoding"] + portions, behind + [case["before"]] * len(portions)
    if case["kind"] == "latent_attention":
        portions = split(case["tokens"], case["requests"])
        return portions, [case["before"]] * len(portions)
    if case["kind"] in RECURRENT:
        return split(case["tokens"], case["requests"]), [100 if case["continued"] else 0] * case["requests"]
    return [case["tokens"]], [0]


def contexts(case: dict) -> list[int]:
    """Tokens each request of a decode step holds before the steps in front of the timed one."""
    lengths = [max(16, int(case["context"] * (1.0 - 0.1 * math.sin(1.7 * i) ** 2))) for i in range(case["requests"])]
    # An engine replays a step it has captured for this many keys; all steps of a case stay inside one such range.
    return [n - 16 if n <= 1024 < n + 8 or n <= 2048 < n + 8 else n for n in lengths]


class Draw:
    """Tensors from one seed, each by its own name."""

    def __init__(self, seed: int) -> None:
        self.seed = seed
        self.count = 0

    def generator(self) -> torch.Generator:
        self.count += 1
        return torch.Generator(device=DEVICE).manual_seed((self.seed * 1000003 + self.count * 7919) % (1 << 62))

    def normal(self, *shape: int, std: float = 0.02, mean: float = 0.0, dtype=torch.bfloat16) -> torch.Tensor:
        values = torch.empty(shape, dtype=torch.float32, device=DEVICE)
        return values.normal_(mean, std, generator=self.generator()).to(dtype)

    def uniform(self, *shape: int, low: float, high: float, dtype=torch.bfloat16) -> torch.Tensor:
        return torch.empty(shape, dtype=torch.float32, device=DEVICE).uniform_(low, high, generator=self.generator()).to(dtype)

    def integers(self, high: int, *shape: int) -> torch.Tensor:
        return torch.randint(0, high, shape, generator=self.generator(), device=DEVICE, dtype=torch.int32)


def softplus_inverse(y: torch.Tensor) -> torch.Tensor:
    return y + torch.log(-torch.expm1(-y))


def part_weights(case: dict, d: Draw) -> dict[str, torch.Tensor]:
    kind, width = case["kind"], case["width"]
    heads, kv_heads, ff = SIZES[width]
    w: dict[str, torch.Tensor] = {}
    if kind == "attention":
        for name, rows in (("q_proj", heads * 128), ("k_proj", kv_heads * 128), ("v_proj", kv_heads * 128)):
            w[name + ".weight"], w[name + ".bias"] = d.normal(rows, width), d.normal(rows)
        w["o_proj.weight"] = d.normal(width, heads * 128)
    elif kind == "swiglu":
        w["gate_proj.weight"], w["up_proj.weight"], w["down_proj.weight"] = d.normal(ff, width), d.normal(ff, width), d.normal(width, ff)
    elif kind == "latent_attention":
        w["q"], w["dkv"], w["dkv.norm"] = d.normal(heads * (128 + ROTATED), width), d.normal(RANK + ROTATED, width), d.normal(RANK, mean=1.0)
        w["uk"], w["uv"], w["o"] = d.normal(heads * 128, RANK), d.normal(heads * 128, RANK), d.normal(width, heads * 128)
        w["sink"], w["g"] = d.normal(heads), d.normal(heads, width)
    elif kind in ("channel_delta", "head_delta"):
        kvh = heads if kind == "channel_delta" else heads // 2
        for name, rows in (("q", kvh * 128), ("k", kvh * 128), ("v", heads * 128)):
            w[name], w[name + ".conv"] = d.normal(rows, width), d.normal(rows, TAPS, mean=0.5)
        w["b"], w["norm"], w["o"] = d.normal(heads, width), d.normal(128, mean=1.0), d.normal(width, heads * 128)
        w["A_log"] = torch.log(d.uniform(heads, low=1.0, high=16.0, dtype=torch.float32)).bfloat16()
        steps = heads * 128 if kind == "channel_delta" else heads
        w["dt_bias"] = softplus_inverse(torch.exp(d.uniform(steps, low=math.log(1e-3), high=math.log(0.1), dtype=torch.float32))).bfloat16()
        if kind == "channel_delta":
            for pair, rows in (("a", heads * 128), ("g", heads * 128)):
                w[pair + "1"], w[pair + "2"] = d.normal(DECAY_RANK, width), d.normal(rows, DECAY_RANK)
        else:
            w["a"], w["g"] = d.normal(heads, width), d.normal(heads * 128, width)
    elif kind == "wkv":
        for name in "rkvgw":
            w["mu." + name] = d.normal(width, mean=0.5)
        for name in "rkvg":
            w[name] = d.normal(width, width)
        w["w1"], w["w2"], w["w0"] = d.normal(DECAY_RANK, width), d.normal(width, DECAY_RANK), d.uniform(width, low=-6.0, high=-1.0)
        w["u"], w["norm"], w["o"] = d.normal(width // 64, 64, std=0.3), d.normal(width, mean=1.0), d.normal(width, width)
    elif kind == "general_delta":
        for name in ("r", "k", "v", "a", "g"):
            w[name] = d.normal(width, width)
        w["a.b"], w["w1"], w["w2"] = d.normal(width), d.normal(DECAY_RANK, width), d.normal(width, DECAY_RANK)
        w["w0"], w["norm"], w["o"] = d.uniform(width, low=-6.0, high=0.0), d.normal(width, mean=1.0), d.normal(width, width)
    elif kind == "matrix_memory":
        for name, rows in (("q", heads * 128), ("k", heads * 128), ("v", heads * 128), ("g", heads * 128), ("i", heads), ("f", heads)):
            w[name] = d.normal(rows, width)
        w["i.b"], w["f.b"] = d.normal(heads), d.uniform(heads, low=2.0, high=6.0)
        w["norm"], w["o"] = d.normal(heads * 128, mean=1.0), d.normal(width, heads * 128)
    elif kind == "routed_experts":
        w["router"] = d.normal(EXPERTS, width)
        for name, size in [(f"e{e}", ff // 8) for e in range(EXPERTS)] + [("shared", ff // 2)]:
            w[name + ".gate"], w[name + ".up"], w[name + ".down"] = d.normal(size, width), d.normal(size, width), d.normal(width, size)
    return w


def part_spec(case: dict) -> tuple[str, PartSpec]:
    kind, width = case["kind"], case["width"]
    heads, kv_heads, ff = SIZES[width]
    if kind == "attention":
        return "mixer", PartSpec("gqa_attention", dict(prefix="", hidden_size=width, q_heads=heads, kv_heads=kv_heads, head_dim=128,
                                                       position=PartSpec("rotary", dict(head_dim=128, theta=1e6))))
    if kind == "swiglu":
        return "feed_forward", PartSpec("swiglu", dict(prefix="", hidden_size=width, intermediate_size=ff))
    if kind == "latent_attention":
        position = PartSpec("rotary", dict(head_dim=ROTATED, theta=1e6, rotary_dims=ROTATED, interleaved=True))
        return "mixer", PartSpec("latent_attention", dict(prefix="", hidden_size=width, heads=heads, dim=128, rot_dim=ROTATED, vdim=128, rank=RANK,
                                                          scale=192**-0.5, eps=EPS, position=position))
    if kind in ("channel_delta", "head_delta"):
        kvh = heads if kind == "channel_delta" else heads // 2
        return "mixer", PartSpec(kind, dict(prefix="", hidden_size=width, heads=heads, kv_heads=kvh, dim=128, vdim=128, taps=TAPS, eps=EPS))
    if kind in ("wkv", "general_delta"):
        return "mixer", PartSpec(kind, dict(prefix="", hidden_size=width, heads=width // 64, dim=64, eps=EPS))
    if kind == "matrix_memory":
        return "mixer", PartSpec(kind, dict(prefix="", hidden_size=width, heads=heads, dim=128, vdim=128, gate_cap=GATE_CAP, eps=EPS))
    return "feed_forward", PartSpec("routed_experts", dict(
        prefix="", hidden_size=width, experts=EXPERTS, top=TOP, intermediate_size=ff // 8, limit=CLAMP, route_scale=ROUTE_SCALE,
        group_count=GROUPS, group_keep=KEPT_GROUPS, shared_size=ff // 2))


def past(case: dict, d: Draw) -> list[torch.Tensor]:
    """What the cache holds in front of the step: key/value rows of every request, or the per-request state."""
    kind, width = case["kind"], case["width"]
    heads, kv_heads, _ = SIZES[width]
    runs, starts = layout(case)
    n = len(runs)
    dtype = torch.float32 if case.get("dtype") == "float32" else torch.bfloat16
    if kind in ("attention", "latent_attention"):
        rows = (kv_heads, PAGE, 128) if kind == "attention" else (1, PAGE, RANK + ROTATED)
        pages = sum(-(-(r + s) // PAGE) for r, s in zip(runs, starts)) + 1
        return [d.normal(pages, *rows, std=0.8, dtype=dtype) for _ in range(2 if kind == "attention" else 1)]
    scale = 1.0 if case.get("continued") else 0.0
    f32 = torch.float32
    if kind in ("channel_delta", "head_delta"):
        kvh = heads if kind == "channel_delta" else heads // 2
        return [d.normal(n, heads, 128, 128, std=0.1 * scale, dtype=f32), d.normal(n, TAPS - 1, (2 * kvh + heads) * 128, std=0.8 * scale)]
    if kind == "wkv":
        return [d.normal(n, width // 64, 64, 64, std=scale, dtype=f32), d.normal(n, width, std=scale)]
    if kind == "general_delta":
        return [d.normal(n, width // 64, 64, 64, std=scale, dtype=f32)]
    return [d.normal(n, heads, 128, 128, std=scale, dtype=f32), d.normal(n, heads, 128, std=scale, dtype=f32),
            d.uniform(n, heads, low=0.0, high=2.0 * scale, dtype=f32)]


def page_order(case: dict) -> list[list[int]]:
    """The pages of each request, scattered over the arena."""
    runs, starts = layout(case)
    need = [-(-(r + s) // PAGE) for r, s in zip(runs, starts)]
    order = np.random.default_rng(5).permutation(sum(need)).tolist()
    tables, at = [], 0
    for count in need:
        tables.append(order[at : at + count])
        at += count
    return tables


def inputs(case: dict, d: Draw) -> torch.Tensor:
    return d.normal(sum(layout(case)[0]), case["width"], std=1.0, dtype=torch.float32 if case.get("dtype") == "float32" else torch.bfloat16)


def step_config():
    return parse_config(dict(PRESETS[STEP_MODEL]))


def step_weights(raw: dict, d: Draw) -> dict[str, torch.Tensor]:
    hidden, heads, kv_heads, inter = (raw[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "intermediate_size"))
    dim = hidden // heads
    w = {"model.embed_tokens.weight": d.normal(raw["vocab_size"], hidden), "model.norm.weight": d.normal(hidden, mean=1.0)}
    into_stream = 0.02 / math.sqrt(2 * raw["num_hidden_layers"])  # what adds into the residual stream starts out smaller, by the number of additions
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, rows in (("q_proj", heads * dim), ("k_proj", kv_heads * dim), ("v_proj", kv_heads * dim)):
            w[p + f"self_attn.{name}.weight"], w[p + f"self_attn.{name}.bias"] = d.normal(rows, hidden), d.normal(rows)
        w[p + "self_attn.o_proj.weight"] = d.normal(hidden, heads * dim, std=into_stream)
        for name, shape, std in (("gate_proj", (inter, hidden), 0.02), ("up_proj", (inter, hidden), 0.02), ("down_proj", (hidden, inter), into_stream)):
            w[p + f"mlp.{name}.weight"] = d.normal(*shape, std=std)
        for name in ("input_layernorm", "post_attention_layernorm"):
            w[p + name + ".weight"] = d.normal(hidden, mean=1.0)
    return w


def step_tokens(case: dict, raw: dict, d: Draw) -> list[list[int]]:
    """Each request's token ids: its prompt, the steps in front, and the token that the timed step feeds."""
    return [d.integers(raw["vocab_size"], n + STEPS_BEFORE + 1).tolist() for n in contexts(case)]


# --- the calls that are measured -----------------------------------------------------------------


def prepare(case: dict, seed: int) -> dict:
    return prepare_step(case, seed) if case["kind"] == "decode_step" else prepare_part(case, seed)


def prepare_step(case: dict, seed: int) -> dict:
    entry, config = step_config()
    raw, d = PRESETS[STEP_MODEL], Draw(seed)
    model = Model(entry.recipe(config))
    model.load(step_weights(raw, d), torch.bfloat16, torch.device(DEVICE))
    tokens = step_tokens(case, raw, d)
    batch, budget = len(tokens), 4096
    pages = sum(-(-len(t) // PAGE) + 1 for t in tokens)
    cache = PagedCache(model.cache_specs(), dtype=torch.bfloat16, device=DEVICE, page_size=PAGE, max_num_sequences=batch, max_model_length=4096,
                       step_tokens=budget, num_pages=pages)
    runner = ModelRunner(model, cache, max_batch_tokens=budget, options={"workspace_rows": budget})
    ids = list(range(1, batch + 1))
    entries: list[StepEntry] = []
    for rid, row in zip(ids, tokens):
        cache.open(rid)
        prompt = row[: -STEPS_BEFORE - 1]
        if entries and sum(len(e.tokens) for e in entries) + len(prompt) > budget:
            runner.step(entries)
            entries = []
        entries.append(StepEntry(rid, prompt))
    runner.step(entries)
    for j in range(STEPS_BEFORE):
        runner.step([StepEntry(rid, (row[j - STEPS_BEFORE - 1],), (0,)) for rid, row in zip(ids, tokens)], check=j == 0)
    feed = torch.tensor([row[-1] for row in tokens], dtype=torch.int32, device=DEVICE)
    return dict(runner=runner, ids=ids, feed=feed)


def prepare_part(case: dict, seed: int) -> dict:
    d = Draw(seed)
    device = torch.device(DEVICE)
    dtype = torch.float32 if case.get("dtype") == "float32" else torch.bfloat16
    part = build_part(*part_spec(case))
    part.load(part_weights(case, d), dtype, device)
    held, h = past(case, d), inputs(case, d)
    runs, starts = layout(case)
    n = len(runs)
    q_start = np.concatenate([[0], np.cumsum(runs)[:-1]])
    arrays = dict(
        token_ids=np.zeros(sum(runs)), positions=np.concatenate([np.arange(s, s + r) for r, s in zip(runs, starts)]),
        token_seq=np.repeat(np.arange(n), runs), seq_q_start=q_start, seq_q_len=np.array(runs), seq_kv_len=np.array(runs) + np.array(starts),
        seq_slot=np.arange(n), logit_rows=np.zeros(0),
    )
    arrays = {k: v.astype(np.int32) for k, v in arrays.items()}
    ctx = StepContext(
        lib=kernels(), dtype=dtype, device=device, num_tokens=sum(runs), num_seqs=n, host=HostBatch(**arrays), workspace=Workspace(device),
        err=torch.zeros(1, dtype=torch.int32, device=device), num_decode_seqs=case.get("decoding", 0),
        max_kv_len=int(arrays["seq_kv_len"].max()), max_q_len=max(runs), **{k: torch.from_numpy(v).to(device) for k, v in arrays.items()},
    )
    view = None
    if case["kind"] in ("attention", "latent_attention"):
        tables = page_order(case)
        table = np.zeros((n, max(map(len, tables))), dtype=np.int32)
        for row, pages in zip(table, tables):
            row[: len(pages)] = pages
        view = CacheView(0, keys=held[0], values=held[1] if len(held) > 1 else None, block_table=torch.from_numpy(table).to(device),
                         num_pages=held[0].shape[0], max_pages=table.shape[1], page_size=PAGE)
    elif case["kind"] in RECURRENT:
        view = CacheView(0, state=held)
    return dict(part=part, ctx=ctx, view=view, h=h, held=held)


def run(state: dict):
    if "runner" in state:
        # One decode step over the requests, as the engine launches it; nothing is committed, so the same step can run again.
        return state["runner"].step_ahead(state["ids"], state["feed"]).logits
    if state["view"] is None:
        return state["part"].forward(state["ctx"], state["h"])
    return state["part"].forward(state["ctx"], state["view"], state["h"]), state["held"]


# --- what a pass cannot do without ---------------------------------------------------------------


def work(case: dict) -> dict:
    if case["kind"] == "decode_step":
        raw = PRESETS[STEP_MODEL]
        hidden, layers, inter, vocab = (raw[k] for k in ("hidden_size", "num_hidden_layers", "intermediate_size", "vocab_size"))
        dim = hidden // raw["num_attention_heads"]
        kv = raw["num_key_value_heads"] * dim
        weights = layers * (hidden * (2 * hidden + 2 * kv + 3 * inter)) + vocab * hidden
        keys = sum(contexts(case)) + (STEPS_BEFORE + 1) * case["requests"]
        return dict(bytes=2.0 * weights + 4.0 * layers * keys * kv + 4.0 * case["requests"] * vocab,
                    flops=2.0 * weights * case["requests"] + 4.0 * layers * keys * hidden)
    kind, width = case["kind"], case["width"]
    heads, kv_heads, ff = SIZES[width]
    size = 4 if case.get("dtype") == "float32" else 2
    runs, starts = layout(case)
    tokens, n = sum(runs), len(runs)
    io = 2.0 * size * tokens * width
    seen = sum(r * s + r * (r + 1) / 2 for r, s in zip(runs, starts))  # (query, key) pairs
    keys = sum(r + s for r, s in zip(runs, starts))
    inner = heads * 128
    if kind == "attention":
        weights = width * (2 * inner + 2 * kv_heads * 128)
        return dict(bytes=io + size * (weights + 2.0 * keys * kv_heads * 128), flops=2.0 * tokens * weights + 4.0 * seen * inner)
    if kind == "swiglu":
        return dict(bytes=io + size * 3.0 * width * ff, flops=6.0 * tokens * width * ff)
    if kind == "latent_attention":
        weights = width * (heads * (128 + ROTATED) + RANK + ROTATED + inner + heads) + 2 * inner * RANK
        return dict(bytes=io + 2.0 * (weights + keys * (RANK + ROTATED)),
                    flops=2.0 * tokens * weights + 2.0 * seen * heads * (128 + ROTATED + 128))
    if kind == "routed_experts":
        used = min(EXPERTS, TOP * tokens)
        return dict(bytes=io + 2.0 * width * (EXPERTS + 3 * used * (ff // 8) + 3 * (ff // 2)),
                    flops=2.0 * tokens * width * (EXPERTS + 3 * TOP * (ff // 8) + 3 * (ff // 2)))
    if kind in ("channel_delta", "head_delta"):
        qk = inner if kind == "channel_delta" else inner // 2
        low = 2 * DECAY_RANK * (width + inner) if kind == "channel_delta" else width * (heads + inner)
        weights = width * (2 * qk + inner + heads + inner) + low
        per_state, state = 7.0, inner * 128
    elif kind in ("wkv", "general_delta"):
        weights = width * width * (5 if kind == "wkv" else 6) + 2 * DECAY_RANK * width
        per_state, state = (5.0 if kind == "wkv" else 7.0), width * 64
    else:
        weights = width * (4 * inner + 2 * heads) + inner * width
        per_state, state = 5.0, inner * 128
    return dict(bytes=io + 2.0 * weights + 8.0 * n * state, flops=2.0 * tokens * weights + per_state * tokens * state)


def tolerance(case: dict) -> dict:
    """About four times what two orders of the same sums differ by (the tuned kernels beside the plain ones, products beside
    64-bit ones): 28 layers of bfloat16 2.6e-2 (as far as either is from 64 bits, and no four times of it is stated), attention
    3.9e-3, a layer's other parts 1.4e-3, 32-bit 2e-6."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    if case["kind"] == "decode_step":
        return {"rel": 3e-2}
    return {"rel": 1.5e-2 if case["kind"] in ("attention", "latent_attention") else 6e-3}


# --- the same in 64 bits ---------------------------------------------------------------------------


def linear(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    y = x @ weight.double().t()
    return y if bias is None else y + bias.double()


def unit_rms(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(x: torch.Tensor) -> torch.Tensor:
    return x * torch.sigmoid(x)


def rotate(x: torch.Tensor, positions: torch.Tensor, interleaved: bool) -> torch.Tensor:
    """``[tokens, heads, dims]`` turned at ``positions``; angles are products of 32-bit numbers, as the models define them."""
    dims = x.shape[-1]
    inverse = torch.from_numpy(np.float32(1e6) ** (-np.arange(0, dims // 2, dtype=np.float32) * np.float32(2) / np.float32(dims)))
    angles = (positions.float().cpu()[:, None] * inverse[None, :]).double().to(x.device)[:, None, :]
    cos, sin = torch.cos(angles), torch.sin(angles)
    if interleaved:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cos - b * sin, b * cos + a * sin], dim=-1).flatten(-2)
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def causal_weights(scores: torch.Tensor, start: int, sink: torch.Tensor | None = None) -> torch.Tensor:
    """Softmax of ``[heads, queries, keys]``; query i sees keys up to ``start + i``, the sink counts in the denominator only."""
    queries, keys = scores.shape[-2:]
    late = torch.arange(keys, device=scores.device)[None, :] > torch.arange(start, start + queries, device=scores.device)[:, None]
    scores = scores.masked_fill(late, -math.inf)
    if sink is not None:
        scores = torch.cat([scores, sink.double()[:, None, None].expand(-1, queries, 1)], dim=-1)
    weights = torch.softmax(scores, dim=-1)
    return weights[..., :-1] if sink is not None else weights


def exact(case: dict, seed: int):
    if case["kind"] == "decode_step":
        return exact_step(case, seed)
    d = Draw(seed)
    w = part_weights(case, d)
    held, h = past(case, d), inputs(case, d).double()
    kind = case["kind"]
    if kind == "swiglu":
        return linear(silu(linear(h, w["gate_proj.weight"])) * linear(h, w["up_proj.weight"]), w["down_proj.weight"])
    if kind == "routed_experts":
        return exact_experts(w, h)
    runs, starts = layout(case)
    tables = page_order(case) if kind in ("attention", "latent_attention") else None
    outs, states, at = [], [], 0
    for i, (r, s) in enumerate(zip(runs, starts)):
        rows = h[at : at + r]
        if tables is not None:
            before = [x[tables[i]].double().transpose(1, 2).flatten(0, 1)[:s] for x in held]  # [s, heads, numbers]
            outs.append((exact_attention if kind == "attention" else exact_latent)(case, w, rows, s, before))
        else:
            out, state = {"channel_delta": exact_delta, "head_delta": exact_delta, "wkv": exact_wkv, "general_delta": exact_general,
                          "matrix_memory": exact_memory}[kind](case, w, rows, [x[i].double() for x in held])
            outs.append(out)
            states.append(state)
        at += r
    out = torch.cat(outs)
    if tables is not None:
        return out, [None] * len(held)
    return out, [torch.stack(x) for x in zip(*states)]


def grouped_attention(q, k, v, start: int, scale: float) -> torch.Tensor:
    """``q [tokens, heads, dim]`` over ``k, v [keys, kv heads, dim]``."""
    share = q.shape[1] // k.shape[1]
    out = torch.empty_like(q)
    for g in range(k.shape[1]):
        mine = slice(g * share, (g + 1) * share)
        weights = causal_weights(torch.einsum("thd,kd->htk", q[:, mine], k[:, g]) * scale, start)
        out[:, mine] = torch.einsum("htk,kd->thd", weights, v[:, g])
    return out


def exact_attention(case, w, h, start, before):
    heads, kv_heads, _ = SIZES[case["width"]]
    positions = torch.arange(start, start + h.shape[0], device=h.device)
    q, k, v = (linear(h, w[n + ".weight"], w[n + ".bias"]).view(h.shape[0], -1, 128) for n in ("q_proj", "k_proj", "v_proj"))
    keys = torch.cat([before[0], rotate(k, positions, False)])
    values = torch.cat([before[1], v])
    out = grouped_attention(rotate(q, positions, False), keys, values, start, 128**-0.5)
    return linear(out.flatten(1), w["o_proj.weight"])


def exact_latent(case, w, h, start, before):
    heads = SIZES[case["width"]][0]
    t = h.shape[0]
    positions = torch.arange(start, start + t, device=h.device)
    q = linear(h, w["q"]).view(t, heads, 128 + ROTATED)
    down = linear(h, w["dkv"])
    latent = unit_rms(down[:, :RANK], EPS) * w["dkv.norm"].double()
    rows = torch.cat([before[0][:, 0], torch.cat([latent, rotate(down[:, None, RANK:], positions, True)[:, 0]], dim=1)])
    q_rot = rotate(q[..., 128:], positions, True)
    gate = torch.sigmoid(linear(h, w["g"]))
    uk, uv = w["uk"].double().view(heads, 128, RANK), w["uv"].double().view(heads, 128, RANK)
    out = torch.empty(t, heads, 128, dtype=torch.float64, device=h.device)
    for n in range(heads):
        scores = (q[:, n, :128] @ uk[n] @ rows[:, :RANK].t() + q_rot[:, n] @ rows[:, RANK:].t()) * 192**-0.5
        weights = causal_weights(scores[None], start, w["sink"][n : n + 1])[0]
        out[:, n] = weights @ rows[:, :RANK] @ uv[n].t() * gate[:, n : n + 1]
    return linear(out.flatten(1), w["o"])


def exact_delta(case, w, h, held):
    """Both delta rules with a short convolution; the decay is per channel or per head."""
    heads = SIZES[case["width"]][0]
    channelwise = case["kind"] == "channel_delta"
    kvh, t = (heads if channelwise else heads // 2), h.shape[0]
    state, history = held
    raw = torch.cat([history, torch.cat([linear(h, w[n]) for n in "qkv"], dim=1)])
    taps = torch.cat([w[n + ".conv"] for n in "qkv"]).double()
    mixed = silu(sum(raw[j : j + t] * taps[:, j] for j in range(TAPS)))
    q, k, v = (x.view(t, -1, 128) for x in mixed.split([kvh * 128, kvh * 128, heads * 128], dim=1))
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    share = heads // kvh
    q, k = ((unit(x) * s).repeat_interleave(share, dim=1) for x, s in ((q, 128**-0.5), (k, 1.0)))
    beta = torch.sigmoid(linear(h, w["b"]))
    step = linear(linear(h, w["a1"]), w["a2"], w["dt_bias"]) if channelwise else linear(h, w["a"], w["dt_bias"])
    rate = torch.exp(w["A_log"].double())[None, :, None]
    decay = torch.exp(-rate * torch.nn.functional.softplus(step, threshold=1e9).view(t, heads, -1))
    out = torch.empty(t, heads, 128, dtype=torch.float64, device=h.device)
    for i in range(t):
        state = state * decay[i][..., None]
        u = beta[i][:, None] * (v[i] - torch.einsum("hkv,hk->hv", state, k[i]))
        state = state + k[i][..., None] * u[:, None]
        out[i] = torch.einsum("hkv,hk->hv", state, q[i])
    gate = torch.sigmoid(linear(linear(h, w["g1"]), w["g2"])) if channelwise else silu(linear(h, w["g"]))
    y = (unit_rms(out, EPS) * w["norm"].double()).flatten(1) * gate
    return linear(y, w["o"]), [state, raw[t:]]


def exact_wkv(case, w, h, held):
    t, width = h.shape
    heads = width // 64
    state, previous = held
    before = torch.cat([previous[None], h[:-1]])
    blend = {n: h + (before - h) * w["mu." + n].double() for n in "rkvgw"}
    r, k, v = (linear(blend[n], w[n]).view(t, heads, 64) for n in "rkv")
    decay = torch.exp(-torch.exp(linear(torch.tanh(linear(blend["w"], w["w1"])), w["w2"], w["w0"]))).view(t, heads, 64)
    bonus = w["u"].double()[..., None]
    out = torch.empty(t, heads, 64, dtype=torch.float64, device=h.device)
    for i in range(t):
        kv = k[i][..., None] * v[i][:, None]
        out[i] = torch.einsum("hkv,hk->hv", state + bonus * kv, r[i])
        state = decay[i][..., None] * state + kv
    y = unit_rms(out, EPS).flatten(1) * w["norm"].double() * silu(linear(blend["g"], w["g"]))
    return linear(y, w["o"]), [state, h[-1]]


def exact_general(case, w, h, held):
    t, width = h.shape
    heads = width // 64
    (state,) = held
    r, k, v = (linear(h, w[n]).view(t, heads, 64) for n in "rkv")
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(linear(torch.tanh(linear(h, w["w1"])), w["w2"], w["w0"]))).view(t, heads, 64)
    share = torch.sigmoid(linear(h, w["a"], w["a.b"])).view(t, heads, 64)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    out = torch.empty(t, heads, 64, dtype=torch.float64, device=h.device)
    for i in range(t):
        removed = (share[i] * u[i])[..., None] * torch.einsum("hkv,hk->hv", state, u[i])[:, None]
        state = decay[i][..., None] * state - removed + k[i][..., None] * v[i][:, None]
        out[i] = torch.einsum("hkv,hk->hv", state, r[i])
    y = unit_rms(out, EPS).flatten(1) * w["norm"].double() * torch.sigmoid(linear(h, w["g"]))
    return linear(y, w["o"]), [state]


def exact_memory(case, w, h, held):
    heads, t = SIZES[case["width"]][0], h.shape[0]
    state, norm, peak = held
    q, k, v = (linear(h, w[n]).view(t, heads, 128) for n in "qkv")
    q = q * 128**-0.5
    cap = lambda x: GATE_CAP * torch.tanh(x / GATE_CAP)  # noqa: E731
    put = cap(linear(h, w["i"], w["i.b"]))
    keep = -torch.nn.functional.softplus(-cap(linear(h, w["f"], w["f.b"])), threshold=1e9)
    out = torch.empty(t, heads, 128, dtype=torch.float64, device=h.device)
    for i in range(t):
        top = torch.maximum(keep[i] + peak, put[i])
        a, b = torch.exp(keep[i] + peak - top), torch.exp(put[i] - top)
        state = a[:, None, None] * state + b[:, None, None] * k[i][..., None] * v[i][:, None]
        norm = a[:, None] * norm + b[:, None] * k[i]
        peak = top
        size = torch.maximum((norm * q[i]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out[i] = torch.einsum("hkv,hk->hv", state, q[i]) / size[:, None]
    y = unit_rms(out, EPS).flatten(1) * w["norm"].double() * torch.sigmoid(linear(h, w["g"]))
    return linear(y, w["o"]), [state, norm, peak]


def exact_experts(w, h):
    def unit(name: str, x: torch.Tensor) -> torch.Tensor:
        gate = torch.clamp(linear(x, w[name + ".gate"]), max=CLAMP)
        up = torch.clamp(linear(x, w[name + ".up"]), -CLAMP, CLAMP)
        return linear(gate * torch.sigmoid(1.702 * gate) * (up + 1.0), w[name + ".down"])

    scores = torch.sigmoid(linear(h, w["router"]))
    grouped = scores.view(-1, GROUPS, EXPERTS // GROUPS)
    best = grouped.topk(2, dim=-1).values.sum(-1).topk(KEPT_GROUPS, dim=-1).indices
    allowed = torch.zeros(grouped.shape[:2], dtype=torch.bool, device=h.device).scatter_(1, best, True)
    open_ = allowed[..., None].expand_as(grouped).reshape_as(scores)
    chosen = scores.masked_fill(~open_, -1.0).topk(TOP, dim=-1)
    weights = chosen.values / (chosen.values.sum(-1, keepdim=True) + 1e-20) * ROUTE_SCALE
    out = unit("shared", h)
    for e in range(EXPERTS):
        token, place = (chosen.indices == e).nonzero(as_tuple=True)
        out[token] += weights[token, place, None] * unit(f"e{e}", h[token])
    return out


def exact_step(case, seed):
    raw, d = PRESETS[STEP_MODEL], Draw(seed)
    w = step_weights(raw, d)
    tokens = step_tokens(case, raw, d)
    heads, kv_heads, layers, eps = (raw[k] for k in ("num_attention_heads", "num_key_value_heads", "num_hidden_layers", "rms_norm_eps"))
    norm = lambda x, name: unit_rms(x, eps) * w[name + ".weight"].double()  # noqa: E731
    lengths = [len(t) for t in tokens]
    x = w["model.embed_tokens.weight"][torch.tensor(sum(tokens, []), device=DEVICE)].double()
    ends = np.cumsum(lengths).tolist()
    for i in range(layers):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm")
        q, k, v = (linear(h, w[p + f"self_attn.{n}.weight"], w[p + f"self_attn.{n}.bias"]).view(x.shape[0], -1, 128) for n in ("q_proj", "k_proj", "v_proj"))
        mixed = []
        for end, length in zip(ends, lengths):
            rows, positions = slice(end - length, end), torch.arange(length, device=DEVICE)
            mixed.append(grouped_attention(rotate(q[rows], positions, False), rotate(k[rows], positions, False), v[rows], 0, 128**-0.5))
        x = x + linear(torch.cat(mixed).flatten(1), w[p + "self_attn.o_proj.weight"])
        h = norm(x, p + "post_attention_layernorm")
        for rows in h.split(16384):
            rows.copy_(linear(silu(linear(rows, w[p + "mlp.gate_proj.weight"])) * linear(rows, w[p + "mlp.up_proj.weight"]), w[p + "mlp.down_proj.weight"]))
        x = x + h
    return linear(norm(x[torch.tensor(ends, device=DEVICE) - 1], "model.norm"), w["model.embed_tokens.weight"])
