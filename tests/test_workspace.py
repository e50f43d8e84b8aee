"""Scratch that grows with prompt portions: on the CPU how it grows, on the GPU that captured decode steps outlive portions that are
longer than any before them."""

from __future__ import annotations

import pytest
import torch


def test_scratch_apart_from_captured_steps_grows_without_a_new_generation():
    from llm_inference_b200.parts.context import Workspace

    workspace = Workspace(torch.device("cpu"))
    workspace.get("tokens", (8, 4), torch.float32)
    generation, sizes = workspace.generation, set()
    limit = 6000  # bytes
    for rows in range(1, 93):  # a long prompt in portions: every one sees more keys than the one before
        view = workspace.apart("keys", (rows, 16), torch.float32, limit)
        assert tuple(view.shape) == (rows, 16) and view.is_contiguous()
        sizes.add(workspace._apart["keys:torch.float32"].numel())
    assert workspace.generation == generation and len(sizes) <= 8 and max(sizes) == limit // 4
    assert workspace.apart("keys", (3, 5), torch.float32, limit).data_ptr() == view.data_ptr()
    workspace.apart("keys", (99, 16), torch.float32, limit)  # past the limit: what is asked for and no more
    assert workspace.generation == generation and workspace.bytes() == 4 * (32 + 99 * 16)


def test_captured_steps_have_a_buffer_of_their_own():
    from types import SimpleNamespace

    from llm_inference_b200.parts.context import StepContext, Workspace

    workspace = Workspace(torch.device("cpu"))
    step = SimpleNamespace(workspace=workspace, dtype=torch.float32, captured=True)
    step.buffer = lambda *args, **kw: StepContext.buffer(step, *args, **kw)
    held = StepContext.portion_buffer(step, "scratch", (10,), torch.float32, 1 << 10)
    generation = workspace.generation
    step.captured = False
    other = StepContext.portion_buffer(step, "scratch", (200,), torch.float32, 1 << 10)
    assert workspace.generation == generation and other.data_ptr() != held.data_ptr()
    step.captured = True
    assert StepContext.portion_buffer(step, "scratch", (10,), torch.float32, 1 << 10).data_ptr() == held.data_ptr()


@pytest.mark.gpu
def test_captured_decode_steps_outlive_growing_portions():
    """A model of delta rules and latent attention whose portions run in chunks and on expanded keys."""
    import copy

    from llm_inference_b200.cache import PagedCache
    from llm_inference_b200.cli.presets import PRESETS
    from llm_inference_b200.config import parse_config
    from llm_inference_b200.engine.loading import random_model
    from llm_inference_b200.engine.runner import ModelRunner, StepEntry

    raw = copy.deepcopy(PRESETS["tosipel-small"])
    for layer in raw["layers"]:
        if layer["type"] == "latent_attention":
            layer["mixer"]["dim"] = 128
    model = random_model(parse_config(raw)[1], 3)
    cache = PagedCache(model.cache_specs(), dtype=torch.bfloat16, device=model.device, page_size=64, max_num_sequences=4, max_model_length=2048,
                       step_tokens=1024, num_pages=64)
    runner = ModelRunner(model, cache, max_batch_tokens=1024, options={"workspace_rows": 1024})
    for rid in (1, 2):
        cache.open(rid)

    def decode(count):
        for _ in range(count):
            runner.step([StepEntry(1, (7,), (0,))])

    runner.step([StepEntry(1, [5] * 20)])
    runner.step([StepEntry(2, [9] * 260)])  # every scratch of a portion has been asked for once
    decode(4)
    assert {"state_chunks", "latent_rows", "latent_expanded"} <= {key.split(":")[0] for key in runner.workspace._apart}
    held, replays = dict(runner._graphs), runner.graph_replays
    assert held and replays > 0
    for portion in (260, 270, 300, 500):  # each sees more keys, the later ones hold more tokens
        runner.step([StepEntry(2, [9] * portion)])
        decode(1)
    runner.check()
    assert runner.graph_replays == replays + 4
    assert all(runner._graphs[key] is value for key, value in held.items())
