"""From which length on a rule's prompt portions run in chunks: two rules go over later where a step holds many (request, head) chains."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch


@pytest.mark.parametrize("requests,decoding,heads,line", [(1, 0, 24, 256), (3, 0, 24, 256), (4, 0, 24, 512), (1, 0, 80, 256), (2, 0, 80, 512), (65, 63, 24, 256), (67, 63, 24, 512)])
def test_many_chains_go_over_later(requests, decoding, heads, line, monkeypatch):
    from llm_inference_b200.parts import ops

    asked = []
    monkeypatch.setattr(ops, "_chunk_scratch", lambda ctx, rule, longer_than, *sizes: (asked.append((rule, longer_than)), (None, ctx.num_seqs))[1])
    ctx = SimpleNamespace(num_seqs=requests, num_decode_seqs=decoding)
    rows = torch.zeros(1, 1)
    general = ops._linear_chunks(ctx, rows, rows, rows, rows, rows, rows, None, rows, rows, heads, 64, 64)
    wkv = ops._linear_chunks(ctx, rows, rows, rows, rows, None, None, rows, rows, rows, heads, 64, 64)
    assert general == wkv == requests  # nothing ran in chunks: all are left to be walked
    assert asked == [(ops._GENERAL_DELTA, line), (ops._LINEAR, ops.LINEAR_CHUNK_FROM)]
    assert ops._chunk_from(ctx, ops.MEMORY_CHUNK_FROM, heads) == line
