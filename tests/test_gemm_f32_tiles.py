"""The true 32-bit product on both of its tiles (16 x 32 and 64 x 64 outputs): against 64 bits at ragged sizes, the same bits for a row
whichever tile computes it, batches with strides of their own, rows that are no whole 16-byte steps."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def product(a, w, out, bias=None):
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops

    return ops.linear(make_ctx(positions=[0] * a.shape[0]), a, w, out, bias)


@pytest.mark.parametrize("n,k", [(2080, 96), (1999, 33), (65, 1027), (4097, 64)])
def test_rows_have_the_same_bits_on_either_tile(n, k):
    torch.manual_seed(n)
    a, w, bias = torch.randn(1203, k, device="cuda"), torch.randn(n, k, device="cuda"), torch.randn(n, device="cuda")
    want = a.double() @ w.double().T + bias.double()
    whole = product(a, w, torch.empty(1203, n, device="cuda"), bias)
    assert (whole.double() - want).abs().max().item() < 2e-5 * math.sqrt(k)
    for rows in (1, 16, 17, 64, 100):
        some = product(a[:rows].contiguous(), w, torch.empty(rows, n, device="cuda"), bias)
        assert torch.equal(some, whole[:rows]), rows


@pytest.mark.parametrize("heads,rows,n,k,wide", [(3, 5, 40, 24, 100), (12, 300, 512, 128, 192), (2, 65, 33, 30, 61)])
def test_a_batch_with_strides(heads, rows, n, k, wide):
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops

    torch.manual_seed(rows)
    x = torch.randn(rows, heads * wide, device="cuda").view(rows, heads, wide)[:, :, :k].transpose(0, 1)
    w, out = torch.randn(heads, n, k, device="cuda"), torch.empty(heads, rows, n, device="cuda")
    ops.linear_per_head(make_ctx(positions=[0] * rows), x, w, out)
    want = torch.einsum("hrk,hnk->hrn", x.double(), w.double())
    assert (out.double() - want).abs().max().item() < 2e-5 * math.sqrt(k)
