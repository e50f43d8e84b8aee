"""The true 32-bit product on the tensor cores: against 64 bits at the ends of its tiles and stages, nearer than chains of FMAs, the same bits for
a row whatever tile computes it, numbers of very different sizes, operands that are not finite."""

from __future__ import annotations

from ctypes import c_int

import pytest
import torch

pytestmark = pytest.mark.gpu


def product(a, w, bias=None, tokens=0):
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.csrc.library import ptr

    ctx = make_ctx(positions=[0] * a.shape[0])
    (m, k), n = a.shape, w.shape[0]
    out = torch.full((m, n), float("nan"), device="cuda")
    ctx.lib.call("b200_gemm_f32_split", ptr(a), ptr(w), ptr(bias), ptr(out), *(c_int(v) for v in (m, n, k, k, k, n, tokens)), ptr(ctx.err), ctx.stream)
    assert int(ctx.err.item()) == 0
    return out


# A part is exact; what is left out of a product is at most 2^-24 of it (2 x 2^-8 x 2^-17 and less; its sign changes from product to product unless it is
# made not to); a stage of 64 numbers ends in four roundings towards zero inside the tensor core (2^-23 each of what has been summed by then: 2.5
# of them on sums of one sign), and K / 64 stages add up with ordinary rounding. Random signs: 2^-22 and what is left out, 3e-7, with room.
CLOSE = 5e-7


@pytest.mark.parametrize("m,n,k", [(1, 128, 256), (17, 129, 260), (65, 300, 516), (130, 1000, 1028), (500, 256, 2052)])
@pytest.mark.parametrize("tokens", [16, 32, 64, 128])
def test_against_64_bits(m, n, k, tokens):
    torch.manual_seed(m + n)
    a, w, bias = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda"), torch.randn(n, device="cuda")
    want = a.double() @ w.double().T + bias.double()
    got = product(a, w, bias, tokens)
    assert ((got.double() - want).norm() / want.norm()).item() < CLOSE
    assert torch.equal(got, product(a, w, bias))


@pytest.mark.parametrize("n,k", [(2080, 260), (151, 1024)])
def test_rows_and_the_call_they_are_in(n, k):
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops

    torch.manual_seed(n)
    a, w = torch.randn(700, k, device="cuda"), torch.randn(n, k, device="cuda")
    linear = lambda x: ops.linear(make_ctx(positions=[0] * x.shape[0]), x, w, torch.empty(x.shape[0], n, device="cuda"))
    whole = linear(a)
    for rows in (1, 16, 17, 33, 64, 200):
        assert torch.equal(linear(a[:rows].contiguous()), whole[:rows]), rows


def test_sizes_far_apart_and_what_is_not_finite():
    torch.manual_seed(0)
    a = torch.randn(40, 512, device="cuda") * 10.0 ** torch.randint(-18, 18, (40, 1), device="cuda")
    w = torch.randn(200, 512, device="cuda") * 10.0 ** torch.randint(-18, 18, (200, 1), device="cuda")
    want = a.double() @ w.double().T
    got = product(a, w)
    rms = want.norm() / want.numel() ** 0.5
    scale = (a.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None])  # each output against the size of what it sums
    assert torch.isfinite(rms) and ((got.double() - want).abs() / scale).max().item() < CLOSE
    a[3, 7], w[5, 100] = float("inf"), float("nan")
    spoilt = product(a, w)
    rows, cols = torch.arange(40) != 3, torch.arange(200) != 5
    assert not torch.isfinite(spoilt[3]).any() and not torch.isfinite(spoilt[:, 5]).any()
    assert torch.equal(spoilt[rows][:, cols], got[rows][:, cols])


@pytest.mark.parametrize("operand", ["a", "w"])
@pytest.mark.parametrize("value", ["inf", "-inf", "3.4028234e38", "-3.397e38"])
@pytest.mark.parametrize("tokens", [16, 32, 64, 128])
def test_infinite_and_very_large_operands(operand, value, tokens):
    """As chains of FMAs have them: infinities with their signs, sums of very large numbers where they are finite."""
    torch.manual_seed(1)
    m, n, k = 130, 200, 516
    operands = dict(a=0.5 * torch.rand(m, k, device="cuda") - 0.25, w=torch.rand(n, k, device="cuda") - 0.5)
    bias = torch.randn(n, device="cuda")
    clean = product(*operands.values(), bias, tokens)
    operands[operand][17, 33] = float(value)
    want = operands["a"].double() @ operands["w"].double().T + bias.double()
    got = product(*operands.values(), bias, tokens).double()
    finite = torch.isfinite(want)
    assert torch.equal(got[~finite], want[~finite]) and torch.isfinite(got[finite]).all()
    assert ((got - want)[finite].norm() / want[finite].norm()).item() < CLOSE
    other = torch.ones(m if operand == "a" else n, dtype=torch.bool, device="cuda")
    other[17] = False
    assert torch.equal(got[other] if operand == "a" else got[:, other], (clean[other] if operand == "a" else clean[:, other]).double())


@pytest.mark.parametrize("small,large", [(-118, 100), (-122, 0), (-130, 60), (-142, 90)])
@pytest.mark.parametrize("operand", ["a", "w"])
def test_the_smallest_operands(operand, small, large):
    """Numbers whose last bits lie below bfloat16's smallest number, from 2^-149 on, beside ordinary and large ones."""
    torch.manual_seed(2)
    m, n, k = 33, 200, 320
    few = torch.randint(1, 1 << 24, (m, k), device="cuda").float() if small > -130 else torch.randint(1, 1 << 7, (m, k), device="cuda").float()
    tiny = torch.ldexp(few, torch.tensor(small - (24 if small > -130 else 7), device="cuda"))
    other = torch.ldexp(torch.rand(n, k, device="cuda") + 0.5, torch.tensor(large, device="cuda"))
    a, w = (tiny, other) if operand == "a" else (other, tiny)
    want = a.double() @ w.double().T
    got = product(a.contiguous(), w.contiguous())
    assert ((got.double() - want).abs() / want).max().item() < CLOSE + 2.0**-149 / want.min().item()


@pytest.mark.parametrize("k", [256, 516, 1028])
def test_what_is_left_out_with_one_sign(k):
    """1 + 2^-8 - 2^-17 splits into parts as large as they get, so every product leaves out its 2^-24, all on the same side."""
    x = 1 + 2.0**-8 - 2.0**-17
    got = product(torch.full((40, k), x, device="cuda"), torch.full((150, k), -x, device="cuda"))
    # left out, the four roundings towards zero of each stage, half an ulp for each of the K / 64 sums
    bound = 2.0**-24 + 2.5 * 2.0**-23 + (k // 64 + 1) / 2 * 2.0**-24
    assert ((got.double() + k * x * x).abs() / (k * x * x)).max().item() < bound
