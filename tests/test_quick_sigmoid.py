"""The sigmoid of the wide gating passes: against 64 bits from one end of its range to the other, where the quotient is no normal number, at
infinities and NaN."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

WIDTH = 64


def gate(z, sigmoid):
    """The gate alone: rows of ones have a root mean square of one."""
    from llm_inference_b200.cli.microbench import make_ctx
    from llm_inference_b200.parts import ops

    z = z.view(-1, WIDTH)
    ones = torch.ones_like(z)
    return ops.wkv_output(make_ctx(positions=[0] * z.shape[0]), ones, torch.ones(WIDTH, device="cuda"), z, 1, WIDTH, 0.0, torch.empty_like(z), sigmoid_gate=sigmoid).view(-1)


@pytest.mark.parametrize("sigmoid", [True, False])
def test_against_64_bits(sigmoid):
    torch.manual_seed(0)
    z = torch.cat([torch.linspace(-120, 120, 1 << 20, device="cuda"), torch.linspace(-88.8, -87.2, 1 << 20, device="cuda"), torch.randn(1 << 20, device="cuda")])
    got, want = gate(z, sigmoid).double(), torch.sigmoid(z.double()) * (1.0 if sigmoid else z.double())
    within = z >= -88.7  # e^-z passes the range below
    # the error that common.cuh states, an ulp of the numbers that are no normal ones, and the roundings of silu's product
    assert ((got - want).abs()[within] <= (2.1e-7 + (0.0 if sigmoid else 6e-8)) * want.abs()[within] + (1.0 if sigmoid else 89.0) * 2.0**-149).all()
    assert (got[z < -88.8] == 0).all()


def test_infinities_and_nan():
    inf = float("inf")
    z = torch.tensor([inf, -inf, float("nan"), 0.0], device="cuda").repeat(WIDTH)
    got = gate(z, True)
    assert (got[0::4] == 1).all() and (got[1::4] == 0).all() and torch.isnan(got[2::4]).all() and (got[3::4] == 0.5).all()
