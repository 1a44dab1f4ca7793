"""The activations' quotients (csrc/act.cuh) against 64 bits, over the whole range of fp32, and where the exponential overflows or the number is not finite."""
import math

import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("std", [1e-3, 0.3, 3.0, 20.0])
def test_gated_silu_is_rounded_as_a_division_is(std):
    """expf is off by up to 2 ulp and the sum, the quotient and the product with the other half by half an ulp each: 4 ulp of 2^-23 at most, wherever the result is normal."""
    g = torch.Generator(device="cuda").manual_seed(3)
    ff = 512
    gu = (torch.randn(300, 2 * ff, generator=g, device="cuda") * std).contiguous()
    out = torch.empty(300, ff, device="cuda")
    ops.gated_act(gu, ff, out, ops.ACT_SILU, up_off=ff)
    z, u = gu.double().split(ff, 1)
    want = z * torch.sigmoid(z) * u
    normal = (want.abs() > 1e-30) & (z > -80)
    assert bool(((out.double() - want).abs() <= 4 * 2.0 ** -23 * want.abs())[normal].all())


def test_silu_where_the_exponential_overflows_and_of_numbers_that_are_not_finite():
    z = torch.tensor([math.inf, -math.inf, math.nan, 0.0, 3e38, -3e38, -88.0, -88.6, -88.8, -200.0, 88.0, 1e-38, -1e-38, 16.7, -16.7, 1.0], device="cuda")
    gu = torch.cat([z, torch.ones_like(z)])[None].repeat(2, 1).contiguous()
    out = torch.empty(2, z.numel(), device="cuda")
    ops.gated_act(gu, z.numel(), out, ops.ACT_SILU, up_off=z.numel())
    want = z / (1.0 + torch.exp(-z))
    assert torch.equal(torch.isnan(out[0]), torch.isnan(want))
    assert torch.allclose(out[0].nan_to_num(nan=1.0), want.nan_to_num(nan=1.0), rtol=2.0 ** -21, atol=1e-42)


@pytest.mark.parametrize("size", [1e-28, 1e-33, 1e-36, 1e-38, 1e-41])
def test_silu_of_the_smallest_numbers(size):
    """Where 1 + exp(-z) is 2 the quotient is half of z, rounded once, subnormal numbers too."""
    g = torch.Generator(device="cuda").manual_seed(5)
    ff = 512
    z = torch.randn(40, ff, generator=g, device="cuda").double().mul(size).float()
    out = torch.empty(40, ff, device="cuda")
    ops.gated_act(torch.cat([z, torch.ones_like(z)], 1).contiguous(), ff, out, ops.ACT_SILU, up_off=ff)
    assert torch.equal(out, (z.double() / 2).float())


@pytest.mark.parametrize("dt,rows", [(torch.bfloat16, 2048), (torch.float32, 8192)])
@pytest.mark.parametrize("act", [ops.ACT_NONE, ops.ACT_RELU, ops.ACT_SILU, ops.ACT_GELU_ERF, ops.ACT_GELU_TANH, ops.ACT_RELU_SQUARED])
@pytest.mark.parametrize("up", [True, False])
def test_many_rows_give_what_few_give(dt, rows, act, up):
    """Eight columns a thread from ``rows`` rows of 1024 on, four below: the same bits, routing weights among the factors too."""
    g = torch.Generator(device="cuda").manual_seed(act)
    ff = 1024
    x = torch.randn(rows + 2, 2 * ff, generator=g, device="cuda").to(dt)
    perm = torch.arange(rows + 2, dtype=torch.int32, device="cuda")
    perm[5::7] = -1
    for kw in ({}, dict(perm=perm, wt=torch.rand(rows + 2, generator=g, device="cuda"))):
        whole, few = torch.empty(rows + 2, ff, device="cuda", dtype=dt), torch.empty(rows - 1, ff, device="cuda", dtype=dt)
        ops.gated_act(x, ff, whole, act, up_off=ff if up else -1, **kw)
        ops.gated_act(x[:rows - 1], ff, few, act, up_off=ff if up else -1, **kw)
        assert torch.equal(whole[:rows - 1], few)
