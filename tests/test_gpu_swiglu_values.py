"""silu's fast form for every bf16 value, each in a block of its own, whose scale is then the magnitude of silu(a) * b to the last bit."""
import pytest
import torch

from gpu_util import u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [0, 60, 127, -40])      # of b: makes small products large enough for a scale of their own
def test_every_value_by_itself(exponent):
    import kernel
    from dsv3_b200 import swiglu_quant
    a = torch.zeros(65536, 128, dtype=torch.bfloat16, device="cuda")
    a[:, 0] = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)
    b = torch.full_like(a, 2.0 ** exponent)
    q, s = swiglu_quant(a, b)
    wq, ws = kernel.act_quant(torch.nn.functional.silu(a) * b)
    finite = torch.isfinite(ws.view(-1))
    assert torch.equal(s.view(-1)[finite], ws.view(-1)[finite]) and bool((~torch.isfinite(s.view(-1)[~finite])).all())
    assert (u8(q[finite]) == u8(wq[finite])).all()


@pytest.mark.parametrize("fmt", [None, "ue8m0"])
@pytest.mark.parametrize("exponent", [-40, 0, 60, 120])      # of b: scales of the smallest size, of their own, and products that overflow
def test_products_of_full_significands(exponent, fmt):
    """Every significand of silu(a) (which is a itself from 64 to 128, and a result of its own from -4 to 4) times every one of b, each
    product in a block of its own.  (Products below 2^-126 leave no trace: no scale is below 1e-4 / 448.)"""
    import kernel
    from dsv3_b200 import swiglu_quant
    bits = torch.arange(128, dtype=torch.int32, device="cuda")
    large, small = (0x4280 + bits).to(torch.int16).view(torch.bfloat16), torch.linspace(-4, 4, 128, device="cuda").bfloat16()
    b128 = ((127 + exponent) * 128 + bits).to(torch.int16).view(torch.bfloat16) * torch.where(bits % 2 == 0, 1.0, -1.0).bfloat16()
    one = torch.cat([large, small])[:, None].expand(256, 128).reshape(-1)
    a, b = (torch.zeros(256 * 128, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    a[:, 0], b[:, 0] = one, b128[None].expand(256, 128).reshape(-1)
    a[:, 64], b[:, 64] = one / 2, b[:, 0]                    # another code in the same block
    q, s = swiglu_quant(a, b, fmt)
    wq, ws = kernel.act_quant(torch.nn.functional.silu(a) * b, 128, fmt)
    finite = torch.isfinite(ws.view(-1))
    assert bool(finite.any()) and torch.equal(s.view(-1)[finite], ws.view(-1)[finite]) and bool((~torch.isfinite(s.view(-1)[~finite])).all())
    assert (u8(q[finite]) == u8(wq[finite])).all()
