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
