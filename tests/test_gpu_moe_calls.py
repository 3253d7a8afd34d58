"""Forms of a call of the expert layer at the edge of what it takes."""
import pytest
import torch

from test_gpu_moe import _MoE
from test_gpu_stream import _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


def _layer_and_input(rows=24):
    g = torch.Generator(device="cuda").manual_seed(4)
    return _MoE(256, 128, 4, 2, 0, 4, seed=9), torch.randn(rows, 256, generator=g, device="cuda", dtype=torch.float32).bfloat16()


def test_strided_input_is_refused_as_by_act_quant():
    import dsv3_b200
    moe, x = _layer_and_input()
    moe.shared_experts = lambda x: torch.zeros_like(x)
    strided = torch.empty(24, 512, device="cuda")[:, :256].copy_(x)
    with pytest.raises(AssertionError, match="contiguous"):
        dsv3_b200.grouped_moe_forward(moe, strided)


@pytest.mark.parametrize("form", ["offset", "strided", "float32", "row", "needs_grad"])
def test_any_shared_result_that_can_be_added(form):
    """A host's own shared experts: 16-byte loads and the combine kernel are for plain bf16 results."""
    import dsv3_b200
    moe, x = _layer_and_input()
    z = torch.randn(24, 256, device="cuda")
    z = {"offset": lambda: torch.empty(24 * 256 + 3, device="cuda")[3:].view(24, 256).copy_(z), "strided": lambda: z.t().contiguous().t(),
         "float32": lambda: z.float(), "row": lambda: z[:1], "needs_grad": lambda: z.clone().requires_grad_()}[form]()
    moe.shared_experts = lambda x: torch.zeros_like(x)
    y = dsv3_b200.grouped_moe_forward(moe, x)
    moe.shared_experts = lambda x: z
    got = dsv3_b200.grouped_moe_forward(moe, x)
    assert got.dtype == (y + z).dtype and torch.equal(got, y + z)
    if form == "needs_grad":
        got.sum().backward()
        assert torch.equal(z.grad, torch.ones_like(z))
