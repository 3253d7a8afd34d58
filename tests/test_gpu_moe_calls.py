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
