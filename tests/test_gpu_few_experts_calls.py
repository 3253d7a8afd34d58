"""The expert layer for a handful of tokens as its callers use it: what it takes and refuses, and when the weights are read."""
import pytest
import torch

from test_gpu_moe import _MoE, _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


def _layer(topk=2, tokens=2, n_routed=64, local=4, dim=512, inter=256):
    moe = _MoE(dim, inter, n_routed, topk, 0, local, seed=17)
    x = torch.randn(tokens, dim, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda", dtype=torch.float32).bfloat16()
    return moe, x


def test_more_experts_per_token_than_the_dispatch_takes_are_refused():
    """At most 32, as with more tokens."""
    import dsv3_b200
    moe, x = _layer(tokens=1, local=2)
    for topk in (32, 33):
        indices = torch.arange(topk, device="cuda").view(1, topk)
        moe.gate = lambda x: (torch.ones(1, topk, device="cuda"), indices)
        if topk == 32:
            assert dsv3_b200.grouped_moe_forward(moe, x).shape == x.shape
        else:
            with pytest.raises(dsv3_b200.Dsv3Error) as e:
                dsv3_b200.grouped_moe_forward(moe, x)
            assert e.value.status == -2
