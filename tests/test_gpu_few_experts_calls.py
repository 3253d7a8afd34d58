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


@pytest.mark.parametrize("world_size", [1, 2])
def test_weights_are_read_before_the_shared_experts_are_called(world_size, monkeypatch):
    """A host may give the routed experts' weights other contents (the next layer's, say) from there on."""
    import dsv3_b200
    monkeypatch.setattr(torch.distributed, "all_reduce", lambda y: y.mul_(2))
    moe, x = _layer()
    moe.gate = lambda x: (torch.ones(2, 2, device="cuda"), torch.tensor([[0, 1], [3, 60]], device="cuda"))
    z = torch.randn(2, 512, device="cuda")
    moe.shared_experts = lambda x: z
    want = dsv3_b200.grouped_moe_forward(moe, x, world_size=world_size)

    def overwrite(x):
        for e in moe.experts[:4]:
            e.w2.weight.view(torch.uint8).zero_()
        return z

    moe.shared_experts = overwrite
    assert torch.equal(dsv3_b200.grouped_moe_forward(moe, x, world_size=world_size), want)
    assert not torch.equal(want, z)
