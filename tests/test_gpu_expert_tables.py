"""The expert layer works with device tables of its experts' weights and scales: whatever a host exchanges between two
passes has to reach the second one.  Reference: the expert loop on the drop-in operators."""
import pytest
import torch

import test_gpu_moe
from test_gpu_stream import _bf16_default, _weight  # noqa: F401

pytestmark = pytest.mark.gpu


class _Linear(torch.nn.Module):
    """model.py's Linear: a Parameter with its scales as an attribute."""
    scale_fmt = None

    def __init__(self, n, k, g):
        super().__init__()
        w = _weight(n, k, g)
        self.weight = torch.nn.Parameter(w, requires_grad=False)
        self.weight.scale = self.scale = torch.nn.Parameter(w.scale, requires_grad=False)

    def forward(self, x):
        import kernel
        return kernel.fp8_gemm(*kernel.act_quant(x), self.weight, self.weight.scale)


class _Expert(torch.nn.Module):
    def __init__(self, dim, inter, g):
        super().__init__()
        self.w1, self.w2, self.w3 = _Linear(inter, dim, g), _Linear(dim, inter, g), _Linear(inter, dim, g)

    def forward(self, x):
        return self.w2(torch.nn.functional.silu(self.w1(x)) * self.w3(x))


def _replace_scale(e, other):
    e.w1.weight.scale = torch.nn.Parameter(other.w1.weight.scale.clone(), requires_grad=False)


def _scale_data(e, other):
    e.w2.weight.scale.data = other.w2.weight.scale.clone()


def _weight_data(e, other):
    e.w3.weight.data = other.w3.weight.data.clone()


def _replace_parameter(e, other):
    e.w1.weight = other.w1.weight


def _replace_parameters(e, other):
    e.w2._parameters = dict(other.w2._parameters)


def _replace_modules(e, other):
    e._modules = dict(other._modules)


def _swap(e, other):
    torch.utils.swap_tensors(e.w1.weight, other.w1.weight)


@pytest.mark.parametrize("change", [_replace_scale, _scale_data, _weight_data, _replace_parameter, _replace_parameters, _replace_modules, _swap])
@pytest.mark.parametrize("container", [list, torch.nn.ModuleList])
def test_exchanged_weights_and_scales_are_seen(change, container):
    import dsv3_b200
    g = torch.Generator(device="cuda").manual_seed(3)
    moe = test_gpu_moe._MoE(256, 128, 4, 2, 0, 4, seed=9)
    moe.experts = container([_Expert(256, 128, g) for _ in range(4)])
    other = _Expert(256, 128, g)
    x = torch.randn(24, 256, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    before = dsv3_b200.grouped_moe_forward(moe, x)
    change(moe.experts[1], other)
    got = dsv3_b200.grouped_moe_forward(moe, x)
    assert not torch.equal(got, before)
    want, _ = moe.reference_forward(x)
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    assert bool((err <= 2e-2 * (want.float().abs() + rms)).all())         # the bound of test_gpu_moe.py
