"""Forms of a call of the expert layer at the edge of what it takes."""
import types

import pytest
import torch
import torch.nn.functional as F

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


class Linear(torch.nn.Module):
    """model.py's Linear by name, calling the model's linear()."""
    scale_fmt = bias = None

    def __init__(self, n, k, seed, model):
        super().__init__()
        import dsv3_b200
        g = torch.Generator(device="cuda").manual_seed(seed)
        w, s = dsv3_b200.weight_quant((torch.randn(n, k, generator=g, device="cuda", dtype=torch.float32) * 0.02).bfloat16())
        self.weight = torch.nn.Parameter(w, requires_grad=False)
        self.weight.scale = s
        self.model = [model]

    def forward(self, x):
        return self.model[0].linear(x, self.weight, self.bias, self.scale_fmt)


def _host():
    """A model whose three seams are installed, its expert layer with shared experts, and an input."""
    import dsv3_b200
    model = types.SimpleNamespace(gemm_impl="fp8", block_size=128, world_size=1, dist=None)

    class MLP(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.w1, self.w2, self.w3 = Linear(128, 256, 1, model), Linear(256, 128, 2, model), Linear(128, 256, 3, model)

        def forward(self, x):
            return self.w2(F.silu(self.w1(x)) * self.w3(x))

    model.MLP, model.Expert = MLP, type("Expert", (MLP,), {"forward": MLP.forward})
    dsv3_b200.install_linear(model)
    dsv3_b200.install_mlp(model)
    moe, x = _layer_and_input()
    moe.shared_experts = MLP()
    return moe, x


def _own_forward(moe, part, seen):
    module = moe.shared_experts if part == "mlp" else getattr(moe.shared_experts, part)
    inner = module.forward
    module.forward = lambda x: (seen.append(1), inner(x))[1]


def _global_hook(moe, part, seen):
    handle = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(1))
    return handle.remove


@pytest.mark.parametrize("intercept,part", [(_own_forward, "mlp"), (_own_forward, "w1"), (_own_forward, "w3"), (_global_hook, None)])
def test_shared_experts_that_are_intercepted_are_called(intercept, part):
    import dsv3_b200
    moe, x = _host()
    want = dsv3_b200.grouped_moe_forward(moe, x)
    seen = []
    undo = intercept(moe, part, seen)
    try:
        got = dsv3_b200.grouped_moe_forward(moe, x)
    finally:
        if undo:
            undo()
    assert seen
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    assert bool((err <= 2e-2 * (want.float().abs() + rms)).all())         # the bound of test_gpu_moe.py


@pytest.mark.parametrize("rows,topk", [(24, 0), (0, 2)])
def test_no_pairs_leave_the_shared_result(rows, topk):
    import dsv3_b200
    moe, x = _host()
    moe.gate = lambda x: (torch.empty(x.size(0), topk, device="cuda"), torch.zeros(x.size(0), topk, dtype=torch.int64, device="cuda"))
    assert torch.equal(dsv3_b200.grouped_moe_forward(moe, x[:rows]), moe.shared_experts(x[:rows]))
