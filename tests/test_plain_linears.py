"""When an MLP's Linears may be computed without being called: only where their code is a call of the installed linear()."""
import functools
import types

import pytest
import torch

import dsv3_b200
from dsv3_b200 import mlp_seam

MODULE = '''
import torch
world_size, gemm_impl, block_size, dist = 1, "fp8", 128, None
class Linear(torch.nn.Module):
    scale_fmt = None
    def __init__(self):
        super().__init__()
        self.weight, self.bias = torch.nn.Parameter(torch.zeros(128, 128, dtype=torch.uint8), requires_grad=False), None
    def forward(self, x):
        return linear(x, self.weight, self.bias, self.scale_fmt)
class ColumnParallelLinear(Linear):
    def forward(self, x):
        y = linear(x, self.weight, self.bias)
        return y
class RowParallelLinear(Linear):
    def forward(self, x):
        y = linear(x, self.weight)
        if world_size > 1:
            dist.all_reduce(y)
        if self.bias is not None:
            y += self.bias
        return y
class MLP(torch.nn.Module):
    def __init__(self, up=Linear, down=Linear):
        super().__init__()
        self.w1, self.w2, self.w3 = up(), down(), up()
    def forward(self, x):
        return self.w2(torch.nn.functional.silu(self.w1(x)) * self.w3(x))
class Expert(MLP):
    def forward(self, x):
        return self.w2(torch.nn.functional.silu(self.w1(x)) * self.w3(x))
'''
X = torch.zeros(2, 128, dtype=torch.bfloat16)


def _model():
    model = types.ModuleType("model_of_a_host")
    exec(MODULE, model.__dict__)
    dsv3_b200.install_linear(model)
    dsv3_b200.install_mlp(model)
    return model


def _plain(mlp, model):
    """Whether w1 and w3, and whether all three, are taken for plain."""
    return mlp_seam._plain_up(mlp, model) is not None, mlp_seam.plain_weights(mlp, X, None) is not None


def test_the_models_own_linears_are_plain():
    model = _model()
    assert _plain(model.MLP(), model) == (True, True) and _plain(model.Expert(), model) == (True, True)
    assert _plain(model.MLP(model.ColumnParallelLinear, model.RowParallelLinear), model) == (True, True)
    for up, fmt in ((model.Linear, "ue8m0"), (model.ColumnParallelLinear, None)):      # the parallel ones hand over none
        mlp = model.MLP(up)
        mlp.w1.scale_fmt = mlp.w3.scale_fmt = "ue8m0"
        assert mlp_seam._plain_up(mlp, model)[2] == fmt


class _Plain:
    """The same outside of torch.nn, reaching the model through a name, a closure or an attribute."""
    weight, bias, scale_fmt = torch.zeros(128, 128, dtype=torch.uint8), None, None


def _by_closure(model):
    class Linear(_Plain):
        def __call__(self, x):
            return model.linear(x, self.weight, self.bias, self.scale_fmt)
    return Linear


def _by_attribute(model):
    class Linear(_Plain):
        def __init__(self):
            self.host = [model]

        def forward(self, x):
            return self.host[0].linear(x, self.weight, self.bias, self.scale_fmt)

        def __call__(self, x):
            return self.forward(x)
    return Linear


@pytest.mark.parametrize("made", [_by_closure, _by_attribute])
def test_a_hosts_own_way_to_the_installed_linear(made):
    model = _model()
    cls = made(model)
    assert _plain(model.MLP(cls, cls), model) == (True, True)
    if made is _by_attribute:
        mlp = model.MLP(cls, cls)
        mlp.w3.host = [_model()]                            # another model's linear()
        assert _plain(mlp, model) == (False, False)


def _class_forward(model, mlp, seen):
    inner = model.Linear.forward
    model.Linear.forward = lambda self, x: (seen.append(1), inner(self, x))[1]


def _new_code(model, mlp, seen):
    def forward(self, x):
        return linear(x, self.weight, self.bias, self.scale_fmt) * 2  # noqa: F821
    model.Linear.forward.__code__ = forward.__code__


def _subclass(body):
    """w1 and w3 of a class that is called Linear too, its forward written in the model's own module."""
    def change(model, mlp, seen):
        names = {}
        model.seen = seen
        exec(body, model.__dict__, names)
        cls = type("Linear", (model.Linear,), {"forward": names["forward"]})
        mlp.w1, mlp.w3 = cls(), cls()
    return change


def test_a_class_of_that_name_with_the_same_code_is_plain():
    model = _model()
    mlp = model.MLP()
    _subclass("def forward(self, x):\n y = linear(x, self.weight, self.bias, scale_fmt=self.scale_fmt)\n return y")(model, mlp, [])
    assert _plain(mlp, model) == (True, True)


def _class_call(model, mlp, seen):
    cls = type("Linear", (model.Linear,), {"__call__": lambda self, x: (seen.append(1), self.forward(x))[1]})
    mlp.w1, mlp.w3 = cls(), cls()


def _wrapped_linear(model, mlp, seen):
    inner = model.linear

    @functools.wraps(inner)
    def linear(*args):
        seen.append(1)
        return inner(*args)
    model.linear = linear


def _compiled(model, mlp, seen):
    mlp.w1._compiled_call_impl = lambda x: x


CHANGES = {
    "class": _class_forward, "code": _new_code, "call": _class_call, "wraps": _wrapped_linear, "compiled": _compiled,
    "adapter": _subclass("def forward(self, x):\n return linear(x, self.weight, self.bias, self.scale_fmt) + self.up(self.down(x))"),
    "scaled": _subclass("def forward(self, x):\n return 2 * linear(x, self.weight, self.bias, self.scale_fmt)"),
    "twice": _subclass("def forward(self, x):\n linear(x, self.weight)\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "counted": _subclass("def forward(self, x):\n seen.append(1)\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "caught": _subclass("def forward(self, x):\n try:\n  seen.append(1)\n except Exception:\n  pass\n return linear(x, self.weight, self.bias)"),
    "stored": _subclass("def forward(self, x):\n self.x = x\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "global": _subclass("def forward(self, x):\n global last\n last = x\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "class attribute": _subclass("def forward(self, x):\n self.__class__.last = x\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "operand's class": _subclass("def forward(self, x):\n x.__class__.last = x\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "dictionary": _subclass("def forward(self, x):\n self.__dict__['last'] = x\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "training": _subclass("def forward(self, x):\n if self.training: x = x + 1\n return linear(x, self.weight, self.bias, self.scale_fmt)"),
    "other weight": _subclass("def forward(self, x):\n return linear(x, self.weight_b, self.bias, self.scale_fmt)"),
}


@pytest.mark.parametrize("seen_before", [False, True])
@pytest.mark.parametrize("change", CHANGES)
def test_code_of_the_hosts_is_called(change, seen_before):
    model = _model()
    mlp, seen = model.MLP(), []
    if seen_before:
        assert _plain(mlp, model) == (True, True)
    CHANGES[change](model, mlp, seen)
    assert _plain(mlp, model) == (False, False)
    assert not seen


def test_an_mlp_of_the_hosts_is_called():
    model = _model()
    inner = model.MLP.forward

    class MLP(model.MLP):
        @functools.wraps(inner)
        def forward(self, x):
            return inner(self, x) * 2

    class Called(model.MLP):
        def __call__(self, x):
            return self.forward(x) * 2

    for cls in (MLP, Called):
        assert mlp_seam.plain_weights(cls(), X, None) is None
    assert mlp_seam.plain_weights(type("Own", (model.MLP,), {})(), X, None) is not None


def _hook(model, mlp, seen):
    mlp.w2.register_forward_hook(lambda m, i, o: seen.append(1))


def _own_forward(model, mlp, seen):
    inner = mlp.w2.forward
    mlp.w2.forward = lambda x: (seen.append(1), inner(x))[1]


def _global_hook(model, mlp, seen):
    return torch.nn.modules.module.register_module_forward_pre_hook(lambda m, i: seen.append(1) if m is mlp.w2 else None).remove


def _adapter(model, mlp, seen):
    def forward(self, x):
        seen.append(1)
        return model.linear(x, self.weight)
    mlp.w2 = type("Linear", (model.Linear,), {"forward": forward})()


def _patched_class(model, mlp, seen):
    mlp.w1, mlp.w3 = model.ColumnParallelLinear(), model.ColumnParallelLinear()
    inner = model.Linear.forward
    model.Linear.forward = lambda self, x: (seen.append(1), inner(self, x))[1]


@pytest.mark.parametrize("change", [_hook, _own_forward, _global_hook, _adapter, _patched_class])
def test_w2_that_is_intercepted_is_called(change):
    model = _model()
    mlp, seen = model.MLP(), []
    model.linear = lambda x, weight, bias=None, scale_fmt=None: x + 1
    undo = change(model, mlp, seen)
    try:
        y = mlp(X)
    finally:
        if undo:
            undo()
    assert seen == [1] and torch.equal(y, torch.nn.functional.silu(X + 1) * (X + 1) + 1)


def test_weights_that_are_no_fp8_tensors_are_the_hosts():
    model = _model()
    for weight in (torch.zeros(128, 128), object()):
        mlp = model.MLP()
        model.linear = lambda x, w, bias=None, scale_fmt=None: x + 1
        del mlp.w3.weight
        mlp.w3.weight = weight
        assert torch.equal(mlp(X), torch.nn.functional.silu(X + 1) * (X + 1) + 1)
