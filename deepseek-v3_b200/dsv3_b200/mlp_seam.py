"""Seam above the operators: ``MLP.forward`` and ``Expert.forward`` with the SwiGLU folded into the quantisation.

Both compute ``w2(F.silu(w1(x)) * w3(x))`` (model.py:532, 633).  In FP8 mode the product is quantised straight away by
the ``linear()`` call of ``w2`` (model.py:158-159), so silu, multiply and act_quant are three launches and two bf16
round trips through HBM for what is one pass over the data.  Where ``w1`` and ``w3`` are plain Linears of the installed
``linear`` and the library's rules on sizes say that it pays (few rows, or tiles that fit one round of the SMs; on the
device, or outside of a graph capture for the host that launches),
``mlp_forward`` is three launches behind one host call: the quantisation of ``x``, ``w1`` and ``w3`` with SwiGLU and the
quantisation in front of ``w2``, and ``w2``.  With more tokens, where ``w1`` and ``w3`` leave most of their last rounds of the SMs
idle, it is four: both GEMMs are one launch and share that round.  Otherwise it calls ``w1`` and ``w3`` (through whatever ``linear`` is
installed), then ``swiglu_quant`` (one launch, same rounding points, bit-identical FP8 codes and scales) and feeds
``fp8_gemm`` of ``w2`` directly.  What ``w2.forward`` would have done after its GEMM follows: the all-reduce of a
``RowParallelLinear`` (model.py:263-264) and the bias.

    import model, dsv3_b200
    dsv3_b200.install_mlp(model)        # model.MLP.forward, model.Expert.forward
"""
from __future__ import annotations

import torch
from torch.nn.modules import module as _nn_module

from . import linear_seam
from ._lib import host
from .ops import fp8_gemm, swiglu_quant
from .plain import calls_forward, installed_linear, linear_takes_fmt


def _fusable(self, x, model_module) -> bool:
    return (getattr(model_module, "gemm_impl", "fp8") == "fp8" and getattr(model_module, "block_size", 128) == 128
            and host.fp8_weights(self.w1.weight, self.w3.weight, self.w2.weight) and x.dtype is torch.bfloat16)


def mlp_forward(self, x: torch.Tensor, *, model_module, original) -> torch.Tensor:
    """Same inputs and outputs as ``MLP.forward`` / ``Expert.forward`` (model.py:520-532, 622-633)."""
    if not _fusable(self, x, model_module):
        return original(self, x)
    w2 = self.w2
    if host.intercepted(w2) or _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
        return original(self, x)                          # w2 is not called below
    up, down = _plain_up(self, model_module), type(w2).__name__
    if down == "Linear" and not (up and type(w2) is type(self.w1)) and linear_takes_fmt(w2, model_module) is None:
        return original(self, x)                          # an adapter of that name, say
    row_parallel = down == "RowParallelLinear"
    # only plain Linear hands its scale_fmt to linear() (model.py:205); the parallel Linears do not (model.py:233, 262)
    scale_fmt = None if (row_parallel or down == "ColumnParallelLinear") else getattr(w2, "scale_fmt", None)
    y = host.mlp(x, up[0], up[1], w2.weight, up[2], scale_fmt, linear_seam._assume_no_inplace) if up else None
    if y is None:
        hq, hs = swiglu_quant(self.w1(x), self.w3(x), scale_fmt)
        y = fp8_gemm(hq, hs, w2.weight, w2.weight.scale)
    if row_parallel:
        if model_module.world_size > 1:
            model_module.dist.all_reduce(y)
        if w2.bias is not None:
            y += w2.bias
    elif getattr(w2, "bias", None) is not None:
        y += w2.bias
    return y


_UP, _DOWN = ("Linear", "ColumnParallelLinear"), ("Linear", "RowParallelLinear")


def _plain_format(model, w1, w3, w2=None):
    """The scale_fmt that the Linears, which nothing intercepts, all hand to the installed ``linear``, where they do nothing but that
    (classes of the names above, no bias, no code of their own); otherwise False."""
    if (getattr(model, "world_size", 1) != 1 or not installed_linear(model) or _nn_module._global_forward_hooks
            or _nn_module._global_forward_pre_hooks):
        return False
    up = type(w1)
    if up.__name__ not in _UP or getattr(w1, "bias", None) is not None or getattr(w3, "bias", None) is not None:
        return False
    takes_fmt = linear_takes_fmt(w1, model, w3 if type(w3) is up else None)
    if takes_fmt is None:
        return False
    fmt = w1.scale_fmt if takes_fmt else None
    if type(w3) is not up:
        takes_fmt = linear_takes_fmt(w3, model) if type(w3).__name__ in _UP else None
        if takes_fmt is None:
            return False
    if (w3.scale_fmt if takes_fmt else None) != fmt:
        return False
    if w2 is not None:
        if type(w2).__name__ not in _DOWN or getattr(w2, "bias", None) is not None:
            return False
        takes_fmt = linear_takes_fmt(w2, model)
        if takes_fmt is None or (w2.scale_fmt if takes_fmt else None) != fmt:
            return False
    return fmt


def _plain_up(mlp, model):
    """``(w1, w3, scale_fmt)`` where both do nothing but the GEMM, through the installed ``linear``, on equally quantised
    activations; otherwise None.  The three launches of ``host.mlp`` (the quantisation, w1 and w3 with everything up to w2's
    quantisation, w2) are then as good as theirs."""
    w1, w3 = mlp.w1, mlp.w3
    if host.intercepted(w1, w3):
        return None
    fmt = _plain_format(model, w1, w3)
    return None if fmt is False else (w1.weight, w3.weight, fmt)


def plain_weights(mlp, x: torch.Tensor, scale_fmt):
    """``(w1, w3, w2)`` weights of an MLP that ``mlp_forward`` serves and whose Linears do nothing but the GEMM in
    ``scale_fmt``, so that a caller may run them itself; otherwise None."""
    installed = getattr(type(mlp), "forward", None)
    seen, model = getattr(installed, "_dsv3_mlp", (None, None))
    if seen is None or seen is not installed:
        return None
    w1, w2, w3 = mlp.w1, mlp.w2, mlp.w3
    if (host.intercepted(mlp, w1, w2, w3) or not calls_forward(mlp, model) or _plain_format(model, w1, w3, w2) != scale_fmt
            or not _fusable(mlp, x, model)):
        return None
    return w1.weight, w3.weight, w2.weight


def install_mlp(model_module) -> None:
    """Replace ``model_module.MLP.forward`` and ``model_module.Expert.forward``; ``gemm_impl``, ``block_size``,
    ``world_size`` and ``dist`` of the module are read at call time."""
    for cls_name in ("MLP", "Expert"):
        cls = getattr(model_module, cls_name)
        original = cls.forward

        def forward(self, x, _original=original):
            return mlp_forward(self, x, model_module=model_module, original=_original)

        forward.__doc__ = mlp_forward.__doc__
        forward._dsv3_mlp = forward, model_module        # itself: a wrapper that copies attributes is told from it
        cls.forward = forward
