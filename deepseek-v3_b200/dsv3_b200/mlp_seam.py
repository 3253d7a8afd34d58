"""Seam above the operators: ``MLP.forward`` and ``Expert.forward`` with the SwiGLU folded into the quantisation.

Both compute ``w2(F.silu(w1(x)) * w3(x))`` (model.py:532, 633).  In FP8 mode the product is quantised straight away by
the ``linear()`` call of ``w2`` (model.py:158-159), so silu, multiply and act_quant are three launches and two bf16
round trips through HBM for what is one pass over the data.  Where ``w1`` and ``w3`` are plain Linears of the installed
``linear`` and the library's rule on sizes says that it pays (few rows, or tiles that fit one round of the SMs),
``mlp_forward`` is three launches behind one host call: the quantisation of ``x``, ``w1`` and ``w3`` with SwiGLU and the
quantisation in front of ``w2``, and ``w2``.  Otherwise it calls ``w1`` and ``w3`` (through whatever ``linear`` is
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


def _fusable(self, x, model_module) -> bool:
    w2 = self.w2
    return (getattr(model_module, "gemm_impl", "fp8") == "fp8" and getattr(model_module, "block_size", 128) == 128
            and w2.weight.element_size() == 1 and self.w1.weight.element_size() == 1 and self.w3.weight.element_size() == 1
            and w2.weight.size(1) % 128 == 0 and x.dtype == torch.bfloat16)


def mlp_forward(self, x: torch.Tensor, *, model_module, original) -> torch.Tensor:
    """Same inputs and outputs as ``MLP.forward`` / ``Expert.forward`` (model.py:520-532, 622-633)."""
    if not _fusable(self, x, model_module):
        return original(self, x)
    w2 = self.w2
    row_parallel = type(w2).__name__ == "RowParallelLinear"
    # only plain Linear hands its scale_fmt to linear() (model.py:205); the parallel Linears do not (model.py:233, 262)
    scale_fmt = None if (row_parallel or type(w2).__name__ == "ColumnParallelLinear") else getattr(w2, "scale_fmt", None)
    up = _plain_up(self, model_module)
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


def _plain_up(mlp, model):
    """``(w1, w3, scale_fmt)`` where both do nothing but the GEMM, through the installed ``linear``, on equally quantised
    activations; otherwise None.  The three launches of ``host.mlp`` (the quantisation, w1 and w3 with everything up to w2's
    quantisation, w2) are then as good as theirs."""
    if getattr(model, "world_size", 1) != 1 or not getattr(getattr(model, "linear", None), "_dsv3_linear", False):
        return None
    if _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
        return None
    w1, w3 = mlp.w1, mlp.w3
    for lin in (w1, w3):
        if type(lin).__name__ not in ("Linear", "ColumnParallelLinear") or getattr(lin, "bias", None) is not None or _intercepted(lin):
            return None
    fmt = _scale_fmt_of(w1)
    return (w1.weight, w3.weight, fmt) if _scale_fmt_of(w3) == fmt else None


def _scale_fmt_of(lin):
    """The scale_fmt a Linear hands to linear(): only the plain one does (model.py:205; not :233, :262)."""
    return getattr(lin, "scale_fmt", None) if type(lin).__name__ == "Linear" else None


def _intercepted(module) -> bool:
    """Whether a call of the module does more than its class's forward: hooks, or a forward of its own."""
    return bool(getattr(module, "_forward_hooks", None) or getattr(module, "_forward_pre_hooks", None)
                or "forward" in getattr(module, "__dict__", ()))


def plain_weights(mlp, x: torch.Tensor, scale_fmt):
    """``(w1, w3, w2)`` weights of an MLP that ``mlp_forward`` serves and whose Linears do nothing but the GEMM in
    ``scale_fmt`` (no bias, no hooks, no forward of their own, the installed ``linear``), so that a caller may run them
    itself; otherwise None."""
    model = getattr(getattr(type(mlp), "forward", None), "_dsv3_model", None)
    if model is None or getattr(model, "world_size", 1) != 1 or not getattr(getattr(model, "linear", None), "_dsv3_linear", False):
        return None
    if _intercepted(mlp) or _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
        return None
    w1, w2, w3 = mlp.w1, mlp.w2, mlp.w3
    for lin, names in ((w1, ("Linear", "ColumnParallelLinear")), (w3, ("Linear", "ColumnParallelLinear")), (w2, ("Linear", "RowParallelLinear"))):
        if (type(lin).__name__ not in names or getattr(lin, "bias", None) is not None or _scale_fmt_of(lin) != scale_fmt
                or _intercepted(lin)):
            return None
    if not _fusable(mlp, x, model):
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
        forward._dsv3_model = model_module
        cls.forward = forward
