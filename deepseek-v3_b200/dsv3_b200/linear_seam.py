"""Seam above the three operators: a replacement for ``linear()`` of the reference's ``model.py``.

``model.py:131-163`` dispatches every projection through the module-level function ``linear``;
``Linear.forward``, ``ColumnParallelLinear.forward``, ``RowParallelLinear.forward`` and
``Gate.forward`` look the name up at call time (model.py:205, 233, 262, 576), so one assignment

    import model, dsv3_b200
    dsv3_b200.install_linear(model)

redirects all of them without touching the file.  The replacement keeps the reference's three
branches and changes how the FP8 branch is launched:

* 1 or 2 rows (a decode step at small batch) and at most 16 MB of weights, or 3 or 4 rows and at most 6 MB: one
  launch, the activations are quantised in the GEMM's prologue (``fp8_linear``) instead of ``act_quant`` followed by ``fp8_gemm`` and an FP8
  round trip through HBM;
* more rows: the quantisation of an activation tensor is remembered while that tensor is alive and unmodified,
  so that Linears fed the same input (``wq_a``/``wkv_a`` in MLA, ``w1``/``w3`` in MLP and Expert) quantise it
  once.  Results are bit-identical to the unfused path because the very same ``act_quant`` output is reused.

The memo holds the two most recent inputs (``wq_a(x)``, ``wq_b(q_norm(..))``, ``wkv_a(x)`` of model.py:464-468
touch two tensors alternately).  An entry is reused only for the same tensor object, on the same CUDA stream,
with an unchanged in-place modification counter, and inside a graph capture only for that capture (the quantisation is
then part of the graph).  Tensors created under ``torch.inference_mode()`` have no such
counter: for them the memo is off unless ``assume_no_inplace=True`` is passed to ``install_linear`` -- the host
then promises not to modify a projection's input in place between two Linears (the reference's model.py never
does).
"""
from __future__ import annotations

from typing import Optional

import torch
import torch.nn.functional as F

from ._lib import host
from .ops import weight_dequant, FUSED_LINEAR_MAX_ROWS, FUSED_LINEAR_MAX_WEIGHT_BYTES, FUSED_LINEAR_MAX_WEIGHT_BYTES_3_ROWS

stats = {"act_quant_calls": 0, "act_quant_reused": 0, "fused_linear_calls": 0}
_assume_no_inplace = False
host.set_stats(stats)


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
           scale_fmt: Optional[str] = None, *, gemm_impl: str = "fp8", block_size: int = 128) -> torch.Tensor:
    """``y = x @ weight.T + bias`` with the reference's dispatch (model.py:153-163)."""
    if weight.element_size() > 1:
        return F.linear(x, weight, bias)
    if gemm_impl == "bf16":
        return F.linear(x, weight_dequant(weight, weight.scale), bias)
    y = host.linear(x, weight, block_size, scale_fmt, _assume_no_inplace, FUSED_LINEAR_MAX_ROWS, FUSED_LINEAR_MAX_WEIGHT_BYTES,
                    FUSED_LINEAR_MAX_WEIGHT_BYTES_3_ROWS)
    if bias is not None:
        y += bias
    return y


def install_linear(model_module, assume_no_inplace: bool = False) -> None:
    """Point ``model_module.linear`` at this implementation; ``model_module.gemm_impl`` and
    ``model_module.block_size`` keep their meaning and are read at call time, as in the reference."""
    global _assume_no_inplace
    _assume_no_inplace = bool(assume_no_inplace)

    def _linear(x, weight, bias=None, scale_fmt=None):
        return linear(x, weight, bias, scale_fmt, gemm_impl=model_module.gemm_impl,
                      block_size=model_module.block_size)
    _linear.__doc__ = linear.__doc__
    _linear._dsv3_linear = _linear        # itself: a wrapper that copies attributes is told from it
    model_module.linear = _linear


def reset_memo() -> None:
    host.forget()
    stats.update(act_quant_calls=0, act_quant_reused=0, fused_linear_calls=0)
