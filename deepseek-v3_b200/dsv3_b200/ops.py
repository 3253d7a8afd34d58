"""The three operators of the reference's ``inference/kernel.py`` on sm_100a.

Signatures, argument meaning, allocation behaviour and assertion messages follow
``kernel.py`` (``act_quant`` :38-57, ``weight_dequant`` :89-110, ``fp8_gemm``
:175-196) so that ``model.py`` and ``generate.py`` run unchanged on top of them.
The work is done by hand-written CUDA behind a C ABI; tensors must live on a CUDA
device and nothing here falls back to another implementation.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib
from ._lib import host, lib

KERNEL_AUTO, KERNEL_CUDA_CORE, KERNEL_TC_TOKEN_MAJOR, KERNEL_TC_WEIGHT_MAJOR, KERNEL_TC_TOKEN_PAIR, KERNEL_DECODE = 0, 1, 2, 3, 4, 5
KERNEL_TC_TOKEN_PAIR_WIDE = 6


def _require_cuda(*tensors: torch.Tensor) -> torch.device:
    dev = tensors[0].device
    for t in tensors:
        if t.device.type != "cuda":
            raise RuntimeError("dsv3_b200 runs on CUDA tensors only (there is no CPU path); got a "
                               f"{t.device.type} tensor")
        if t.device != dev:
            raise RuntimeError("all tensors of one call must be on the same device")
    return dev


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def act_quant(x: torch.Tensor, block_size: int = 128, scale_fmt: Optional[str] = None
              ) -> Tuple[torch.Tensor, torch.Tensor]:
    """Block-wise FP8 quantisation of activations (kernel.py:38-57).

    Returns ``(y, s)``: ``y`` float8_e4m3fn of x's shape, ``s`` float32 of shape
    ``[..., K // block_size]`` with ``s = max(amax, 1e-4) / 448`` per block (rounded up to a
    power of two when ``scale_fmt == "ue8m0"``).
    """
    return host.act_quant(x, block_size, scale_fmt)


def swiglu_quant(a: torch.Tensor, b: torch.Tensor, scale_fmt: Optional[str] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    """``act_quant(F.silu(a) * b, 128, scale_fmt)`` in one launch (model.py:532 / 633 followed by :158-159), with the
    rounding points of the three-launch form; the bf16 product is never written."""
    return host.swiglu_quant(a, b, scale_fmt)


# Cache of de-quantised weights (off by default).  MLA.forward in "absorb" mode de-quantises wkv_b on every call of
# every layer (model.py:481) although the weight never changes; with the cache on, the call after the first returns
# the tensor computed before and launches nothing.  An entry is keyed on the weight's and the scales' storage
# address, shape and in-place modification counter and holds a weak reference to the weight, so loading new values
# into the parameter (copy_, load_model) or freeing it invalidates the entry.
_dequant_cache = None            # OrderedDict when enabled
_dequant_cache_limit = 0
dequant_stats = {"launches": 0, "hits": 0}


def enable_weight_dequant_cache(max_bytes: int = 2 << 30) -> None:
    """Remember the results of ``weight_dequant`` (up to ``max_bytes`` of bf16 copies, oldest dropped first).
    The caller must treat the returned tensors as read-only (model.py:481-495 only views and multiplies them).
    Meant for inference loops; leave it off for one-pass tools such as ``fp8_cast_bf16.py``."""
    global _dequant_cache, _dequant_cache_limit
    import collections
    _dequant_cache = collections.OrderedDict()
    _dequant_cache_limit = int(max_bytes)


def disable_weight_dequant_cache() -> None:
    global _dequant_cache
    _dequant_cache = None


def _version_or_none(t: torch.Tensor):
    try:
        return t._version
    except RuntimeError:          # inference tensors carry no counter: never cached
        return None


def weight_dequant(x: torch.Tensor, s: torch.Tensor, block_size: int = 128) -> torch.Tensor:
    """De-quantise a block-scaled FP8 weight to the default dtype (kernel.py:89-110)."""
    key = None
    if _dequant_cache is not None:
        vx, vs = _version_or_none(x), _version_or_none(s)
        if vx is not None and vs is not None:
            key = (x.data_ptr(), s.data_ptr(), tuple(x.shape), block_size, vx, vs, torch.get_default_dtype())
            hit = _dequant_cache.get(key)
            if hit is not None and hit[0]() is x:
                _dequant_cache.move_to_end(key)
                dequant_stats["hits"] += 1
                return hit[1]
    y = host.weight_dequant(x, s, block_size)
    dequant_stats["launches"] += 1
    if key is not None and not torch.cuda.is_current_stream_capturing():      # (a recorded launch has computed nothing yet)
        import weakref
        try:
            _dequant_cache[key] = (weakref.ref(x), y)
        except TypeError:
            return y
        total = sum(v[1].numel() * v[1].element_size() for v in _dequant_cache.values())
        while total > _dequant_cache_limit and len(_dequant_cache) > 1:
            _, old = _dequant_cache.popitem(last=False)
            total -= old[1].numel() * old[1].element_size()
    return y


def fp8_gemm(a: torch.Tensor, a_s: torch.Tensor, b: torch.Tensor, b_s: torch.Tensor) -> torch.Tensor:
    """Block-scaled FP8 GEMM ``c = a @ b.T`` with fp32 accumulation (kernel.py:175-196)."""
    return host.fp8_gemm(a, a_s, b, b_s)


def fp8_linear(x: torch.Tensor, weight: torch.Tensor, scale: torch.Tensor, scale_fmt: Optional[str] = None) -> torch.Tensor:
    """``fp8_gemm(*act_quant(x, 128, scale_fmt), weight, scale)`` (model.py:158-160) in one launch, for at most 16
    rows: the activations are quantised in the GEMM's prologue.  Raises ``Dsv3Error`` (status -2) for other shapes."""
    return host.fp8_linear(x, weight, scale, scale_fmt)


# The kernel takes up to 16 rows; the seam uses it where quantising the activations inside every CTA is cheaper than a launch of
# its own: up to 2 rows for weights of at most 16 MB, 3 and 4 rows for at most 6 MB.  B200, us, one launch / two, replayed from
# a graph with the weights in HBM, at 1, 2 and 4 rows: 7168 -> 576 4.2 / 5.6, 4.6 / 5.6, 4.8 / 5.7; 2048 -> 2816 4.1 / 5.5, 4.8 / 6.1,
# 5.0 / 6.2; 5120 -> 1536 (7.5 MB) 5.6 / 6.4, 5.6 / 6.5, 7.0 / 6.7; 7168 -> 1536 (10.5 MB) 6.8 / 6.7, 7.0 / 6.9, 8.2 / 7.0.  Launched one
# by one the host needs about 4 us for each, so that one launch is ahead up to 8 us: the line for 1 and 2 rows is drawn for
# that.  (Near 16 MB, at 1 row: 2304 -> 7168 7.5 / 7.4, 7168 -> 2304 7.4 / 7.8.)
FUSED_LINEAR_MAX_ROWS = 4
FUSED_LINEAR_MAX_WEIGHT_BYTES = 16 << 20
FUSED_LINEAR_MAX_WEIGHT_BYTES_3_ROWS = 6 << 20


def weight_quant(w: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """Harness quantiser: bf16 ``[N, K]`` -> (float8_e4m3fn ``[N, K]``, float32 ``[ceil(N/128), ceil(K/128)]``)
    with ``s = max(amax, 1e-4) / 448`` per 128x128 block; the inverse of ``weight_dequant``."""
    assert w.is_contiguous() and w.dim() == 2
    dev = _require_cuda(w)
    if w.dtype != torch.bfloat16:
        raise NotImplementedError("weight_quant takes a bfloat16 weight")
    N, K = w.shape
    q = torch.empty_like(w, dtype=torch.float8_e4m3fn)
    s = w.new_empty((N + 127) // 128, (K + 127) // 128, dtype=torch.float32)
    with torch.cuda.device(dev):
        _lib.check(lib.dsv3_weight_quant(w.data_ptr(), N, K, q.data_ptr(), s.data_ptr(), _stream()))
    return q, s


def set_gemm_policy(kernel: int = KERNEL_AUTO, split_k: int = 0) -> None:
    """Pin the fp8_gemm kernel / split-K factor (tests and benchmarks); (0, 0) restores automatic choice."""
    _lib.check(lib.dsv3_set_gemm_policy(kernel, split_k))


def set_num_sms(n: int = 0) -> None:
    """SMs the persistent GEMM kernels may occupy from now on (0 = all): leave a concurrent collective its SMs."""
    _lib.check(lib.dsv3_set_num_sms(int(n)))


def check_device_status() -> None:
    """Synchronise the current stream and raise if a kernel's bounded wait gave up."""
    import ctypes
    detail = (ctypes.c_uint32 * 4)()
    rc = lib.dsv3_check_device_status(_stream(), ctypes.byref(detail))
    if rc != _lib.OK:
        host.drop_workspaces()            # tickets may be left non-zero by an aborted launch
        _lib.check(rc)
