"""Seam above the operators: the MoE expert loop as grouped GEMMs.

``MoE.forward`` of the reference (model.py:669-693) walks over the local experts in Python; every
expert costs two host synchronisations (``bincount(...).tolist()``, ``torch.where``) and about six
small launches.  ``grouped_moe_forward`` keeps inputs, outputs and arithmetic (same quantisation per
token row, same bf16 rounding points, same ascending-expert accumulation order) but runs in
four launches: routing bookkeeping with the quantisation of the tokens, w1 and w3 of all local experts with SwiGLU and
the quantisation in front of w2, w2 of all local experts, and the weighted sum with the shared experts' output; or, where
few pairs are expected, two (w1 and w3 with everything in front of them, w2 with the weighted sum).  Nothing is read back
to the host.

    import model, dsv3_b200
    dsv3_b200.install_moe(model)        # model.MoE.forward = grouped_moe_forward
"""
from __future__ import annotations

import ctypes
from typing import List

import torch

from . import _lib, linear_seam
from ._lib import host, lib
from .mlp_seam import plain_weights
from .ops import _stream

# Up to this many tokens the shared experts are worked on in the routed experts' launches, which saves two launches of
# 3-8 us and their fill and drain; their tiles take the routed experts' token width, so with many tokens their own GEMMs use
# the machine better.  B200, us, inline / separate, at 64, 150, 333, 512 and 700 tokens: 64 experts of 2048 x 1408 105 / 118,
# 114 / 129, 135 / 148, 149 / 169, 171 / 178; 160 of 5120 x 1536 427 / 440, 532 / 557, 598 / 620, 650 / 660, 670 / 675; 256 of
# 7168 x 2048 1136 / 1160, 1418 / 1438, 1640 / 1650, 1765 / 1800, 1930 / 1889; 32 of those 256 186 / 208, 210 / 234, 246 / 275, 296 / 305,
# 352 / 340.
SHARED_INLINE_MAX_ROWS = 512
# On a rank with few of the experts, their narrow tiles read the shared experts' weights from L2 once per tile of 16, 32 or 64
# tokens: when that is more than the local experts' own weights (and than what launches cost, hence the floor) it is what the
# launch waits for.  Inline / separate at 128, 256, 333 and 512 tokens: 20 of 160 experts of 5120 x 1536 101 / 120, 121 / 133, 140 / 132,
# 167 / 144; 10 of those 80 / 91, 105 / 101, 107 / 102, 133 / 115; 8 of 256 of 7168 x 2048 (at 128 tiles of 16) 100 / 104, 111 / 115,
# 137 / 132, 145 / 144; 16 of those 134 / 141, 149 / 156, 161 / 175, 191 / 187; but 16 of 64 of 2048 x 1408, whose weights are small,
# 57 / 67, 65 / 79, at 512 (tiles of 64) 69 / 85.
SHARED_INLINE_REREAD_FLOOR = 400 << 20
# Up to 64 rows are at most four tiles: four times these weights are below the floor, and the rule costs the host 1 us.
SHARED_INLINE_FEW_ROWS, SHARED_INLINE_FEW_ROWS_MAX_WEIGHT = 64, 32 << 20
# With more tokens they still are where the routed experts' launches have tiles of 128 tokens (more than 40 pairs per expert on
# average) and little enough to read that launches, last rounds and the SwiGLU pass of a separate MLP weigh.  At 1024, 1500 and
# 2048 tokens, inline / separate: 64 experts of 2048 x 1408 200 / 216, 255 / 258, 308 / 317; 8 of those 64 68 / 90, 89 / 111,
# 100 / 123; 20 of 160 of 5120 x 1536 (64-token tiles at 1024) 229 / 199, 216 / 224, 261 / 272; 32 of 256 of 7168 x 2048 (64-token
# tiles at 1024) 370 / 357, 411 / 426, 483 / 483; but 160 of 5120 x 1536 (64-token tiles at 1024) 790 / 768, 876 / 862, 1000 / 1024,
# 256 of 7168 x 2048 2326 / 2295 at 2048, and at 4096 32 of those 256 765 / 747: those draw the board's full power either way, and
# pairs of SMs multiply with fewer operand bytes.
SHARED_INLINE_MAX_ROWS_SMALL = 2048
SHARED_INLINE_MAX_BYTES_SMALL = 1500 << 20      # of the local experts' weights


def _shared_inline(st, rows: int, topk: int, n_routed: int, shared_width: int) -> bool:
    local_bytes = 3 * st.n * st.inter * st.dim
    pairs = -(-rows * topk // max(n_routed, st.n))                    # of an expert: what the tiles' width is chosen by (stream_tile)
    if pairs <= 40:
        reread = 3 * shared_width * st.dim * rows // (16 if pairs <= 4 else 32 if pairs <= 24 else 64)
        return rows <= SHARED_INLINE_MAX_ROWS and reread <= max(local_bytes, SHARED_INLINE_REREAD_FLOOR)
    return rows <= SHARED_INLINE_MAX_ROWS or rows <= SHARED_INLINE_MAX_ROWS_SMALL and local_bytes <= SHARED_INLINE_MAX_BYTES_SMALL


def _look_up(obj, name):
    """The attribute and the dictionary entries it was found through (one None where it lives elsewhere)."""
    value = getattr(obj, name)
    own = getattr(obj, "__dict__", None)
    if type(own) is dict:
        if own.get(name) is value:
            return value, [(own, name, value)]
        for kind in ("_parameters", "_modules", "_buffers"):
            d = own.get(kind)
            if type(d) is dict and d.get(name) is value:
                return value, [(own, kind, d), (d, name, value)]
    return value, [None]


class GroupedExperts:
    """Device tables (tensor maps, pointers of scales and weights) of the local experts' three projections."""

    def __init__(self, container, experts: List, start: int):
        self.start = start
        self.n = len(experts)
        self.container = container
        e0 = experts[0]
        self.dim = e0.w1.weight.size(1)
        self.inter = e0.w1.weight.size(0)
        self.scale_fmt = getattr(e0.w1, "scale_fmt", None)
        self.device = e0.w1.weight.device
        # every look-up from the container to a weight's and its scales' storage that the tables depend on
        found, weights, scales, by_name = [], [], [], {"w1": [], "w3": [], "w2": []}
        if not isinstance(container, list):
            members = getattr(container, "_modules", None)
            if type(members) is dict:
                found.append((container.__dict__, "_modules", members))
            found += [(members, str(start + i), e) if type(members) is dict else None for i, e in enumerate(experts)]
        for e in experts:
            for name in by_name:
                lin, step = _look_up(e, name)
                w, step2 = _look_up(lin, "weight")
                s, step3 = _look_up(w, "scale")
                found += step + step2 + step3
                weights.append(w)
                scales.append(s)
                by_name[name].append((w, s))
        self.watched = all(f is not None for f in found)      # otherwise they are looked up on every pass
        tables = {}
        for name, N, K in (("w1", self.inter, self.dim), ("w3", self.inter, self.dim), ("w2", self.dim, self.inter)):
            pairs, shape = by_name[name], torch.Size((N, K))
            for w, s in pairs:
                assert w.element_size() == 1 and w.is_contiguous() and s.is_contiguous() and s.dtype == torch.float32
                assert w.shape == shape
            table = torch.empty(lib.dsv3_group_table_bytes(self.n), dtype=torch.uint8, device=self.device)
            wp = (ctypes.c_void_p * self.n)(*[w.data_ptr() for w, _ in pairs])
            sp = (ctypes.c_void_p * self.n)(*[s.data_ptr() for _, s in pairs])
            with torch.cuda.device(self.device):
                _lib.check(lib.dsv3_group_table_build(table.data_ptr(), wp, sp, self.n, N, K, _stream()))
            tables[name] = table
        self._keep = (experts, scales)                        # the tables point into these
        self.signature = None if self.watched else self._addresses(container)
        self.handle = host.experts(self.n, start, self.dim, self.inter, self.scale_fmt, tables["w1"], tables["w3"], tables["w2"],
                                   container if isinstance(container, list) else None, list(experts),
                                   found if self.watched else [], weights + scales)

    def _addresses(self, container):
        """Storage of every weight and its scales, looked up from the container."""
        found = []
        for i in range(self.start, self.start + self.n):
            for name in ("w1", "w3", "w2"):
                w = getattr(container[i], name).weight
                found += [w.data_ptr(), w.scale.data_ptr()]
        return found

    def current(self, moe) -> bool:
        """Whether ``moe``'s local experts are still the ones the tables were built from."""
        if moe.experts is not self.container or moe.experts_start_idx != self.start or moe.experts_end_idx != self.start + self.n:
            return False
        if not self.watched and self.signature != self._addresses(self.container):
            return False
        return host.experts_current(self.handle)

    def run(self, x: torch.Tensor, weights: torch.Tensor, indices: torch.Tensor, n_routed: int = 0, shared=None):
        """The local experts' outputs for the routed tokens (model.py:683-688), to be handed to ``combine``: routing
        bookkeeping and quantisation, w1 / w3 with SwiGLU and quantisation, w2, nothing read back.  With few pairs w2 is
        left to ``combine`` (``host.weights_pending``): until then, and on the same stream, the weights must stay what they
        were.  ``n_routed``: experts of the whole layer (this rank owns ``self.n`` of them and, on average, that share of the
        pairs).  ``shared``: the shared experts' (w1, w3, w2), to be worked on in the same launches; ``combine`` then adds
        their output."""
        return host.run_experts(self.handle, x, weights, indices, n_routed, linear_seam._assume_no_inplace, shared)

    def routed(self, x: torch.Tensor, weights: torch.Tensor, indices: torch.Tensor, n_routed: int = 0) -> torch.Tensor:
        """Sum over the local experts of ``expert(x[idx]) * weights`` (model.py:683-689)."""
        return host.combine(self.run(x, weights, indices, n_routed), None)


def _grouped(moe) -> GroupedExperts:
    st = getattr(moe, "_dsv3_grouped", None)
    if st is None or not st.current(moe):
        local = [moe.experts[i] for i in range(moe.experts_start_idx, moe.experts_end_idx)]
        st = GroupedExperts(moe.experts, local, moe.experts_start_idx)
        object.__setattr__(moe, "_dsv3_grouped", st)      # not a Module/Parameter: keep it out of the registry
    return st


def grouped_moe_forward(self, x: torch.Tensor, *, world_size: int = 1, fallback=None) -> torch.Tensor:
    """Same inputs and outputs as ``MoE.forward`` (model.py:669-693)."""
    e0 = self.experts[self.experts_start_idx]
    if e0.w1.weight.element_size() != 1 or x.dtype != torch.bfloat16 or self.n_local_experts > 256:
        if fallback is None:
            raise NotImplementedError("grouped MoE needs FP8 expert weights, bf16 activations and <= 256 local experts")
        return fallback(self, x)
    shape = x.size()
    flat = len(shape) == 2 and shape[1] == self.dim       # (a view costs the host 2 us)
    if not flat:
        x = x.view(-1, self.dim)
    weights, indices = self.gate(x)
    st = _grouped(self)
    n_routed = getattr(self, "n_routed_experts", 0)
    shared = None
    rows = x.size(0)
    if world_size == 1 and rows <= SHARED_INLINE_MAX_ROWS_SMALL and 0 < indices.numel():     # (no pairs: no launch to join)
        shared = plain_weights(self.shared_experts, x, st.scale_fmt)
        if (shared is not None and (rows > SHARED_INLINE_FEW_ROWS or shared[0].numel() > SHARED_INLINE_FEW_ROWS_MAX_WEIGHT)
                and not _shared_inline(st, rows, indices.size(-1), n_routed, shared[0].size(0))):
            shared = None
    routed = st.run(x, weights, indices, n_routed, shared)
    if shared is not None:
        y = host.combine(routed, None)
    else:
        # the shared experts may be any code of the host's: what still reads the routed experts' weights is launched before it
        y = host.combine(routed, None) if world_size > 1 or host.weights_pending(routed) else None
        z = self.shared_experts(x)
        if y is not None:
            if world_size > 1:
                import torch.distributed as dist
                dist.all_reduce(y)
            y = y + z
        elif (z.dtype == torch.bfloat16 and z.is_contiguous() and z.size() == x.size() and z.data_ptr() % 16 == 0
              and not z.requires_grad):
            y = host.combine(routed, z)
        else:
            y = host.combine(routed, None) + z          # any tensor that can be added, with its gradient
    return y if flat else y.view(shape)


def install_moe(model_module) -> None:
    """Replace ``model_module.MoE.forward``; ``model_module.world_size`` is read at call time."""
    original = model_module.MoE.forward

    def forward(self, x):
        if getattr(model_module, "gemm_impl", "fp8") != "fp8":
            return original(self, x)
        return grouped_moe_forward(self, x, world_size=model_module.world_size, fallback=original)

    forward.__doc__ = grouped_moe_forward.__doc__
    model_module.MoE.forward = forward
