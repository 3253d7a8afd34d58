"""The expert layer's dispatch where a CTA's blocks end inside a round of the half-warps: every token's FP8 row and scales, and their
copies at the rows of its local pairs, against act_quant."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# blocks of a CTA: one per token (dim 128), fewer than a round, a round and a remainder, several rounds; topk up to the largest
@pytest.mark.parametrize("T,topk,dim,n", [(1, 1, 128, 4), (1000, 2, 128, 8), (40, 32, 384, 64), (300, 6, 7168, 16), (2000, 8, 1152, 5), (5, 3, 16384, 256)])
@pytest.mark.parametrize("fmt", [0, 1])
def test_rows_and_their_copies(T, topk, dim, n, fmt):
    import kernel
    from dsv3_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(T + dim)
    start, E, P = 3, n + 7, T * topk
    x = torch.randn(T, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    w, idx = torch.rand(T, max(E, topk), generator=g, device="cuda", dtype=torch.float32).topk(topk, dim=-1)
    i32 = dict(dtype=torch.int32, device="cuda")
    seg, pos = torch.empty(n + 1, **i32), torch.empty(T, topk, **i32)
    ws, xq, xs = torch.empty(T, topk, device="cuda", dtype=torch.bfloat16), torch.empty(T, dim, dtype=torch.uint8, device="cuda"), torch.empty(T, dim // 128, device="cuda", dtype=torch.float32)
    xr, xst = torch.zeros(P, dim, dtype=torch.uint8, device="cuda"), torch.full((dim // 128, P), -1.0, device="cuda", dtype=torch.float32)
    p, i64 = (lambda t: ctypes.c_void_p(t.data_ptr())), ctypes.c_int64
    _lib.check(_lib.lib.dsv3_moe_dispatch(p(x), i64(T), i64(dim), p(idx), p(w), 0, topk, start, n, fmt, p(seg), p(pos), p(ws), p(xq), p(xs), p(xr),
                                          p(xst), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want, scales = kernel.act_quant(x, 128, "ue8m0" if fmt else None)
    want = want.view(torch.uint8)
    assert torch.equal(xq, want) and torch.equal(xs, scales)
    order = idx.sort(dim=1).indices
    key = idx.gather(1, order) - start
    local = (key >= 0) & (key < n)
    assert torch.equal(pos >= 0, local) and torch.equal(ws, w.gather(1, order).bfloat16())
    rows, tok = pos[local].long(), torch.arange(T, device="cuda")[:, None].expand(T, topk)[local]
    assert torch.equal(rows.sort().values, torch.arange(int(seg[n]), device="cuda"))
    assert bool(((rows >= seg[key[local]]) & (rows < seg[key[local] + 1])).all())
    assert torch.equal(xr[rows], want[tok]) and torch.equal(xst.t()[rows], scales[tok])
    assert not bool(xr[int(seg[n]):].any()) and bool((xst[:, int(seg[n]):] == -1).all())
