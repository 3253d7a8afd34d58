"""Tiles of the expert GEMMs (w1/w3 with SwiGLU and quantisation, w2): whole and cut over K.

References: the separate operators per group of rows.  Whole tiles fold every chunk as the other tcgen05 kernels do, so
with the operators pinned to one split the results are equal bit for bit; a cut tile adds the same terms in another
order and is held to the bounds of test_gpu_stream.py."""
import ctypes

import pytest
import torch

from gpu_util import assert_gemm_close
from test_gpu_stream import _Side, _bf16_default, _h_close, _table, _weight  # noqa: F401

pytestmark = pytest.mark.gpu


class _Layer:
    """w1 / w3 / w2 of len(counts) groups, their rows, and an ordinary weight of side_rows rows next to them."""

    def __init__(self, counts, inter, dim, side_rows, seed=0):
        import kernel
        from dsv3_b200 import _lib
        self.counts, self.inter, self.dim, self.side_rows = counts, inter, dim, side_rows
        g = torch.Generator(device="cuda").manual_seed(seed + sum(counts) * 7 + dim)
        rows = lambda m, k: torch.randn(m, k, generator=g, device="cuda", dtype=torch.float32).bfloat16()
        self.n, self.rows = len(counts), sum(counts)
        self.w1, self.w3, self.w2 = ([_weight(a, b, g) for _ in counts] for a, b in ((inter, dim), (inter, dim), (dim, inter)))
        self.tables = [_table(_lib.lib, _lib.check, w, *w[0].shape) for w in (self.w1, self.w3, self.w2)]
        self.xq, self.xs = kernel.act_quant(rows(self.rows, dim))
        self.xs_t = self.xs.t().contiguous()
        self.seg = torch.tensor([sum(counts[:i]) for i in range(self.n + 1)], dtype=torch.int32, device="cuda")
        if side_rows:
            self.sq, self.ss = kernel.act_quant(rows(side_rows, dim))
            self.s1, self.s3, self.s2 = _weight(256, dim, g), _weight(256, dim, g), _weight(dim, 256, g)
        lib = _lib.lib
        lib.dsv3_gemm_rows_workspace_bytes.restype = ctypes.c_size_t
        self.need = lib.dsv3_gemm_rows_workspace_bytes(self.n, ctypes.c_int64(self.rows), ctypes.c_int64(0))

    def run(self, workspace=None, between=lambda: None):
        """(hq, hs_t, o) and, with side_rows, (zq, zs_t, z)."""
        from dsv3_b200 import _lib
        lib, i64, p = _lib.lib, ctypes.c_int64, lambda t: ctypes.c_void_p(t.data_ptr())
        f8, f32 = dict(dtype=torch.uint8, device="cuda"), dict(dtype=torch.float32, device="cuda")
        hq, hs, o = torch.zeros(self.rows, self.inter, **f8), torch.zeros(self.inter // 128, self.rows, **f32), torch.zeros(self.rows, self.dim, device="cuda")
        out, up, down = [hq, hs, o], None, None
        if self.side_rows:
            m = self.side_rows
            zq, zs, z = torch.zeros(m, 256, **f8), torch.zeros(2, m, **f32), torch.zeros(m, self.dim, device="cuda")
            out += [zq, zs, z]
            up = ctypes.byref(_Side(self.sq.data_ptr(), self.ss.data_ptr(), 0, m, 256, self.dim, self.s1.data_ptr(), self.s1.scale.data_ptr(),
                                    self.s3.data_ptr(), self.s3.scale.data_ptr(), zq.data_ptr(), zs.data_ptr()))
            down = ctypes.byref(_Side(zq.data_ptr(), zs.data_ptr(), 1, m, self.dim, 256, self.s2.data_ptr(), self.s2.scale.data_ptr(), None, None,
                                      z.data_ptr(), None))
        tail = (p(workspace) if workspace is not None else None, ctypes.c_size_t(workspace.numel() if workspace is not None else 0),
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        t1, t3, t2 = self.tables
        _lib.check(lib.dsv3_swiglu_gemm_rows(p(t1), p(t3), self.n, p(self.xq), p(self.xs_t), p(self.seg), i64(self.rows), i64(0), i64(self.inter),
                                             i64(self.dim), 0, p(hq), p(hs), up, *tail))
        between()
        _lib.check(lib.dsv3_fp8_gemm_rows(p(t2), self.n, p(hq), p(hs), p(self.seg), i64(self.rows), i64(0), i64(self.dim), i64(self.inter), p(o), down,
                                          *tail))
        torch.cuda.synchronize()
        return out

    def operators(self, hq, hs, zq=None, zs=None):
        """The operators' results per group; w2 works on the given hq / hs (and s2 on zq / zs)."""
        import kernel
        from dsv3_b200 import swiglu_quant
        f8 = torch.float8_e4m3fn
        parts = []
        for e, c in enumerate(self.counts):
            if c:
                r = slice(sum(self.counts[:e]), sum(self.counts[:e + 1]))
                a = (self.xq[r].contiguous(), self.xs[r].contiguous())
                q, s = swiglu_quant(kernel.fp8_gemm(*a, self.w1[e], self.w1[e].scale), kernel.fp8_gemm(*a, self.w3[e], self.w3[e].scale))
                parts.append((q, s.t(), kernel.fp8_gemm(hq[r].contiguous().view(f8), hs[:, r].t().contiguous(), self.w2[e], self.w2[e].scale)))
        out = [torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts], dim=1), torch.cat([p[2] for p in parts])]
        if zq is not None:
            q, s = swiglu_quant(kernel.fp8_gemm(self.sq, self.ss, self.s1, self.s1.scale), kernel.fp8_gemm(self.sq, self.ss, self.s3, self.s3.scale))
            out += [q, s.t(), kernel.fp8_gemm(zq.view(f8), zs.t().contiguous(), self.s2, self.s2.scale)]
        return out


# every tile width (16, 32, 64 tokens with the weights on the M side, 128 with the tokens there), tiles with one row more
@pytest.mark.parametrize("counts,policy", [([3, 0, 1, 17, 1, 0, 2, 5], 3), ([16, 33, 0, 7], 3), ([64, 5, 65, 30], 3), ([128, 60, 0, 7, 129], 2)],
                         ids=["tile16", "tile32", "tile64", "tile128"])
def test_whole_tiles_equal_the_operators_bit_for_bit(counts, policy):
    import dsv3_b200
    layer = _Layer(counts, 384, 1152, 9)
    got = layer.run()
    dsv3_b200.set_gemm_policy(policy, 1)             # one split, chunks in order
    want = layer.operators(got[0], got[1], got[3], got[4])
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8) if a.element_size() == 1 else a, b.view(torch.uint8) if b.element_size() == 1 else b)


# Both launches are cut (33 and 16 K chunks; 33 weight blocks, so that w2's last tile holds one): two token tiles of one group,
# the second with one row, each in about five parts; and one round and a bit, where a range holds a head, a whole tile and a tail
_ONE = {16: [17, 0, 0, 0, 0, 0, 0], 32: [33, 0, 0], 64: [65, 0]}
_TEN = {16: [1, 2, 3, 4, 1, 2, 3, 4, 5, 2], 32: [9, 20, 3, 14, 11, 12, 23, 4, 15, 32], 64: [29, 40, 33, 64, 31, 32, 23, 44, 35, 32]}


@pytest.mark.parametrize("side_rows", [0, 9])
@pytest.mark.parametrize("tile", [16, 32, 64])
@pytest.mark.parametrize("groups", [_ONE, _TEN], ids=["parts", "ranges"])
def test_cut_tiles(groups, tile, side_rows):
    from dsv3_b200 import _lib
    header = _lib.WORKSPACE_HEADER_BYTES
    layer = _Layer(groups[tile], 2048, 4224, side_rows)
    ws = torch.zeros(layer.need, dtype=torch.uint8, device="cuda")
    ws[header:] = 0x55
    cut = []

    def parked():
        cut.append(bool((ws[header:] != 0x55).any()))
        assert not bool(ws[:header].any()), "tickets are left clean"
        ws[header:] = 0x55

    got = layer.run(ws, parked)
    parked()
    assert cut == [True, True], "partial tiles were parked by both launches"
    for a, b in zip(got, layer.run(ws)):
        assert torch.equal(a, b), "parts are added in K order, whoever comes last"
    want = layer.operators(got[0], got[1], *got[3:5])
    for i in range(0, len(got), 3):
        _h_close(got[i].view(torch.float8_e4m3fn), got[i + 1], want[i], want[i + 1].t())
        assert_gemm_close(got[i + 2].cpu(), want[i + 2].cpu())


# fewer and more than one pair per thread of a warp, one CTA's limit of pairs, more tokens than CTAs, few SMs; repeated experts
@pytest.mark.parametrize("T,topk,E,start,n,sms", [(1, 8, 256, 0, 256, 0), (40, 8, 16, 4, 8, 0), (1400, 8, 64, 0, 64, 0), (300, 32, 40, 8, 32, 2),
                                                   (4099, 6, 256, 128, 128, 0), (513, 2, 4, 0, 4, 4)])
def test_rows_of_an_expert_are_in_the_order_of_the_pairs(T, topk, E, start, n, sms):
    import dsv3_b200
    from dsv3_b200 import _lib
    lib, dim = _lib.lib, 128
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    idx = torch.randint(0, E, (T, topk), generator=g, device="cuda")
    w = torch.rand(T, topk, generator=g, device="cuda", dtype=torch.float32)
    P, i32, p, i64 = T * topk, dict(dtype=torch.int32, device="cuda"), (lambda t: ctypes.c_void_p(t.data_ptr())), ctypes.c_int64
    seg, pos, ws = torch.empty(n + 1, **i32), torch.empty(T, topk, **i32), torch.empty(T, topk, device="cuda")
    xq, xs = torch.empty(T, dim, dtype=torch.uint8, device="cuda"), torch.empty(T, 1, dtype=torch.float32, device="cuda")
    xr, xst = torch.empty(P, dim, dtype=torch.uint8, device="cuda"), torch.empty(1, P, dtype=torch.float32, device="cuda")
    dsv3_b200.set_num_sms(sms)
    try:
        _lib.check(lib.dsv3_moe_dispatch(p(x), i64(T), i64(dim), p(idx), p(w), 0, topk, start, n, 0, p(seg), p(pos), p(ws), p(xq), p(xs), p(xr),
                                         p(xst), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    finally:
        dsv3_b200.set_num_sms(0)
    key = (idx - start).flatten()
    local = (key >= 0) & (key < n)
    order = torch.where(local, key, n).sort(stable=True).indices           # pairs by expert, then as they come
    row = torch.empty_like(order)
    row[order] = torch.arange(P, device="cuda")
    row = torch.where(local, row, -1).view(T, topk)
    assert torch.equal(pos.long(), row.gather(1, idx.sort(dim=1, stable=True).indices))
