"""dsv3_expert_gemms: w2's launch reads its weights while w1's and w3's still runs, and everything that launch writes behind it.

Reference: the two launches by themselves with a synchronisation in between, whose order of sums is the same: equal bit for bit."""
import ctypes

import pytest
import torch

from test_gpu_expert_tiles import _Layer
from test_gpu_stream import _Side, _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


def _together(layer, ws, out):
    from dsv3_b200 import _lib
    i64, p = ctypes.c_int64, lambda t: ctypes.c_void_p(t.data_ptr())
    up = down = None
    if layer.side_rows:
        m = layer.side_rows
        up = ctypes.byref(_Side(layer.sq.data_ptr(), layer.ss.data_ptr(), 0, m, 256, layer.dim, layer.s1.data_ptr(), layer.s1.scale.data_ptr(),
                                layer.s3.data_ptr(), layer.s3.scale.data_ptr(), out[3].data_ptr(), out[4].data_ptr()))
        down = ctypes.byref(_Side(out[3].data_ptr(), out[4].data_ptr(), 1, m, layer.dim, 256, layer.s2.data_ptr(), layer.s2.scale.data_ptr(), None,
                                  None, out[5].data_ptr(), None))
    t1, t3, t2 = layer.tables
    _lib.check(_lib.lib.dsv3_expert_gemms(p(t1), p(t3), p(t2), layer.n, p(layer.xq), p(layer.xs_t), p(layer.seg), i64(layer.rows), i64(0),
                                          i64(layer.inter), i64(layer.dim), 0, p(out[0]), p(out[1]), p(out[2]), up, down,
                                          p(ws) if ws is not None else None, ctypes.c_size_t(ws.numel() if ws is not None else 0),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


# one tile and fewer than the CTAs; cut tiles; whole tiles, K shorter and longer than the ring; divided, with second token tiles; CTAs without
# work; a budget
@pytest.mark.parametrize("counts,inter,dim,side_rows,workspace,sms", [
    ([1], 128, 128, 0, True, 0), ([0, 3, 1], 256, 1152, 9, True, 0), ([17, 0, 3, 16], 2048, 4224, 9, True, 0), ([16, 33, 0, 7], 384, 1152, 9, False, 0),
    ([64, 5, 65, 30], 1408, 512, 0, False, 0), ([128, 60, 0, 7, 129], 384, 1152, 9, False, 0), ([300, 200, 64, 65], 1024, 2048, 130, False, 0),
    ([300, 3, 64], 256, 512, 9, False, 8), ([5, 3, 2], 256, 512, 9, True, 2)],
    ids=["one", "few", "cut", "tile32", "tile64", "divided", "rounds", "budget", "budget2"])
def test_like_the_launches_one_after_the_other(counts, inter, dim, side_rows, workspace, sms):
    import dsv3_b200
    dsv3_b200.set_num_sms(sms)
    try:
        layer = _Layer(counts, inter, dim, side_rows)
        ws = torch.zeros(max(layer.need, 1), dtype=torch.uint8, device="cuda") if workspace else None
        other = layer.xq.flip(0).contiguous()
        inputs, weights = [layer.xq.clone(), other], [[w.clone() for w in layer.w2], [w.flip(0).clone() for w in layer.w2]]
        want = []
        for x, w2 in zip(inputs, weights):
            layer.xq.copy_(x)
            for w, v in zip(layer.w2, w2):
                w.copy_(v)
            want.append([t.clone() for t in layer.run(ws, torch.cuda.synchronize)])
        # the same memory for every pass, nothing waited for in between, activations and weights written on the stream
        out, got = [torch.empty_like(t) for t in want[0]], []
        for i in (0, 1, 1, 0, 1):
            layer.xq.copy_(inputs[i])
            for w, v in zip(layer.w2, weights[i]):
                w.copy_(v)
            for t in out:
                t.zero_()
            _together(layer, ws, out)
            got.append((i, [t.clone() for t in out]))
        for i, tensors in got:
            for a, b in zip(tensors, want[i]):
                assert torch.equal(a.view(torch.uint8) if a.element_size() == 1 else a, b.view(torch.uint8) if b.element_size() == 1 else b)
    finally:
        dsv3_b200.set_num_sms(0)


@pytest.mark.parametrize("wrong", ["table", "out", "dim"])
def test_refused_as_one(wrong):
    """An argument that only w2's launch is refused for leaves w1's and w3's results alone, too."""
    from dsv3_b200 import _lib
    i64, p = ctypes.c_int64, lambda t, at=0: ctypes.c_void_p(t.data_ptr() + at)
    layer = _Layer([5, 3, 2], 256, 512, 9)
    m, dim, (t1, t3, t2) = layer.side_rows, layer.dim, layer.tables
    out = [torch.full((layer.rows * 2048,), 7, dtype=torch.uint8, device="cuda") for _ in range(6)]
    hq, hs, o, zq, zs, z = out
    up = _Side(layer.sq.data_ptr(), layer.ss.data_ptr(), 0, m, 256, dim, layer.s1.data_ptr(), layer.s1.scale.data_ptr(), layer.s3.data_ptr(),
               layer.s3.scale.data_ptr(), zq.data_ptr(), zs.data_ptr())
    down = _Side(zq.data_ptr(), zs.data_ptr(), 1, m, dim, 256, layer.s2.data_ptr(), layer.s2.scale.data_ptr(), None, None,
                 z.data_ptr() + (2 if wrong == "out" else 0), None)
    if wrong == "dim":
        down.K = 8                     # no multiple of 16
    rc = _lib.lib.dsv3_expert_gemms(p(t1), p(t3), None if wrong == "table" else p(t2), layer.n, p(layer.xq), p(layer.xs_t), p(layer.seg),
                                    i64(layer.rows), i64(0), i64(layer.inter), i64(dim), 0, p(hq), p(hs), p(o), ctypes.byref(up), ctypes.byref(down),
                                    None, ctypes.c_size_t(0), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc != _lib.OK
    torch.cuda.synchronize()
    assert all(bool((t == 7).all()) for t in out)


# 3, 10, 30 and 100 rows per group: every tile width, whole and cut
@pytest.mark.parametrize("T,topk,n,inter,dim", [(6, 2, 4, 256, 512), (40, 2, 8, 2048, 1152), (120, 2, 8, 384, 1152), (400, 2, 8, 384, 512)])
@pytest.mark.parametrize("workspace", [True, False])
def test_routing_that_changes_from_pass_to_pass(T, topk, n, inter, dim, workspace):
    """The row offsets, which w2's launch reads while w1's and w3's still runs, are written by the dispatch in front of both, to the same
    memory in every pass and with other counts in each.  Reference: the launches with a synchronisation behind each."""
    from dsv3_b200 import _lib
    lib, i64, p = _lib.lib, ctypes.c_int64, lambda t: ctypes.c_void_p(t.data_ptr())
    layer = _Layer([1] * n, inter, dim, 0)
    t1, t3, t2 = layer.tables
    g = torch.Generator(device="cuda").manual_seed(T)
    E, P, start = n + 3, T * topk, 1
    x = torch.randn(T, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    w = torch.rand(T, topk, generator=g, device="cuda", dtype=torch.float32)
    # all experts alike; the first and the last local one only; half of the pairs elsewhere; no local ones
    prefer = [torch.zeros(E), torch.tensor([0.0, 9.0] + [0.0] * (n - 2) + [9.0] + [0.0] * (E - n - 1)), torch.tensor([9.0] + [0.0] * (E - 1)),
              torch.tensor([9.0] + [0.0] * n + [1.0] * (E - n - 1))]
    routings = [(torch.rand(T, E, generator=g, device="cuda") + q.cuda()).topk(topk, dim=-1).indices for q in prefer]
    size = dict(seg=4 * (n + 1), pos=4 * P, ws=2 * P, xq=T * dim, xs=4 * T * (dim // 128), xr=P * dim, xst=4 * P * (dim // 128), hq=P * inter,
                hs=4 * P * (inter // 128), o=2 * P * dim)
    b = {k: torch.zeros(v, dtype=torch.uint8, device="cuda") for k, v in size.items()}
    idx = torch.empty_like(routings[0])
    need = lib.dsv3_gemm_rows_workspace_bytes(n, i64(P), i64(0))
    space = torch.zeros(max(need, 1), dtype=torch.uint8, device="cuda") if workspace else None
    tail = (p(space) if workspace else None, ctypes.c_size_t(need if workspace else 0))
    results = ("seg", "hq", "hs", "o")

    def one_pass(i, between):
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for k in results[1:]:
            b[k].zero_()
        idx.copy_(routings[i])
        _lib.check(lib.dsv3_moe_dispatch(p(x), i64(T), i64(dim), p(idx), p(w), 0, topk, start, n, 0, p(b["seg"]), p(b["pos"]), p(b["ws"]), p(b["xq"]),
                                         p(b["xs"]), p(b["xr"]), p(b["xst"]), stream))
        rows = (p(b["seg"]), i64(P), i64(0))
        if between:
            between()
            _lib.check(lib.dsv3_swiglu_gemm_rows(p(t1), p(t3), n, p(b["xr"]), p(b["xst"]), *rows, i64(inter), i64(dim), 0, p(b["hq"]), p(b["hs"]), None,
                                                 *tail, stream))
            between()
            _lib.check(lib.dsv3_fp8_gemm_rows(p(t2), n, p(b["hq"]), p(b["hs"]), *rows, i64(dim), i64(inter), p(b["o"]), None, *tail, stream))
            between()
        else:
            _lib.check(lib.dsv3_expert_gemms(p(t1), p(t3), p(t2), n, p(b["xr"]), p(b["xst"]), *rows, i64(inter), i64(dim), 0, p(b["hq"]), p(b["hs"]),
                                             p(b["o"]), None, None, *tail, stream))
        return [b[k].clone() for k in results]

    want = [one_pass(i, torch.cuda.synchronize) for i in range(4)]
    assert all(not torch.equal(want[i][0], want[j][0]) for i in range(4) for j in range(i))
    got = [(i, one_pass(i, None)) for i in (0, 1, 2, 3, 1, 0, 3, 2, 0)]
    for i, tensors in got:
        assert all(torch.equal(a, c) for a, c in zip(tensors, want[i]))
