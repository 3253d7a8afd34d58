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
