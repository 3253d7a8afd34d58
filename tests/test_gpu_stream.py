"""The expert layer's launches (dispatch, w1/w3 with SwiGLU and quantisation, w2, combine), the cluster split-K of fp8_gemm
and the fast SwiGLU arithmetic, at the sizes where tiles, pieces and ranges end.

References: the separate operators (act_quant, fp8_gemm, swiglu_quant), which the other tests hold against the oracle, the
CUDA-core GEMM, and the framework's own silu.  Tolerances: two correct GEMMs differ by accumulation order only (1e-5
relative RMS measured), so bf16 results are held to the fp8_gemm bound 1e-2 (|y| + rms); behind SwiGLU and a quantisation
such a difference can move an e4m3 code by one step, 1/8 of the value, or 2^-9 of the block's scale below the normal range,
and a block's scale by one bf16 step of its maximum, 2^-7."""
import ctypes

import pytest
import torch

from gpu_util import assert_gemm_close, u8

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _bf16_default():
    import dsv3_b200
    torch.set_default_dtype(torch.bfloat16)
    yield
    torch.set_default_dtype(torch.float32)
    dsv3_b200.set_gemm_policy(0, 0)
    dsv3_b200.check_device_status()


def _weight(n, k, g):
    import dsv3_b200
    q, s = dsv3_b200.weight_quant((torch.randn(n, k, generator=g, device="cuda", dtype=torch.float32) * 0.02).bfloat16())
    q.scale = s
    return q


def _table(lib, check, ws, n, k):
    t = torch.empty(lib.dsv3_group_table_bytes(len(ws)), dtype=torch.uint8, device="cuda")
    wp = (ctypes.c_void_p * len(ws))(*[w.data_ptr() for w in ws])
    sp = (ctypes.c_void_p * len(ws))(*[w.scale.data_ptr() for w in ws])
    check(lib.dsv3_group_table_build(t.data_ptr(), wp, sp, len(ws), n, k, torch.cuda.current_stream().cuda_stream))
    return t


class _Side(ctypes.Structure):
    _fields_ = [("a", ctypes.c_void_p), ("a_s", ctypes.c_void_p), ("a_s_transposed", ctypes.c_int), ("rows", ctypes.c_int64),
                ("N", ctypes.c_int64), ("K", ctypes.c_int64), ("w", ctypes.c_void_p), ("w_s", ctypes.c_void_p), ("w3", ctypes.c_void_p),
                ("w3_s", ctypes.c_void_p), ("out", ctypes.c_void_p), ("out_s_t", ctypes.c_void_p)]


def _h_close(hq, hs_t, want_q, want_s):
    """e4m3 rows with transposed scales against the operators' rows, within the bounds of the module's head."""
    s = hs_t.t().repeat_interleave(128, dim=1)
    ws = want_s.repeat_interleave(128, dim=1)
    got, want = hq.float() * s, want_q.float() * ws
    assert bool(((hs_t.t() - want_s).abs() <= 2.0 ** -7 * want_s).all())
    assert bool(((got - want).abs() <= want.abs() / 8 + torch.maximum(s, ws) * 2.0 ** -9 + 2.0 ** -7 * want.abs()).all())


# rows per group: tile widths 16, 32, 64 and 128 and their edges, empty groups, one more row than a tile
@pytest.mark.parametrize("counts,inter,dim,side_rows", [
    ([1, 0, 2], 128, 256, 1),
    ([16, 17, 0, 1, 15], 384, 1024, 5),
    ([33, 31, 1, 24], 256, 640, 40),
    ([64, 65, 0, 20], 256, 768, 16),
    ([128, 129, 60, 0, 7], 256, 512, 130),
    ([0, 0, 3], 128, 7168, 3),
], ids=["decode", "tile16_32", "tile32", "tile64", "tile128", "long_k"])
@pytest.mark.parametrize("split", [True, False], ids=["workspace", "whole_tiles"])
def test_expert_gemms_match_the_operators_per_group(counts, inter, dim, side_rows, split):
    import kernel
    from dsv3_b200 import _lib, swiglu_quant
    lib, check = _lib.lib, _lib.check
    g = torch.Generator(device="cuda").manual_seed(sum(counts) * 7 + dim)
    n, rows = len(counts), sum(counts) + 3                     # three rows beyond the last group: never written
    w1, w3, w2 = ([_weight(a, b, g) for _ in counts] for a, b in ((inter, dim), (inter, dim), (dim, inter)))
    xq, xs = kernel.act_quant(torch.randn(rows, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16())
    xs_t = xs.t().contiguous()
    seg = torch.tensor([sum(counts[:i]) for i in range(n + 1)], dtype=torch.int32, device="cuda")
    sxq, sxs = kernel.act_quant(torch.randn(side_rows, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16())
    s1, s3, s2 = _weight(128, dim, g), _weight(128, dim, g), _weight(dim, 128, g)
    hq = torch.full((rows, inter), 7, dtype=torch.uint8, device="cuda")
    hs = torch.full((inter // 128, rows), -1.0, dtype=torch.float32, device="cuda")
    o = torch.full((rows, dim), 7.0, device="cuda")
    zq = torch.empty(side_rows, 128, dtype=torch.uint8, device="cuda")
    zs = torch.empty(1, side_rows, dtype=torch.float32, device="cuda")
    z = torch.empty(side_rows, dim, device="cuda")
    lib.dsv3_gemm_rows_workspace_bytes.restype = ctypes.c_size_t
    need = lib.dsv3_gemm_rows_workspace_bytes(n, ctypes.c_int64(rows), ctypes.c_int64(0))
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    i64, p = ctypes.c_int64, lambda t: ctypes.c_void_p(t.data_ptr())
    tail = (p(ws) if split else None, ctypes.c_size_t(need if split else 0), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    t1, t3, t2 = _table(lib, check, w1, inter, dim), _table(lib, check, w3, inter, dim), _table(lib, check, w2, dim, inter)
    up = _Side(sxq.data_ptr(), sxs.data_ptr(), 0, side_rows, 128, dim, s1.data_ptr(), s1.scale.data_ptr(), s3.data_ptr(),
               s3.scale.data_ptr(), zq.data_ptr(), zs.data_ptr())
    down = _Side(zq.data_ptr(), zs.data_ptr(), 1, side_rows, dim, 128, s2.data_ptr(), s2.scale.data_ptr(), None, None, z.data_ptr(), None)
    check(lib.dsv3_swiglu_gemm_rows(p(t1), p(t3), n, p(xq), p(xs_t), p(seg), i64(rows), i64(0), i64(inter), i64(dim), 0, p(hq), p(hs),
                                    ctypes.byref(up), *tail))
    check(lib.dsv3_fp8_gemm_rows(p(t2), n, p(hq), p(hs), p(seg), i64(rows), i64(0), i64(dim), i64(inter), p(o), ctypes.byref(down), *tail))
    torch.cuda.synchronize()
    hq8 = hq.view(torch.float8_e4m3fn)
    for e, c in enumerate(counts):
        if c == 0:
            continue
        r = slice(int(seg[e]), int(seg[e + 1]))
        a, a_s = xq[r].contiguous(), xs[r].contiguous()
        wq, wsc = swiglu_quant(kernel.fp8_gemm(a, a_s, w1[e], w1[e].scale), kernel.fp8_gemm(a, a_s, w3[e], w3[e].scale))
        _h_close(hq8[r], hs[:, r], wq, wsc)
        assert_gemm_close(o[r].cpu(), kernel.fp8_gemm(hq8[r].contiguous(), hs[:, r].t().contiguous(), w2[e], w2[e].scale).cpu())
    wq, wsc = swiglu_quant(kernel.fp8_gemm(sxq, sxs, s1, s1.scale), kernel.fp8_gemm(sxq, sxs, s3, s3.scale))
    _h_close(zq.view(torch.float8_e4m3fn), zs, wq, wsc)
    assert_gemm_close(z.cpu(), kernel.fp8_gemm(zq.view(torch.float8_e4m3fn), zs.t().contiguous(), s2, s2.scale).cpu())
    assert bool((hq[-3:] == 7).all()) and bool((hs[:, -3:] == -1).all()) and bool((o[-3:] == 7).all())
    assert not bool(ws[:_lib.WORKSPACE_HEADER_BYTES].any()), "tickets are left clean"


@pytest.mark.parametrize("T,topk,E,start,n,fmt", [(1, 8, 256, 224, 32, 0), (16, 8, 256, 0, 256, 1), (300, 6, 64, 16, 32, 0), (2100, 8, 256, 0, 256, 0)])
def test_dispatch_equals_routing_and_quantisation(T, topk, E, start, n, fmt):
    import kernel
    from dsv3_b200 import _lib
    lib = _lib.lib
    g = torch.Generator(device="cuda").manual_seed(T)
    dim, P = 512, T * topk
    x = torch.randn(T, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    w, idx = torch.rand(T, E, generator=g, device="cuda", dtype=torch.float32).topk(topk, dim=-1)
    i32 = dict(dtype=torch.int32, device="cuda")
    seg, pos, ws = torch.empty(n + 1, **i32), torch.empty(T, topk, **i32), torch.empty(T, topk, device="cuda")
    xq, xs = torch.empty(T, dim, dtype=torch.uint8, device="cuda"), torch.empty(T, dim // 128, dtype=torch.float32, device="cuda")
    xr, xst = torch.empty(P, dim, dtype=torch.uint8, device="cuda"), torch.empty(dim // 128, P, dtype=torch.float32, device="cuda")
    p, i64 = (lambda t: ctypes.c_void_p(t.data_ptr())), ctypes.c_int64
    _lib.check(lib.dsv3_moe_dispatch(p(x), i64(T), i64(dim), p(idx), p(w), 0, topk, start, n, fmt, p(seg), p(pos), p(ws), p(xq), p(xs), p(xr),
                                     p(xst), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    wq, wsc = kernel.act_quant(x, 128, "ue8m0" if fmt else None)
    assert torch.equal(xq, wq.view(torch.uint8)) and torch.equal(xs, wsc)
    key = idx - start
    local = (key >= 0) & (key < n)
    counts = torch.bincount(key[local], minlength=n)
    assert torch.equal(seg.long(), torch.cat([counts.new_zeros(1), counts.cumsum(0)]))
    order = idx.sort(dim=1).indices
    k_s, l_s = key.gather(1, order), local.gather(1, order)
    assert torch.equal(pos >= 0, l_s) and torch.equal(ws, w.gather(1, order).bfloat16())
    rows, tok = pos[l_s].long(), torch.arange(T, device="cuda")[:, None].expand(T, topk)[l_s]
    assert torch.equal(rows.sort().values, torch.arange(int(seg[n]), device="cuda"))
    assert bool(((rows >= seg[k_s[l_s]]) & (rows < seg[k_s[l_s] + 1])).all())
    assert torch.equal(xr[rows], xq[tok]) and torch.equal(xst.t()[rows], xs[tok])


# the automatic plan splits these inside clusters of two to eight CTAs: row shares that do and do not divide 128, the last
# weight tile cut by N, rows not divisible by 8, a K tail, every token tile of the weight-major kernel and the token-major one
@pytest.mark.parametrize("M", [1, 3, 16, 17, 33, 64, 65, 128, 200])
@pytest.mark.parametrize("N,K", [(128, 7168), (576, 7168), (203, 4096), (1536, 5120 + 16), (2048, 7168)])
def test_cluster_split_k_against_the_cuda_core_kernel(M, N, K):
    import dsv3_b200
    import kernel
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    kc = -(-K // 128)
    a = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float32).to(torch.float8_e4m3fn)
    b = torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32).to(torch.float8_e4m3fn)
    a_s = torch.rand(M, kc, generator=g, device="cuda", dtype=torch.float32) + 0.5
    b_s = torch.rand(-(-N // 128), kc, generator=g, device="cuda", dtype=torch.float32) + 0.5
    y = kernel.fp8_gemm(a, a_s, b, b_s)
    assert torch.equal(y, kernel.fp8_gemm(a, a_s, b, b_s)), "the splits are added in a fixed order"
    dsv3_b200.set_gemm_policy(dsv3_b200.KERNEL_CUDA_CORE, 0)
    assert_gemm_close(y.cpu(), kernel.fp8_gemm(a, a_s, b, b_s).cpu())


# up to 8 rows and 8 MB of weights: the decode kernel's warps and CTAs each add a part of K -- one row group and one chunk, rows
# that end inside a group, K tails, the largest N, the longest K
@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("N,K", [(1, 16), (16, 128), (17, 16384), (512, 16384), (576, 7056), (4096, 2048), (4095, 1040)])
def test_decode_kernel_against_the_cuda_core_kernel(M, N, K):
    test_cluster_split_k_against_the_cuda_core_kernel(M, N, K)


def test_swiglu_fast_form_equals_the_frameworks_silu_for_every_bf16():
    """swiglu8 rounds its fast silu a little below and above itself and falls back where the two differ: every finite bf16
    value of a, against act_quant(F.silu(a) * b) bit for bit."""
    import kernel
    from dsv3_b200 import swiglu_quant
    a = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16).reshape(512, 128)
    a = a[torch.isfinite(a.float()).all(dim=1)].contiguous()
    for scale in (1.0, 3.1e-2, 117.0):
        b = torch.full_like(a, scale) * torch.where(torch.arange(128, device="cuda") % 3 == 0, -1.0, 1.0).bfloat16()
        b = torch.where(a.float().abs() > 1e34, torch.ones_like(b), b)        # keep the products finite
        q, s = swiglu_quant(a, b)
        wq, wsc = kernel.act_quant(torch.nn.functional.silu(a) * b)
        assert torch.equal(s, wsc) and (u8(q) == u8(wq)).all()
