"""fp8_gemm of one activation with two weights in one launch: bit for bit what the wide tiles write for either weight alone, at the ends of tiles,
with results that no TMA store can write, scales of every load width, last rounds in strips and a machine of a few pairs (an SM budget);
and the MLPs that it serves against the separate operators."""
import ctypes

import pytest
import torch

from test_gpu_mlp_launches import _host, _i64, _rows
from test_gpu_expert_launches import _kernels
from test_gpu_stream import _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu

WIDE = 6      # kernel policy


def _two(xq, xs, w, ws, M, N, K):
    from dsv3_b200 import _lib
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    y = [torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    rc = _lib.lib.dsv3_fp8_gemm_two(p(xq), p(xs), p(w[0]), p(ws[0]), p(w[1]), p(ws[1]), _i64(M), _i64(N), _i64(K), p(y[0]), p(y[1]),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return rc, y


@pytest.mark.parametrize("M,N,K,sms", [
    (129, 129, 128, 0),        # a tile each, a row and a column into the second halves
    (256, 256, 512, 0),
    (300, 648, 1152, 0),       # three tiles a weight, the last 136 columns wide; 9 chunks
    (700, 1301, 3280, 24),     # 18 a weight on 12 pairs: whole rounds; N odd, a K tail
    (257, 520, 640, 8),        # six a weight on four pairs
    (500, 900, 640, 14),       # eight a weight on seven pairs: a last round of two tiles in strips of 64, which are the second weight's
    (300, 256, 3200, 12),      # two a weight on six pairs
    (256, 600, 3200, 8),       # three a weight on four pairs: strips of 128, the last tile 88 columns wide
    (1100, 2304, 1280, 0),     # 45 a weight
])
def test_equals_the_wide_tiles_of_either_weight(M, N, K, sms):
    import dsv3_b200
    import kernel
    g = torch.Generator(device="cuda").manual_seed(M + N)
    kp = -(-K // 128) * 128
    x = torch.randn(M, kp, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    x[:, K:] = 0
    xq, xs = kernel.act_quant(x)
    xq = xq.view(torch.uint8)[:, :K].contiguous().view(torch.float8_e4m3fn)
    w, ws = zip(*(dsv3_b200.weight_quant((torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32) * 0.02).bfloat16()) for _ in range(2)))
    if sms:
        dsv3_b200.set_num_sms(sms)
    try:
        rc, y = _two(xq, xs, w, ws, M, N, K)
        assert rc == 0
        dsv3_b200.set_gemm_policy(WIDE, 0)
        for i in range(2):
            assert torch.equal(y[i][:M], kernel.fp8_gemm(xq, xs, w[i], ws[i]))
            assert bool((y[i][M] == 7).all()), "rows beyond the last are not written"
    finally:
        dsv3_b200.set_gemm_policy(0, 0)
        dsv3_b200.set_num_sms(0)
        dsv3_b200.check_device_status()


@pytest.mark.parametrize("M,N,K", [(128, 256, 256), (300, 128, 256), (300, 256, 264)])
def test_other_sizes_are_refused(M, N, K):
    t = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    rc, y = _two(t, t, (t, t), (t, t), M, N, K)
    assert rc != 0 and all(bool((r == 7).all()) for r in y)


@pytest.mark.parametrize("dim,inter,M", [(2048, 1408, 2580), (7168, 2304, 2580), (5120, 3072, 2201), (2048, 2816, 3942)])
@pytest.mark.parametrize("fmt", [None, "ue8m0"])
def test_an_mlp_of_four_launches(dim, inter, M, fmt):
    import kernel
    from dsv3_b200 import _lib, swiglu_quant
    from dsv3_b200._lib import host
    pays = _lib.lib.dsv3_fp8_gemm_two_pays
    assert pays(_i64(M), _i64(inter), _i64(dim)) and not _lib.lib.dsv3_swiglu_linear_pays(_i64(M), _i64(inter), _i64(dim))
    mlp, model = _host(dim, inter)
    x = _rows(M, dim)
    got = host.mlp(x, mlp.w1.weight, mlp.w3.weight, mlp.w2.weight, fmt, fmt, False)
    ws = [(lin.weight, lin.weight.scale) for lin in (mlp.w1, mlp.w3, mlp.w2)]
    q = kernel.act_quant(x, 128, fmt)
    h = swiglu_quant(kernel.fp8_gemm(*q, *ws[0]), kernel.fp8_gemm(*q, *ws[1]), fmt)
    assert torch.equal(got, kernel.fp8_gemm(*h, *ws[2]))
    if fmt is None:
        assert torch.equal(got, mlp(x))
        assert len(_kernels(lambda: mlp(x.view(x.shape)))) == 4
        y3 = mlp(x.view(1, M, dim))
        assert y3.shape == (1, M, dim) and torch.equal(y3[0], got)


@pytest.mark.parametrize("dim,inter,M", [(7168, 2304, 2580), (2048, 2816, 3942)])
def test_memory_of_an_mlp_of_four_launches(dim, inter, M):
    """No more at its peak than the operators one by one, each of whose inputs is given back once it has been read."""
    import kernel
    from dsv3_b200 import swiglu_quant
    from dsv3_b200._lib import host
    mlp, model = _host(dim, inter)
    w1, w3, w2 = mlp.w1.weight, mlp.w3.weight, mlp.w2.weight
    x = _rows(M, dim)

    def one_by_one():
        q, s = kernel.act_quant(x)
        y1, y3 = kernel.fp8_gemm(q, s, w1, w1.scale), kernel.fp8_gemm(q, s, w3, w3.scale)
        del q, s
        h = swiglu_quant(y1, y3)
        del y1, y3
        return kernel.fp8_gemm(*h, w2, w2.scale)

    def peak(run):
        run()                                     # workspaces
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        run()
        return torch.cuda.max_memory_allocated() - before

    with torch.inference_mode():                  # a tensor without a modification counter: its quantisation is not kept
        x = x.clone()
        assert peak(lambda: host.mlp(x, w1, w3, w2, None, None, False)) <= peak(one_by_one)


@pytest.mark.parametrize("which", [0, 1])
def test_weights_off_16_bytes_take_the_separate_launches(which):
    import kernel
    from dsv3_b200 import _lib, swiglu_quant
    from dsv3_b200._lib import host
    dim, inter, M = 2048, 1408, 2580
    assert _lib.lib.dsv3_fp8_gemm_two_pays(_i64(M), _i64(inter), _i64(dim))
    mlp, model = _host(dim, inter)
    lin = (mlp.w1, mlp.w3)[which]
    scale = lin.weight.scale
    w = torch.empty(inter * dim + 1, dtype=torch.uint8, device="cuda")[1:].view(lin.weight.dtype).view(inter, dim)
    w.view(torch.uint8).copy_(lin.weight.view(torch.uint8))
    lin.weight = torch.nn.Parameter(w, requires_grad=False)
    lin.weight.scale = scale
    assert lin.weight.data_ptr() % 16
    x = _rows(M, dim)
    assert host.mlp(x, mlp.w1.weight, mlp.w3.weight, mlp.w2.weight, None, None, False) is None
    q = kernel.act_quant(x)
    h = swiglu_quant(*(kernel.fp8_gemm(*q, lin.weight, lin.weight.scale) for lin in (mlp.w1, mlp.w3)))
    assert torch.equal(mlp(x), kernel.fp8_gemm(*h, mlp.w2.weight, mlp.w2.weight.scale))
