"""An MLP of plain Linears in three launches (w1 and w3 with SwiGLU and quantisation in one) against the separate operators, at the sizes
where the tiles of that launch change, cut over K and whole; and the calls that keep the separate launches.  Where no tile is cut both
sum in the same order and the FP8 codes in front of w2 are equal; where one is, a code may move by a step, which test_gpu_stream.py
bounds and which moves the result of w2 by less than the 2e-2 (|y| + rms) of test_gpu_moe.py."""
import types

import pytest
import torch
import torch.nn.functional as F

from test_gpu_expert_launches import _kernels
from test_gpu_moe_calls import Linear
from test_gpu_stream import _bf16_default, _h_close, _weight  # noqa: F401

pytestmark = pytest.mark.gpu


def _host(dim, inter):
    import dsv3_b200
    model = types.SimpleNamespace(gemm_impl="fp8", block_size=128, world_size=1, dist=None)

    class MLP(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.w1, self.w2, self.w3 = Linear(inter, dim, 1, model), Linear(dim, inter, 2, model), Linear(inter, dim, 3, model)

        def forward(self, x):
            return self.w2(F.silu(self.w1(x)) * self.w3(x))

    model.MLP, model.Expert = MLP, type("Expert", (MLP,), {"forward": MLP.forward})
    dsv3_b200.install_linear(model)
    dsv3_b200.install_mlp(model)
    return MLP(), model


def _rows(M, K):
    return torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(M), device="cuda", dtype=torch.float32).bfloat16()


@pytest.mark.parametrize("dim,inter", [(2048, 1408), (1024, 2816), (7168, 2304), (512, 9600)])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 96, 129, 257, 700, 1025])
def test_three_launches_against_the_operators(M, dim, inter):
    import kernel
    from dsv3_b200 import _lib, swiglu_quant
    mlp, model = _host(dim, inter)
    x = _rows(M, dim)
    got = mlp(x)
    ws = [(lin.weight, lin.weight.scale) for lin in (mlp.w1, mlp.w3, mlp.w2)]
    q = kernel.act_quant(x)
    h = swiglu_quant(kernel.fp8_gemm(*q, *ws[0]), kernel.fp8_gemm(*q, *ws[1]))
    want = kernel.fp8_gemm(*h, *ws[2])
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    assert bool((err <= 2e-2 * (want.float().abs() + rms)).all())
    assert torch.equal(got, mlp(x)), "a fixed order"
    pays = _lib.lib.dsv3_swiglu_linear_pays(_i64(M), _i64(inter), _i64(dim))
    if M > 4:
        assert len(_kernels(lambda: mlp(x.view(x.shape)))) == (3 if pays else 5)


def _i64(v):
    import ctypes
    return ctypes.c_int64(v)


@pytest.mark.parametrize("M,N,K,fmt", [(5, 384, 1024, 0), (40, 1408, 2048, 1), (130, 256, 7168, 0), (200, 2816, 2048, 0), (300, 128, 128, 1), (1100, 2304, 512, 0)])
def test_codes_and_scales_in_front_of_w2(M, N, K, fmt):
    """Without a workspace no tile is cut: the codes and scales of the separate launches, bit for bit where their GEMMs cut nothing."""
    import ctypes
    import dsv3_b200
    import kernel
    from dsv3_b200 import _lib, swiglu_quant
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w1, w3 = _weight(N, K, g), _weight(N, K, g)
    xq, xs = kernel.act_quant(_rows(M, K))
    h, hs = torch.full((M + 1, N), 7, dtype=torch.uint8, device="cuda"), torch.full((M + 1, N // 128), -1.0, dtype=torch.float32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(_lib.lib.dsv3_swiglu_linear(p(xq), p(xs), p(w1), p(w1.scale), p(w3), p(w3.scale), _i64(M), _i64(N), _i64(K), fmt, p(h), p(hs), None,
                                           ctypes.c_size_t(0), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert bool((h[M] == 7).all()) and bool((hs[M] == -1).all()), "rows beyond the last are not written"
    for policy in (0, dsv3_b200.KERNEL_CUDA_CORE):
        dsv3_b200.set_gemm_policy(policy, 0)
        want, want_s = swiglu_quant(kernel.fp8_gemm(xq, xs, w1, w1.scale), kernel.fp8_gemm(xq, xs, w3, w3.scale), "ue8m0" if fmt else None)
        _h_close(h[:M].view(torch.float8_e4m3fn), hs[:M].t(), want, want_s)


@pytest.mark.parametrize("change,launches", [(None, 3), ("hook", 5), ("forward", 5), ("world", 5), ("format", 6), ("bias", 6)])
def test_what_keeps_the_separate_launches(change, launches):
    """Against the operators, each with the bias and the format of its Linear; five launches, one more where the activations are
    quantised twice or the bias is added."""
    import kernel
    from dsv3_b200 import swiglu_quant
    mlp, model = _host(1024, 512)
    x = _rows(20, 1024)
    seen = []
    if change == "hook":
        mlp.w1.register_forward_hook(lambda m, i, o: seen.append(1))
    elif change == "forward":
        inner = mlp.w3.forward
        mlp.w3.forward = lambda x: (seen.append(1), inner(x))[1]
    elif change == "world":
        model.world_size = 2
    elif change == "format":
        mlp.w3.scale_fmt = "ue8m0"
    elif change == "bias":
        mlp.w1.bias = torch.linspace(-2, 2, 512, device="cuda")
    got = mlp(x.view(x.shape))
    assert bool(seen) == (change in ("hook", "forward"))

    def up(lin):
        y = kernel.fp8_gemm(*kernel.act_quant(x, 128, lin.scale_fmt), lin.weight, lin.weight.scale)
        return y if lin.bias is None else y + lin.bias
    want = kernel.fp8_gemm(*swiglu_quant(up(mlp.w1), up(mlp.w3), mlp.w2.scale_fmt), mlp.w2.weight, mlp.w2.weight.scale)
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    assert bool((err <= 2e-2 * (want.float().abs() + rms)).all())
    assert change is None or torch.equal(got, want), "the same operators"
    assert len(_kernels(lambda: mlp(x.view(x.shape)))) == launches
