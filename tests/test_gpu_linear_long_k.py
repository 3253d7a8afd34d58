"""The decode-sized Linear at a K whose activations fill its staging buffer: the layout with eight warps per CTA stages twice as much of
them as the one with four, which then takes the call."""
import numpy as np
import pytest
import torch

from gpu_util import assert_gemm_close, bf16_bits
from test_gpu_linear_small import DECODE, _env  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,sms", [
    (1, 4096, 24064, 0),      # the longest K that one CTA of eight warps stages
    (1, 4096, 24192, 0),
    (8, 2353, 24192, 0),
    (2, 4096, 32768, 0),
    (4, 2304, 49152, 0),      # clusters: of two with eight warps, of four with four
    (1, 512, 32768, 32),      # 16 MB of weights, an SM budget
])
def test_long_k(M, N, K, sms):
    import dsv3_b200
    import kernel
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    w = torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32).to(torch.float8_e4m3fn)
    s = torch.rand(-(-N // 128), K // 128, generator=g, device="cuda", dtype=torch.float32) + 0.5
    xq, xs = kernel.act_quant(x)
    dsv3_b200.set_gemm_policy(dsv3_b200.KERNEL_CUDA_CORE, 0)
    want = kernel.fp8_gemm(xq, xs, w, s)
    dsv3_b200.set_num_sms(sms)
    try:
        y = dsv3_b200.fp8_linear(x, w, s)
        dsv3_b200.set_gemm_policy(DECODE, 0)
        y2 = kernel.fp8_gemm(xq, xs, w, s)
    finally:
        dsv3_b200.set_num_sms(0)
    assert_gemm_close(y, want.cpu())
    assert np.array_equal(bf16_bits(y), bf16_bits(y2))
