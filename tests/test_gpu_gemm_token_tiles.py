"""33 to 256 tokens on few weights, where the automatic plan takes several token tiles of 16, 32 or 64 with the weights on the M side, whole
or split inside clusters (test_gemm_plan.py holds which), and sizes beside that range: edges of the token tiles and of the range, weight tiles cut by N, K tails, a K longer than a tile's scale
table, against the CUDA-core kernel."""
import pytest
import torch

from gpu_util import assert_gemm_close
from test_gpu_stream import _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [17, 31, 33, 64, 65, 96, 129, 193, 256, 257])
@pytest.mark.parametrize("N,K", [(576, 7168), (1, 8192), (250, 4096 + 48), (1101, 5120), (7168, 2048), (4096, 512), (2000, 656), (70, 131072), (300, 24576)])
def test_token_tiles_against_the_cuda_core_kernel(M, N, K):
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
    assert_gemm_close(y.cpu(), kernel.fp8_gemm(a, a_s, b, b_s).cpu())            # the fp8_gemm bound, 1e-2 (|y| + rms)
