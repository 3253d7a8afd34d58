"""Token-major tiles of 64 weight rows, whole and cut over a cluster, at the sizes where tiles, parts and rows end.

Reference: the 128-wide tiles with the same split pinned, which add the same parts in the same order: equal bit for bit; and the CUDA-core kernel
within the fp8_gemm bound."""
import pytest
import torch

from gpu_util import assert_gemm_close
from test_gemm_plan import Plan, _plan  # noqa: F401

pytestmark = pytest.mark.gpu


def _chosen(M, N, K):
    import ctypes
    from dsv3_b200 import _lib
    tc_plan = getattr(_lib.lib, "_ZN4dsv37tc_planElllii")
    tc_plan.argtypes, tc_plan.restype = [ctypes.c_int64] * 3 + [ctypes.c_int] * 2, Plan
    p = tc_plan(M, N, K, 0, 0)
    assert not p.swap and p.bn == 64, "the plan takes these tiles"
    return p.splits


# M, N and K at the ends of tiles and inside them; rows of the result that 16-byte stores cannot write; splits that do not divide the chunks;
# scales of a tile in the first and the second half of a weight block
@pytest.mark.parametrize("M,N,K", [(1003, 576, 7168), (1000, 576, 7152), (128, 1536, 7168), (257, 448, 7040), (70, 7168, 2304), (100, 7000, 2304), (529, 1584, 4224),
                                   (300, 1537, 7168), (65, 7004, 3072), (1000, 256, 7168), (650, 800, 896), (400, 260, 7168)])
def test_half_tiles(M, N, K):
    import dsv3_b200
    import kernel
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    torch.set_default_dtype(torch.bfloat16)
    try:
        splits, kc = _chosen(M, N, K), -(-K // 128)
        a, a_s = kernel.act_quant(torch.randn(M, kc * 128, generator=g, device="cuda", dtype=torch.float32).bfloat16())
        b, b_s = dsv3_b200.weight_quant((torch.randn(N, kc * 128, generator=g, device="cuda", dtype=torch.float32) * 0.02).bfloat16())
        a, b = a[:, :K].contiguous(), b[:, :K].contiguous()
        y = kernel.fp8_gemm(a, a_s, b, b_s)
        assert torch.equal(y, kernel.fp8_gemm(a, a_s, b, b_s))
        dsv3_b200.set_gemm_policy(2, splits)
        assert torch.equal(y, kernel.fp8_gemm(a, a_s, b, b_s))
        dsv3_b200.set_gemm_policy(1, 0)
        assert_gemm_close(y.cpu(), kernel.fp8_gemm(a, a_s, b, b_s).cpu())
    finally:
        dsv3_b200.set_gemm_policy(0, 0)
        torch.set_default_dtype(torch.float32)
        dsv3_b200.check_device_status()
