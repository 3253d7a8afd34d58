"""The 256-wide pair kernel's scale loads: four, two or one K chunk at a time, by the number of chunks and the scales' alignment.

Reference: the 256 x 128 pair kernel, whose sums are in the same order: equal bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# chunks a multiple of four, of two, odd, one; scales on 16, 8 and 4 bytes
@pytest.mark.parametrize("kc", [1, 2, 6, 7, 8, 18])
@pytest.mark.parametrize("offset", [0, 2, 1])
def test_equal_whatever_the_loads(kc, offset):
    import dsv3_b200
    import kernel
    M, N, K = 300, 392, 128 * kc
    g = torch.Generator(device="cuda").manual_seed(kc)
    torch.set_default_dtype(torch.bfloat16)
    try:
        a, a_s = kernel.act_quant(torch.randn(M, K, generator=g, device="cuda", dtype=torch.float32).bfloat16())
        b, b_s = dsv3_b200.weight_quant((torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32) * 0.02).bfloat16())
        moved = []
        for s in (a_s, b_s):
            buf = torch.empty(s.numel() + 4, dtype=torch.float32, device="cuda")
            moved.append(buf[offset:offset + s.numel()].view(s.shape).copy_(s))
        out = []
        for policy in (4, 6):
            dsv3_b200.set_gemm_policy(policy, 0)
            out.append(kernel.fp8_gemm(a, moved[0], b, moved[1]))
        assert torch.equal(*out)
    finally:
        dsv3_b200.set_gemm_policy(0, 0)
        torch.set_default_dtype(torch.float32)
        dsv3_b200.check_device_status()


# every remainder of four, every place of a row in the groups of four (rows begin at offset + row * kc), the first and the last row of the scales in
# groups that lie partly outside of them
@pytest.mark.parametrize("kc", [17, 19, 20, 21, 22, 25])
@pytest.mark.parametrize("offset", [1, 2, 3])
@pytest.mark.parametrize("M", [129, 256])
def test_rows_between_the_groups_of_four(kc, offset, M):
    import dsv3_b200
    import kernel
    N, K = 264, 128 * kc
    g = torch.Generator(device="cuda").manual_seed(kc)
    torch.set_default_dtype(torch.bfloat16)
    try:
        a = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float32).to(torch.float8_e4m3fn)
        b = torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32).to(torch.float8_e4m3fn)
        # (NaN around the scales: a scale from beside them would show)
        moved = []
        for rows in (M, -(-N // 128)):
            buf = torch.full((rows * kc + 8,), float("nan"), dtype=torch.float32, device="cuda")
            moved.append(buf[offset:offset + rows * kc].view(rows, kc).copy_(torch.rand(rows, kc, generator=g, device="cuda", dtype=torch.float32) + 0.5))
        out = []
        for policy in (4, 6):
            dsv3_b200.set_gemm_policy(policy, 0)
            out.append(kernel.fp8_gemm(a, moved[0], b, moved[1]))
        assert torch.equal(*out) and bool(out[0].isfinite().all())
    finally:
        dsv3_b200.set_gemm_policy(0, 0)
        torch.set_default_dtype(torch.float32)
        dsv3_b200.check_device_status()
