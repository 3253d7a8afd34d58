"""The 256-wide pair kernel's last round in strips of 64 and 128 columns, alone and behind whole rounds: bit-equal to the 256 x 128
kernel, which cuts nothing, on a machine of a few pairs (an SM budget)."""
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

NARROW, WIDE = 4, 6      # kernel policies


@pytest.fixture(autouse=True)
def _env():
    import dsv3_b200
    torch.set_default_dtype(torch.bfloat16)
    yield
    torch.set_default_dtype(torch.float32)
    dsv3_b200.set_gemm_policy(0, 0)
    dsv3_b200.set_num_sms(0)
    dsv3_b200.check_device_status()


# M, N -> tiles of 256 x 256; pairs
@pytest.mark.parametrize("M,N,K,pairs", [
    (300, 256, 512, 8),       # two tiles, eight strips of 64; the second token tile pair holds 44 rows
    (256, 600, 3200, 6),      # three tiles, strips of 128, the last tile 88 columns wide: a strip beyond N, one cut short
    (500, 900, 640, 7),       # eight tiles: a whole round and one tile in strips of 64, K chunks not a multiple of four
    (700, 1300, 2048, 7),     # 18 tiles: two rounds and four (no strips)
    (700, 1300, 2048, 8),     # two rounds and two tiles in strips of 64
    (700, 1301, 3280, 12),    # a round and six tiles in strips of 128; N odd, a K tail
    (700, 1301, 400, 12),     # the same, K too short for strips of 128
    (260, 330, 208, 36),      # four tiles, strips of 64, K tail
    (260, 200, 128, 74),      # two tiles, one chunk
])
def test_strips_equal_the_narrow_kernel(M, N, K, pairs):
    import dsv3_b200
    import kernel
    g = torch.Generator(device="cuda").manual_seed(M + N)
    kp = -(-K // 128) * 128
    x = torch.randn(M, kp, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    x[:, K:] = 0
    xq, xs = kernel.act_quant(x)
    xq = xq.view(torch.uint8)[:, :K].contiguous().view(torch.float8_e4m3fn)
    w, ws = dsv3_b200.weight_quant((torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32) * 0.02).bfloat16())
    dsv3_b200.set_num_sms(2 * pairs)
    dsv3_b200.set_gemm_policy(WIDE, 0)
    y = kernel.fp8_gemm(xq, xs, w, ws)
    dsv3_b200.set_gemm_policy(NARROW, 0)
    want = kernel.fp8_gemm(xq, xs, w, ws)
    dsv3_b200.check_device_status()
    assert torch.equal(y, want)
    rows = torch.arange(0, M, max(1, M // 5))
    ok, ratio = O.gemm_tolerance_ok(y[rows.cuda()].cpu(), O.fp8_gemm(xq[rows.cuda()].cpu(), xs[rows.cuda()].cpu(), w.cpu(), ws.cpu()), 1e-2)
    assert ok, ratio
