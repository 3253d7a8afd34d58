"""Which layout the decode-sized Linear takes at both sides of the lines, read from a captured graph: a CTA of sixteen or eight warps to
a row tile, or four-warp CTAs in clusters."""
import pytest
import torch

from test_gpu_expert_launches import _kernels
from test_gpu_stream import _bf16_default, _weight  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,ctas,warps", [
    (1408, 2048, 88, 16),
    (1280, 3072, 80, 16),           # 24 chunks: any number of row tiles
    (1280, 3200, 80, 16),           # 25 chunks, 80 row tiles
    (1264, 3200, 316, 4),           # 79: clusters of four
    (1536, 7168, 96, 16),
    (576, 7168, 288, 4),            # clusters of eight
    (2376, 1280, 149, 8),
])
def test_layout(N, K, ctas, warps):
    import dsv3_b200
    g = torch.Generator(device="cuda").manual_seed(N)
    w, x = _weight(N, K, g), torch.randn(1, K, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    assert _kernels(lambda: dsv3_b200.fp8_linear(x, w, w.scale)) == [(ctas, 32 * warps)]
