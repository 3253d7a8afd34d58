"""The decode-sized Linear with eight warps per CTA: without a cluster, with one, uneven K ranges and an edge of the last row tile."""
import pytest

from test_gpu_linear_small import _env, test_fused_linear_vs_oracle_and_two_step_form as _check  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,seed", [
    (1, 3072, 1536, 90),      # 12 chunks over eight warps
    (8, 2393, 1664, 91),      # 13 chunks, nine rows in the last tile
    (2, 2304, 7168, 92),      # clusters of two
    (5, 2272, 6272, 93),      # clusters of two, 49 chunks
])
def test_eight_warps(M, N, K, seed):
    _check(M, N, K, seed)
