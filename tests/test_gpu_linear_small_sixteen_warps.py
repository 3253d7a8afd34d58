"""The decode-sized Linear with sixteen warps, or eight, to a row tile and no cluster: both sides of the lines that the choice is drawn at
(row tiles against SMs, chunks of K), K that leaves warps without a chunk, rows that end inside a tile."""
import pytest

from test_gpu_linear_small import _env, test_fused_linear_vs_oracle_and_two_step_form as _check  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,seed", [
    (1, 1408, 2048, 94),      # a chunk to a warp
    (8, 2359, 1408, 95),      # 148 row tiles, the last of seven rows; 11 chunks
    (3, 2376, 1280, 96),      # 149 row tiles: eight warps; ten chunks
    (2, 576, 1152, 97),       # nine chunks: clusters as before
    (4, 1270, 3200, 98),      # 80 row tiles, 25 chunks
    (2, 1264, 3200, 99),      # 79: clusters
    (1, 4096, 512, 100),      # eight warps, four chunks
    (6, 2304, 7168, 101),     # 56 chunks
])
def test_warps_without_a_cluster(M, N, K, seed):
    _check(M, N, K, seed)
