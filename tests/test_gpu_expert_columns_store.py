"""Results of 64-token tiles, four columns of a token to a store where rows are 16-byte aligned.

Reference: fp8_gemm per group with unsplit weight-major tiles, whose sums are in the same order: equal bit for bit; rows of nobody stay as they were."""
import pytest

from test_gpu_expert_rows_store import test_only_the_groups_rows_are_written as _written
from test_gpu_stream import _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


# tokens that end inside a quad, a piece and a group's half; columns that end inside a warp, a block and a tile, unaligned rows
@pytest.mark.parametrize("N", [256, 200, 392, 264, 201])
@pytest.mark.parametrize("counts", [[64, 1, 0, 62, 33], [30, 31, 65, 16, 17], [5, 50, 47, 18]])
def test_only_the_groups_rows_are_written(counts, N):
    _written(counts, N)
