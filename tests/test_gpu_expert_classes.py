"""Expert GEMMs whose groups are divided between two kinds of tiles (more than 64 rows, and the others): either class empty, both, and
the edge between them, with a side problem among the first CTAs'."""
import pytest

from test_gpu_stream import _bf16_default, test_expert_gemms_match_the_operators_per_group as _check_groups  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,inter,dim,side_rows", [
    ([64, 63, 64, 62], 128, 384, 3),          # no large group
    ([66, 200, 65], 256, 256, 1),             # no small one
    ([64, 65, 0, 300, 1, 16, 129, 17], 384, 640, 200),
])
def test_groups_divided_by_their_rows(counts, inter, dim, side_rows):
    _check_groups(counts, inter, dim, side_rows, True)
