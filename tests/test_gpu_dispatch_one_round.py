"""The expert layer's dispatch where its CTAs have one round of blocks, whose values are read before the pairs are counted, at both sides of that
line and with CTAs along a token's row that have fewer blocks than the others."""
import pytest

from test_gpu_dispatch_blocks import test_rows_and_their_copies as _check

pytestmark = pytest.mark.gpu


# blocks of a token's row: 65 and 97 shared by two CTAs (33 and 32, 49 and 48), 64 and 65 of one CTA, one; two tokens to a CTA
@pytest.mark.parametrize("T,topk,dim,n", [(1, 8, 8320, 32), (37, 2, 12416, 16), (100, 6, 8192, 64), (100, 6, 8320, 64), (3, 32, 128, 256), (148, 1, 128, 1), (200, 4, 4096, 8)])
def test_rows_and_their_copies_in_one_round(T, topk, dim, n):
    _check(T, topk, dim, n, 0)
