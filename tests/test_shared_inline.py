"""Which launches the shared experts are worked on in, at both sides of each line of the rule (moe_seam._shared_inline)."""
from types import SimpleNamespace

import pytest

import dsv3_b200.moe_seam as seam


@pytest.mark.parametrize("local, inter, dim, routed, topk, width, rows, inline", [
    (20, 1536, 5120, 160, 6, 3072, 256, True),           # weights read again less than the local experts' own
    (20, 1536, 5120, 160, 6, 3072, 333, False),
    (20, 1536, 5120, 160, 6, 3072, 512, False),
    (20, 1536, 5120, 160, 6, 3072, 1066, False),         # 40 pairs an expert: 64-token tiles
    (20, 1536, 5120, 160, 6, 3072, 1067, True),          # and 128 above
    (20, 1536, 5120, 160, 6, 3072, 2049, False),
    (32, 2048, 7168, 256, 8, 2048, 512, True),
    (32, 2048, 7168, 256, 8, 2048, 513, False),
    (16, 1408, 2048, 64, 6, 2816, 426, True),            # small weights: up to the floor
    (8, 2048, 7168, 256, 8, 2048, 304, True),
    (8, 2048, 7168, 256, 8, 2048, 306, False),
    (160, 1536, 5120, 160, 6, 3072, 512, True),
    (160, 1536, 5120, 160, 6, 3072, 1500, False),        # too much to read for the larger sizes
    (64, 1408, 2048, 64, 6, 2816, 2048, True),
])
def test_where_shared_experts_run(local, inter, dim, routed, topk, width, rows, inline):
    st = SimpleNamespace(n=local, inter=inter, dim=dim)
    assert bool(seam._shared_inline(st, rows, topk, routed, width)) is inline


@pytest.mark.parametrize("rows, routed, topk, width, inline", [
    (128, 256, 8, 2432, True),             # four pairs an expert: tiles of 16 tokens, eight reads of 3 x 2432 x 7168 bytes
    (128, 256, 8, 2560, False),
    (129, 256, 8, 4736, True),             # five: tiles of 32
    (129, 256, 8, 4864, False),
    (192, 64, 8, 3200, True),              # 24
    (192, 64, 8, 3328, False),
    (200, 64, 8, 6144, True),              # 25: tiles of 64
    (200, 64, 8, 6400, False),
    (40, 256, 8, 7680, True),              # few rows, large weights
    (40, 256, 8, 7808, False),
])
def test_reads_of_the_shared_weights_follow_the_tiles(rows, routed, topk, width, inline):
    st = SimpleNamespace(n=8, inter=1024, dim=7168)
    assert bool(seam._shared_inline(st, rows, topk, routed, width)) is inline


def test_few_rows_without_the_rule_are_below_its_floor():
    assert -(-seam.SHARED_INLINE_FEW_ROWS // 16) * 3 * seam.SHARED_INLINE_FEW_ROWS_MAX_WEIGHT <= seam.SHARED_INLINE_REREAD_FLOOR
