"""Whole tiles of the ordinary weight (the shared experts) among the groups': every tile is worked on once, whatever the distance
between them comes to and however many CTAs there are, up to a layer with more than 512 tokens."""
import pytest
import torch

from test_gpu_expert_launches import _kernels
from test_gpu_moe_calls import _host
from test_gpu_stream import _bf16_default, test_expert_gemms_match_the_operators_per_group as _check_groups  # noqa: F401

pytestmark = pytest.mark.gpu


# CTAs; tiles of the groups and of the ordinary weight in the two launches
@pytest.mark.parametrize("counts,inter,dim,side_rows,ctas", [
    ([9] * 7, 384, 1024, 60, 8),                 # 21 + 2 and 28 + 8: distances 11 and, sharing a factor with 8, 4 -> 3
    ([9] * 7, 384, 1024, 60, 6),
    ([20, 1, 17], 128, 256, 90, 4),              # 3 + 3: distance 2 -> 1, the ordinary weight first
    ([5, 6], 128, 256, 200, 4),                  # more tiles of the ordinary weight: they come last
    ([70, 200, 3, 66], 384, 512, 140, 6),        # tiles of 128 tokens
    ([70, 200, 3, 66], 384, 512, 140, 0),        # the same, beside tiles of 64
])
def test_tiles_of_the_ordinary_weight_among_the_groups(counts, inter, dim, side_rows, ctas):
    import dsv3_b200
    dsv3_b200.set_num_sms(ctas)
    try:
        _check_groups(counts, inter, dim, side_rows, False)
    finally:
        dsv3_b200.set_num_sms(0)


@pytest.mark.parametrize("tokens,inline", [(100, True), (2048, True), (2049, False)])
def test_shared_experts_of_many_tokens(tokens, inline):
    """In the routed experts' four launches or in two of their own: their activations are quantised already."""
    import dsv3_b200
    moe, _ = _host()
    x = torch.randn(tokens, 256, generator=torch.Generator(device="cuda").manual_seed(tokens), device="cuda", dtype=torch.float32).bfloat16()
    launches = len(_kernels(lambda: dsv3_b200.grouped_moe_forward(moe, x)))
    routing = moe.gate(x)
    gate = len(_kernels(lambda: moe.gate(x)))
    assert launches - gate == (4 if inline else 6)
    moe.gate = lambda x: routing
    got = dsv3_b200.grouped_moe_forward(moe, x)
    want, _ = moe.reference_forward(x)
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    assert bool((err <= 2e-2 * (want.float().abs() + rms)).all())         # the bound of test_gpu_moe.py
