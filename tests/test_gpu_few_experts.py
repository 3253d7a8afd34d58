"""The expert layer for a handful of tokens in two launches (csrc/moe_few.cu) against the operators, pair by pair."""
import pytest
import torch

from test_gpu_moe import _MoE, _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


def _pairs_one_by_one(moe, x, weights, indices):
    y = torch.zeros_like(x)
    for t in range(x.size(0)):
        order = sorted(range(indices.size(1)), key=lambda j: (int(indices[t, j]), j))       # ascending experts, model.py:683
        for j in order:
            e = int(indices[t, j])
            if moe.experts_start_idx <= e < moe.experts_end_idx:
                y[t] += (moe.experts[e](x[t:t + 1]) * weights[t, j].to(torch.bfloat16))[0]
    return y


# K chunks: fewer than the warps, not a multiple of warps or ring, more than both; experts: one, some, none of them local;
# rows of a slot: 1 .. 8, two slots where an expert is listed more often than there are tokens
@pytest.mark.parametrize("T,dim,inter,E,topk,start,end,fmt,shared,indices", [
    (1, 128, 128, 64, 8, 0, 16, None, "inline", None),
    (1, 640, 384, 64, 8, 8, 24, "ue8m0", "inline", [[8, 9, 20, 23, 0, 1, 40, 41]]),
    (1, 7168, 256, 32, 4, 0, 8, None, "inline", [[7, 0, 3, 1]]),
    (2, 1152, 2176, 16, 2, 4, 6, None, "z", [[5, 4], [4, 5]]),
    (3, 256, 128, 16, 2, 0, 4, None, "inline", [[9, 10], [11, 12], [13, 14]]),              # none local
    (8, 2048, 1408, 64, 4, 0, 4, None, "inline", [[0, 1, 2, 3]] * 8),
    (8, 512, 128, 64, 8, 3, 5, "ue8m0", "none", [[3, 4, 5, 6, 7, 8, 9, 10]] * 8),
    (1, 256, 256, 16, 4, 0, 8, None, "inline", [[2, 2, 5, 2]]),
])
def test_two_launches_match_the_operators(T, dim, inter, E, topk, start, end, fmt, shared, indices):
    import dsv3_b200
    from dsv3_b200 import _lib
    from dsv3_b200.moe_seam import GroupedExperts
    assert _lib.lib.dsv3_few_experts_pay(T, topk, end - start, E, dim, inter, inter if shared == "inline" else 0) == 1
    moe = _MoE(dim, inter, E, topk, start, end, seed=3 * T + dim)
    for e in [moe.shared] + moe.experts[start:end]:
        for lin in (e.w1, e.w2, e.w3):
            lin.scale_fmt = fmt
    g = torch.Generator(device="cuda").manual_seed(dim + inter)
    x = torch.randn(T, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    weights = torch.rand(T, topk, generator=g, device="cuda", dtype=torch.float32)
    if T % 2 == 0:
        weights = weights.bfloat16()
    indices = torch.tensor(indices, device="cuda") if indices else torch.randint(0, E, (T, topk), generator=g, device="cuda")
    if fmt is not None:                     # the operators of _MoE quantise with fp32 scales
        import kernel
        import test_gpu_moe
        quantise = lambda self, v: kernel.fp8_gemm(*kernel.act_quant(v, 128, self.scale_fmt), self.weight, self.weight.scale)  # noqa: E731
        original, test_gpu_moe._Lin.__call__ = test_gpu_moe._Lin.__call__, quantise
    try:
        want = _pairs_one_by_one(moe, x, weights, indices)
        z = moe.shared_experts(x)
    finally:
        if fmt is not None:
            test_gpu_moe._Lin.__call__ = original
    experts = GroupedExperts(moe.experts, moe.experts[start:end], start)
    inline = (moe.shared.w1.weight, moe.shared.w3.weight, moe.shared.w2.weight) if shared == "inline" else None
    routed = experts.run(x, weights, indices, E, inline)
    got = _lib.host.combine(routed, z if shared == "z" else None)
    again = _lib.host.combine(routed, z if shared == "z" else None)
    dsv3_b200.check_device_status()
    if shared != "none":
        want = want + z
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    assert bool((err <= 2e-2 * (want.float().abs() + rms)).all()), float((err / (want.float().abs() + rms)).max())   # the bound of test_gpu_moe.py
    assert torch.equal(got, again)


def test_the_sizes_that_two_launches_take():
    from dsv3_b200 import _lib
    pay = _lib.lib.dsv3_few_experts_pay
    assert pay(1, 8, 32, 256, 7168, 2048, 256) == 1
    assert pay(9, 1, 4, 256, 512, 256, 0) == 0 and pay(8, 9, 1, 256, 512, 256, 0) == 0          # tokens, pairs
    assert pay(1, 8, 32, 256, 7168 + 64, 2048, 0) == 0 and pay(1, 8, 32, 256, 7168, 2048, 64) == 0
    assert pay(3, 8, 32, 256, 7168, 2048, 0) == 0 and pay(1, 8, 32, 0, 7168, 2048, 0) == 0      # more than two local pairs expected
