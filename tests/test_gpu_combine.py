"""The weighted sum over a token's experts at the edges of its two forms (few tokens; many wide ones), bit for bit against
`y[idx] += expert(x[idx]) * weights` in bf16: the product and every partial sum formed in fp32 and rounded (model.py:689, :693)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,topk,dim", [
    (1, 8, 8), (3, 1, 2056), (399, 6, 4104), (400, 6, 4104), (401, 8, 4096), (400, 7, 7168), (450, 13, 8200), (2, 300, 128),
])
@pytest.mark.parametrize("with_z", [False, True])
def test_combine_rounds_as_the_operators_do(T, topk, dim, with_z):
    from dsv3_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(T * dim + topk)
    rows = max(1, T * topk // 2)
    o = torch.randn(rows, dim, generator=g, device="cuda", dtype=torch.float32).mul_(4).bfloat16()
    o.view(-1)[:8] = torch.tensor([float("inf"), float("-inf"), float("nan"), 3e38, -3e38, 1e-39, -0.0, 2e-41], device="cuda").bfloat16()
    pos = torch.randint(-1, rows, (T, topk), generator=g, device="cuda", dtype=torch.int32)
    pos[torch.rand(T, topk, generator=g, device="cuda") < 0.5] = -1
    pos[0, 0] = 0
    w = (torch.rand(T, topk, generator=g, device="cuda", dtype=torch.float32) * 2).bfloat16()
    z = torch.randn(T, dim, generator=g, device="cuda", dtype=torch.float32).bfloat16() if with_z else None
    y = torch.full((T, dim), 7.0, device="cuda", dtype=torch.bfloat16)
    p, i64 = (lambda t: ctypes.c_void_p(t.data_ptr())), ctypes.c_int64
    _lib.check(_lib.lib.dsv3_moe_combine_add(p(o), p(pos), p(w), p(z) if with_z else None, i64(T), topk, i64(dim), p(y),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want = torch.zeros(T, dim, device="cuda", dtype=torch.float32)
    for j in range(topk):
        at = pos[:, j].long()
        term = (o[at.clamp(min=0)].float() * w[:, j:j + 1].float()).bfloat16().float()
        want = torch.where(at[:, None] >= 0, (want + term).bfloat16().float(), want)
    if with_z:
        want = want + z.float()
    want = want.bfloat16()
    assert bool(((y == want) | (y.isnan() & want.isnan())).all())
