"""Results of 128-token tiles: 32 rows at a time by a TMA store where all of them are the group's, row by row where they are not.

Reference: fp8_gemm per group with unsplit 128-token tiles, whose sums are in the same order: equal bit for bit; rows of nobody stay as they were."""
import ctypes

import pytest
import torch

from test_gpu_stream import _bf16_default, _table, _weight  # noqa: F401

pytestmark = pytest.mark.gpu


# ends of tiles and of 32 rows; columns that end inside a box and inside a block, a tile with one block, rows no store of 16 bytes can write
@pytest.mark.parametrize("N", [256, 200, 392, 201])
@pytest.mark.parametrize("counts", [[96, 97, 0, 95, 128], [127, 129, 65, 160]])
def test_only_the_groups_rows_are_written(counts, N):
    import dsv3_b200
    import kernel
    from dsv3_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(N)
    K, n, rows = 384, len(counts), sum(counts) + 40
    w = [_weight(N, K, g) for _ in counts]
    xq, xs = kernel.act_quant(torch.randn(rows, K, generator=g, device="cuda", dtype=torch.float32).bfloat16())
    xs_t = xs.t().contiguous()
    seg = torch.tensor([sum(counts[:i]) for i in range(n + 1)], dtype=torch.int32, device="cuda")
    out = torch.full((rows, N), 7.0, device="cuda")
    i64, p = ctypes.c_int64, lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(_lib.lib.dsv3_fp8_gemm_rows(p(_table(_lib.lib, _lib.check, w, N, K)), n, p(xq), p(xs_t), p(seg), i64(rows), i64(0), i64(N), i64(K), p(out),
                                           None, None, ctypes.c_size_t(0), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    dsv3_b200.set_gemm_policy(2 if sum(counts) > 40 * n else 3, 1)             # tiles of 128 tokens, or weight-major ones
    at = 0
    for c, e in zip(counts, w):
        if c:
            assert torch.equal(out[at:at + c], kernel.fp8_gemm(xq[at:at + c].contiguous(), xs[at:at + c].contiguous(), e, e.scale))
        at += c
    assert bool((out[at:] == 7.0).all())
