"""Sizes that the automatic plan asks a workspace for, over the range where it chooses between token tiles: a plan of many small tiles
never asks for more than a ticket header and the padded parts of tiles that the machine holds at once."""


def test_workspace_of_narrow_token_tiles():
    from dsv3_b200 import _lib
    ws = _lib.lib.dsv3_fp8_gemm_workspace_bytes
    for M in (33, 48, 64, 65, 100, 256):
        for N, K in ((576, 7168), (7168, 2048), (1408, 2048), (512, 16384), (4096, 512)):
            assert ws(M, N, K) <= _lib.WORKSPACE_HEADER_BYTES + 148 * 128 * 128 * 4
    assert ws(64, 4096, 512) == 0 and ws(128, 3072, 1536) == 0          # enough narrow tiles: none is split
