"""Where w1 and w3 of an MLP share a launch, at both sides of the lines: on the device, and for a host that launches."""
import ctypes

import pytest


def _rules(M, N, K):
    from dsv3_b200 import _lib
    return tuple(bool(f(*map(ctypes.c_int64, (M, N, K)))) for f in (_lib.lib.dsv3_swiglu_linear_pays, _lib.lib.dsv3_swiglu_linear_saves_launches))


@pytest.mark.parametrize("M,N,K,device,host", [
    (1, 1408, 2048, False, True),             # the decode kernel twice, but for few K chunks
    (8, 1408, 2048, False, True),
    (8, 2816, 1024, True, True),
    (2, 1536, 7168, True, True),              # beyond its weights: one or two rows have the fused Linear
    (3, 1536, 7168, False, True),
    (9, 1408, 2048, True, True),
    (16, 1920, 3200, False, True),
    (16, 2048, 3200, True, True),
    (16, 4608, 7168, True, False),
    (17, 4608, 7168, False, False),           # enough weights for the device to be the bound
    (17, 3072, 7168, False, True),
    (32, 2048, 5120, True, True),
    (33, 2304, 7168, True, True),
    (64, 768, 7168, False, True),
    (65, 768, 7168, True, True),
    (1, 18432, 7168, True, False),
    (129, 18432, 7168, False, False),         # no tile
    (2048, 1408, 2048, False, False),
    (16, 1400, 2048, False, False),           # sizes that it does not take
    (0, 1408, 2048, False, False),
])
def test_lines_of_the_rules(M, N, K, device, host):
    assert _rules(M, N, K) == (device, host)


@pytest.mark.parametrize("kernel,split", [(2, 0), (0, 4)])
def test_a_pinned_gemm_keeps_the_separate_launches(kernel, split):
    import dsv3_b200
    assert _rules(64, 1408, 2048) == (True, True)
    dsv3_b200.set_gemm_policy(kernel, split)
    try:
        assert _rules(64, 1408, 2048) == (False, False)
    finally:
        dsv3_b200.set_gemm_policy(0, 0)
