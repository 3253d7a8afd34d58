"""The automatic plan over the range where it chooses between token tiles, and plans that are refused."""
import ctypes

import pytest
import torch


class Plan(ctypes.Structure):
    """TcPlan of csrc/gemm_plan.cuh"""
    _fields_ = [("error", ctypes.c_int), ("swap", ctypes.c_bool), ("pair", ctypes.c_bool), ("wide", ctypes.c_bool), ("cluster", ctypes.c_bool),
                ("bn", ctypes.c_int), ("tiles_p", ctypes.c_int), ("tiles_q", ctypes.c_int), ("splits", ctypes.c_int), ("kc", ctypes.c_int)]


def _plan(M, N, K):
    from dsv3_b200 import _lib
    tc_plan = getattr(_lib.lib, "_ZN4dsv37tc_planElllii")
    tc_plan.argtypes, tc_plan.restype = [ctypes.c_int64] * 3 + [ctypes.c_int] * 2, Plan
    p = tc_plan(M, N, K, 0, 0)
    return (p.bn, p.tiles_p, p.tiles_q, p.splits) if p.swap else None


@pytest.mark.parametrize("M,N,K,plan", [
    (32, 7168, 2048, (32, 56, 1, 2)),       # one tile as wide as M, cut
    (33, 7168, 2048, (32, 56, 2, 1)),       # several, whole
    (64, 4096, 512, (16, 32, 4, 1)),
    (128, 3072, 1536, (32, 24, 4, 1)),
    (256, 1408, 2048, (32, 11, 8, 1)),
    (257, 1408, 2048, None),                # token-major tiles
    (33, 576, 7168, (32, 5, 2, 8)),         # several, cut over clusters
    (128, 512, 16384, (32, 4, 4, 8)),
    (200, 512, 49152, (64, 4, 4, 8)),       # 24 MB of weights
    (200, 512, 49168, None),
    (64, 16384, 1552, (64, 128, 1, 1)),     # beyond: one tile as wide as M
])
def test_narrow_token_tiles(M, N, K, plan):
    """Token tiles, weight tiles and splits at both sides of the lines; the workspace is a padded part of a tile for every split."""
    from dsv3_b200 import _lib
    assert _plan(M, N, K) == plan
    if plan:
        bn, p, q, splits = plan
        assert _lib.lib.dsv3_fp8_gemm_workspace_bytes(M, N, K) == (_lib.WORKSPACE_HEADER_BYTES + splits * p * q * 128 * bn * 4 if splits > 1 else 0)


@pytest.mark.parametrize("bn,splits,chunks,fits", [(64, 1, 73, False), (64, 2, 145, False), (32, 1, 145, False), (16, 1, 145, False),
                                                   (64, 1, 72, True), (64, 2, 144, True), (16, 1, 144, True)])
def test_a_plan_beyond_the_scale_table_is_not_launched(bn, splits, chunks, fits):
    """Refused on the host, before any CUDA call.  What fits is looked at by arguments alone: without tensors to map it fails after the check."""
    if torch.cuda.is_available():
        pytest.skip("on the host without a device only: nothing can be launched there")
    from dsv3_b200 import _lib
    launch = getattr(_lib.lib, "_ZN4dsv318launch_fp8_gemm_tcEPKvPKfS1_S3_lllPvS4_mRKNS_6TcPlanEP11CUstream_st")
    launch.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_int64] * 3 + [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.POINTER(Plan), ctypes.c_void_p]
    plan = Plan(0, True, False, False, splits > 1, bn, 1, 1, splits, chunks)
    rc = launch(None, None, None, None, bn, 128, 128 * chunks, None, None, 0, ctypes.byref(plan), None)
    assert rc != _lib.OK and (b"scale table" in _lib.lib.dsv3_last_error()) == (not fits)


@pytest.mark.parametrize("M,N,K,wide", [
    (1049, 4720, 5504, False),              # one round of 256 x 256 tiles and strips of 128, odd chunks
    (722, 9088, 3968, False),
    (923, 6464, 2944, False),               # a round and 40 % of one
    (684, 8016, 2688, False),
    (1845, 4736, 4096, True),               # rows 4 KB apart
    (4096, 7168, 16384, True),              # many rounds
    (2048, 7168, 7296, True),
])
def test_pair_tiles(M, N, K, wide):
    """256 x 256 or 256 x 128, where 148 SMs decide it (both sum in the same order: no result tells them apart)."""
    from dsv3_b200 import _lib
    tc_plan = getattr(_lib.lib, "_ZN4dsv37tc_planElllii")
    tc_plan.argtypes, tc_plan.restype = [ctypes.c_int64] * 3 + [ctypes.c_int] * 2, Plan
    p = tc_plan(M, N, K, 0, 0)
    assert p.pair and p.wide == wide and p.splits == 1
