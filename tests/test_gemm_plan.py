"""Sizes that the automatic plan asks a workspace for, over the range where it chooses between token tiles: a plan of many small tiles
never asks for more than a ticket header and the padded parts of tiles that the machine holds at once."""
import ctypes

import pytest
import torch


def test_workspace_of_narrow_token_tiles():
    from dsv3_b200 import _lib
    ws = _lib.lib.dsv3_fp8_gemm_workspace_bytes
    for M in (33, 48, 64, 65, 100, 256):
        for N, K in ((576, 7168), (7168, 2048), (1408, 2048), (512, 16384), (4096, 512)):
            assert ws(M, N, K) <= _lib.WORKSPACE_HEADER_BYTES + 148 * 128 * 128 * 4
    assert ws(64, 4096, 512) == 0 and ws(128, 3072, 1536) == 0          # enough narrow tiles: none is split


class Plan(ctypes.Structure):
    """TcPlan of csrc/gemm_plan.cuh"""
    _fields_ = [("error", ctypes.c_int), ("swap", ctypes.c_bool), ("pair", ctypes.c_bool), ("wide", ctypes.c_bool), ("cluster", ctypes.c_bool),
                ("bn", ctypes.c_int), ("tiles_p", ctypes.c_int), ("tiles_q", ctypes.c_int), ("splits", ctypes.c_int), ("kc", ctypes.c_int)]


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
