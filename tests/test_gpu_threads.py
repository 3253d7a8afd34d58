"""The host extension under several threads: calls release the GIL while they launch."""
import threading

import pytest
import torch

from test_gpu_capture import _cut_experts, _split_linear
from test_gpu_stream import _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [_split_linear, _cut_experts])
def test_workspace_that_another_thread_drops(make):
    """One thread repeats calls that use a workspace and fills freed memory behind them; the other passes through more
    streams than workspaces are kept for, so that the first one's is dropped again and again."""
    call = make()
    want = call()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(24)]
    mine, stop, wrong = torch.cuda.Stream(), threading.Event(), []

    def others():
        torch.set_default_dtype(torch.bfloat16)
        while not stop.is_set():
            for s in streams:
                with torch.cuda.stream(s):
                    call()

    t = threading.Thread(target=others)
    t.start()
    try:
        with torch.cuda.stream(mine):
            for _ in range(300):
                y = call()
                torch.full((16 << 20,), 7, dtype=torch.uint8, device="cuda")
                wrong.append((y != want).any())
            mine.synchronize()
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    assert not bool(torch.stack(wrong).any())


def test_after_a_wait_gave_up_workspaces_of_streams_that_are_gone_do_not_matter():
    """check_device_status makes the next calls start with clear tickets, whatever has become of the streams so far."""
    import ctypes
    import dsv3_b200
    from dsv3_b200 import _lib
    call = _split_linear()
    want = call()
    rt, handle = torch.cuda.cudart(), ctypes.c_void_p()
    assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
    with torch.cuda.stream(torch.cuda.ExternalStream(handle.value)):
        assert torch.equal(call(), want)
        torch.cuda.current_stream().synchronize()
    assert int(rt.cudaStreamDestroy(handle.value)) == 0
    _lib.check(_lib.lib.dsv3_selftest_bounded_wait(2_000_000, torch.cuda.current_stream().cuda_stream))
    with pytest.raises(_lib.Dsv3Error):
        dsv3_b200.check_device_status()
    assert torch.equal(call(), want)
