"""Expert GEMMs with cut tiles while another thread sets the SM budget: the partial tiles fit the workspace that was checked."""
import threading

import pytest
import torch

from test_gpu_capture import _cut_experts
from test_gpu_stream import _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


def test_cut_tiles_while_the_budget_changes():
    import dsv3_b200
    from dsv3_b200 import _lib
    call = _cut_experts()
    want = call().float()
    stop, worst = threading.Event(), []

    def change():
        while not stop.is_set():
            _lib.lib.dsv3_set_num_sms(8)
            _lib.lib.dsv3_set_num_sms(0)

    t = threading.Thread(target=change)
    t.start()
    try:
        bound = 2e-2 * (want.abs() + want.pow(2).mean().sqrt())           # that of test_gpu_moe.py: sums in another order
        for _ in range(300):
            worst.append(((call().float() - want).abs() / bound).max())
    finally:
        stop.set()
        t.join()
        dsv3_b200.set_num_sms(0)
    assert float(torch.stack(worst).max()) <= 1.0
    dsv3_b200.check_device_status()
