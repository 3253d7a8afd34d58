"""The SM budget while another thread sets it: what is planned from it is planned for one budget or the other."""
import ctypes
import subprocess
import threading
import time

import pytest
import torch


def _while_it_changes(look, seconds=1.0):
    """Results of `look`, called by two threads while a third sets a budget of 8 SMs and lifts it again."""
    from dsv3_b200 import _lib
    stop, seen = threading.Event(), [set(), set()]

    def change():
        while not stop.is_set():
            _lib.lib.dsv3_set_num_sms(8)
            _lib.lib.dsv3_set_num_sms(0)

    def collect(found):
        while not stop.is_set():
            found.add(look())

    threads = [threading.Thread(target=change)] + [threading.Thread(target=collect, args=(s,)) for s in seen]
    for t in threads:
        t.start()
    time.sleep(seconds)
    stop.set()
    for t in threads:
        t.join()
    _lib.lib.dsv3_set_num_sms(0)
    return seen[0] | seen[1]


def test_number_of_sms():
    from dsv3_b200 import _lib
    num_sms = _lib.lib._ZN4dsv37num_smsEv
    _lib.lib.dsv3_set_num_sms(0)
    assert _while_it_changes(num_sms) <= {8, num_sms()}


_POISONED = r"""
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <thread>
// Rounds after which a thread that planned while the budget changed plans otherwise than before.
extern "C" int poisoned(int (*set)(int), size_t (*plan)(int64_t, int64_t, int64_t), int64_t M, int64_t N, int64_t K, int rounds) {
    set(0);
    const size_t want = plan(M, N, K);
    int bad = 0;
    for (int r = 0; r < rounds; ++r) {
        std::atomic<bool> stop{false};
        std::thread t([&] { while (!stop.load()) { set(8); set(0); } });
        for (int i = 0; i < 200; ++i) plan(M, N, K);
        stop = true;
        t.join();
        bad += plan(M, N, K) != want;
    }
    return bad;
}
"""


@pytest.mark.parametrize("device", [pytest.param("cpu"), pytest.param("cuda", marks=pytest.mark.gpu)])
def test_a_plan_made_for_one_budget_is_not_kept_for_another(device, tmp_path):
    """(In C++: the lines of two Python threads do not meet often enough.)"""
    from dsv3_b200 import _lib
    if device == "cuda":
        torch.cuda.init()
    (tmp_path / "poisoned.cpp").write_text(_POISONED)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-pthread", "-o", tmp_path / "poisoned.so", tmp_path / "poisoned.cpp"], check=True)
    i64 = ctypes.c_int64
    ws = _lib.lib.dsv3_fp8_gemm_workspace_bytes
    _lib.lib.dsv3_set_num_sms(0)
    unlimited = ws(16, 2304, 7168)
    _lib.lib.dsv3_set_num_sms(8)
    assert ws(16, 2304, 7168) != unlimited, "a size whose plan depends on the budget"
    assert ctypes.CDLL(tmp_path / "poisoned.so").poisoned(_lib.lib.dsv3_set_num_sms, ws, i64(16), i64(2304), i64(7168), 20000) == 0
