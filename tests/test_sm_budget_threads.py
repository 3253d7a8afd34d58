"""The SM budget while another thread sets it: what is planned from it is planned for one budget or the other."""
import threading
import time


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
