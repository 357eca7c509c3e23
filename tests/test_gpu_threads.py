"""A launch that waits for room in the GPU's queue (about a thousand launches) does not hold the interpreter's lock: other
threads go on, and one of them may launch what the queue's head waits for."""
import threading
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["builtin", "program"])
def test_a_full_queue_does_not_stop_other_threads(what):
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    from polarai_framework_b200.program import DeviceExecutor, elementwise_chain_program
    d, out, ex = DeviceBuiltins(), torch.empty(64, device="cuda"), DeviceExecutor(elementwise_chain_program(64), "cuda:0")
    call = ex.run if what == "program" else lambda: d.ffill(1.0, out)
    for _ in range(5):
        call()
    torch.cuda.synchronize()
    longest = [0.0]

    def launch_many():
        for _ in range(1500):
            t = time.perf_counter()
            call()
            longest[0] = max(longest[0], time.perf_counter() - t)

    thread = threading.Thread(target=launch_many)
    torch.cuda._sleep(1_500_000_000)                        # 0.8 s of GPU time in front of them
    gap, last = 0.0, time.perf_counter()
    thread.start()
    while thread.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    thread.join()
    torch.cuda.synchronize()
    assert longest[0] > 0.4, "the queue did not fill up"
    assert gap < longest[0] / 2, (gap, longest[0])
