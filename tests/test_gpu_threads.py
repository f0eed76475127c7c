"""The call surface beside other threads and other streams."""
import threading
import time

import pytest
import torch

from oracle import swa_oracle as orc

import dl_templates_b200 as swa

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_other_threads_run_while_a_launch_waits_for_room_in_the_queue():
    """A stream takes about a thousand launches ahead; the next one waits.  Behind a kernel that runs for about a second, calls
    that fill the queue block, and a Python thread beside them goes on."""
    q = torch.randn(1, 1, 64, 64, device=DEV).bfloat16()
    call = lambda: swa.tiled_swa_fwd(q, q, q, 1, 8, 8, 1, 1)
    call()
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def beside():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.002)

    th = threading.Thread(target=beside)
    th.start()
    try:
        t0 = time.perf_counter()
        torch.cuda._sleep(2_000_000_000)                 # about a second of GPU clocks
        for _ in range(4000):
            call()
        blocked = time.perf_counter() - t0
        torch.cuda.synchronize()
    finally:
        stop.set()
        th.join()
    assert blocked > 0.5, "the queue never filled: this run says nothing"
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < 0.25


def test_debug_sync_is_looked_up_on_every_call(monkeypatch):
    """SWA_DEBUG_SYNC set after the first calls of a process makes a call wait for its kernels, and unset it no longer does."""
    q = torch.randn(1, 1, 64, 64, device=DEV).bfloat16()
    for value, waits in ((None, False), ("1", True), (None, False), ("", False)):
        monkeypatch.delenv("SWA_DEBUG_SYNC", raising=False)
        if value is not None:
            monkeypatch.setenv("SWA_DEBUG_SYNC", value)
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)                   # about a tenth of a second
        swa.tiled_swa_fwd(q, q, q, 1, 8, 8, 1, 1)
        assert torch.cuda.current_stream().query() == waits
