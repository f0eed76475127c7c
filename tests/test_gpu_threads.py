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


def test_a_set_status_word_raises_at_the_next_call():
    """What a kernel whose bounded wait gave up leaves in the status word surfaces at the next call of any kind, before it
    launches anything, once."""
    q = torch.randn(1, 1, 64, 64, device=DEV).bfloat16()
    win = (1, 8, 8, 1, 1)
    o, lse = swa.swa_forward(q, q, q, None, *win, 1.0)
    word = swa.tiled_swa._status(torch.device(DEV))
    torch.cuda.synchronize()
    assert word.is_pinned() and int(word[0]) == 0
    for call in (lambda: swa.tiled_swa_fwd(q, q, q, *win), lambda: swa.swa_backward(q, q, q, o, lse, q, None, *win, 1.0),
                 lambda: swa.TiledSwa.apply(q, q, q, *win, 1.0), swa.check_status):
        word[1], word[2], word[3], word[0] = 17, 0, 2, 6
        before = swa._lib.launch_count()
        with pytest.raises(RuntimeError, match=r"bounded-wait timeout on device 0: status=\[6, 17, 0, 2\]"):
            call()
        assert swa._lib.launch_count() == before and int(word[0]) == 0
    swa.check_status()
    assert torch.equal(swa.tiled_swa_fwd(q, q, q, *win), o)


def _step(q, k, v, do, rope, win):
    t = [x.detach().requires_grad_(True) for x in (q, k, v)]
    o = swa.TiledSwaRope2D.apply(*t, *rope, *win)
    return (o.detach(), *torch.autograd.grad(o, t, do))


def _case(th, tw, w, d, dtype, BH, seed=0):
    q, k, v, do = (t.to(DEV) for t in orc.seeded_inputs(1, BH, th * tw, d, d, dtype, seed))
    rope = tuple(t.to(DEV) for t in (orc.encode_idx(th, tw), orc.make_cs_table(8, th), orc.make_cs_table(8, tw)))
    return q, k, v, do, rope, (1, th, tw, w, w, d ** -0.5)


def test_two_threads_on_two_streams():
    """Plans kept per thread, kernel attributes set once, the pinned status word: threads with streams of their own, whose
    geometries meet for the first time and take turns, get what one thread alone gets."""
    cases = [_case(th, tw, w, d, dt, BH, i) for i, (th, tw, w, d, dt, BH) in enumerate(
        [(17, 19, 2, 64, torch.bfloat16, 3), (23, 9, 3, 80, torch.float16, 2), (11, 13, 2, 32, torch.float32, 4), (31, 8, 1, 128, torch.bfloat16, 5)])]
    swa._lib.lib.swa_refresh_env()                           # no plans yet
    torch.cuda.synchronize()
    results, errors = [[], []], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for r in range(12):
                    for j in range(len(cases)):
                        c = (j * (2 * i + 1) + r) % len(cases)
                        results[i].append((c, _step(*cases[c])))
                torch.cuda.current_stream().synchronize()
        except Exception as e:                               # noqa: BLE001 (shown by the assertion below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    torch.cuda.synchronize()
    swa.check_status()
    want = [_step(*c) for c in cases]
    for per_thread in results:
        assert len(per_thread) == 48
        for c, got in per_thread:
            assert all(torch.equal(a, b) for a, b in zip(got, want[c]))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("graph", [False, True])
def test_early_started_kernels_between_foreign_ones(dtype, graph):
    """On a stream of the caller's: a matrix product writes the inputs right before the call, and they are overwritten right
    after it.  The library's kernels start early but must neither read before the one nor after the other; the same when the
    sequence is captured and replayed."""
    q, k, v, do, rope, win = _case(24, 24, 3, 64, dtype, 8)
    srcs = [(_case(24, 24, 3, 64, dtype, 8, s)) for s in range(4)]
    eye = torch.eye(64, device=DEV, dtype=dtype)
    want = [_step(s[0], s[1], s[2], s[3], rope, win) for s in srcs]
    torch.cuda.synchronize()
    staged = [x.clone() for x in srcs[0][:4]]

    def sequence():
        for dst, src in zip((q, k, v, do), staged):
            torch.matmul(src, eye, out=dst)                  # (a product with the unit matrix: the same values)
        got = _step(q, k, v, do, rope, win)
        for dst in (q, k, v, do):
            dst.fill_(float("nan"))
        return got

    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            sequence()
            if graph:
                g = torch.cuda.CUDAGraph()
                torch.cuda.current_stream().synchronize()
                with torch.cuda.graph(g, stream=torch.cuda.current_stream()):
                    outs = sequence()
            for _ in range(5):
                got = []
                for s in srcs:
                    for dst, src in zip(staged, s[:4]):
                        dst.copy_(src)
                    if graph:
                        g.replay()
                    got.append([t.clone() for t in (outs if graph else sequence())])
                torch.cuda.current_stream().synchronize()
                for a, b in zip(got, want):
                    assert all(torch.equal(x, y) for x, y in zip(a, b))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = prev
    swa.check_status()
