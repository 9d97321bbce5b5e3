"""The copy of a large drain when something fails in it: a thread that cannot start is
done without, anything else stops the drain and reaches the caller, and no thread
still writes to bytes that are gone."""
import ctypes
import threading
import time
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest


def _sink(monkeypatch, pool):
    import tuna_gb300 as T
    monkeypatch.setattr(T, "ThreadPoolExecutor", pool)
    ctx = T.Context.__new__(T.Context)
    ctx._pool, ctx.h = None, None
    return ctx, T._DrainSink(ctx)


def _hand_over(sink, src):
    import tuna_gb300 as T
    return T._SINK(sink)(src.ctypes.data, src.size, 1, None)  # as tg_job_drain calls it


@pytest.mark.parametrize("started", [0, 1, 3])
def test_no_thread(monkeypatch, started):
    class Pool(ThreadPoolExecutor):
        left = started

        def submit(self, *a, **kw):
            f = super().submit(*a, **kw)
            if Pool.left == 0:
                raise RuntimeError("can't start new thread")
            Pool.left -= 1
            return f

    ctx, sink = _sink(monkeypatch, Pool)
    src = np.random.default_rng(started).integers(0, 256, (5 << 20) + 7, dtype=np.uint8)
    for _ in range(2):
        assert _hand_over(sink, src) == 0
        assert ctx._pool is None
    assert sink.result() == 2 * src.tobytes()


def test_error_reaches_the_caller(monkeypatch):
    class Pool(ThreadPoolExecutor):
        def __init__(self, *a):
            raise MemoryError

    ctx, sink = _sink(monkeypatch, Pool)
    src = np.zeros(5 << 20, dtype=np.uint8)
    assert _hand_over(sink, src) == 1
    with pytest.raises(MemoryError):
        sink.result()
    assert _hand_over(sink, src[:100]) == 0  # a small one takes no threads


def test_no_write_after_an_error(monkeypatch):
    """The pieces in flight have ended when the copy gives up."""
    import tuna_gb300 as T
    ended = []

    def slow(dst, src, n):
        if threading.current_thread() is not threading.main_thread():
            time.sleep(0.05)
            ended.append(n)
        return dst

    class Pool(ThreadPoolExecutor):
        def submit(self, *a, **kw):
            if self._work_queue.qsize() or len(self._threads) >= 2:
                raise KeyboardInterrupt
            return super().submit(*a, **kw)

    monkeypatch.setattr(T.ctypes, "memmove", slow)
    ctx, sink = _sink(monkeypatch, Pool)
    src = np.zeros(8 << 20, dtype=np.uint8)
    assert _hand_over(sink, src) == 1
    n = len(ended)
    time.sleep(0.2)
    assert len(ended) == n and ctx._pool is None
    with pytest.raises(KeyboardInterrupt):
        sink.result()


@pytest.mark.gpu
def test_drain_stopped():
    import tuna_gb300 as T
    seq = np.frombuffer(b"ACGT", dtype=np.uint8)[np.random.default_rng(1).integers(0, 4, 400_000)]
    with T.Context(0) as ctx:
        def fail(data, nbytes):
            raise MemoryError
        ctx._drained = fail
        with pytest.raises(MemoryError):
            ctx.run(31, 21, seq=seq, drain=0)
        del ctx._drained
        r, _ = ctx.run(31, 21, seq=seq, drain=0)  # the context goes on
        assert r.formatted.count(b"\n") == len(r)
