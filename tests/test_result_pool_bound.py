"""The byte bound of the result pool while batches come and go on other
threads, and the size of the block behind a result."""
from __future__ import annotations

import sys
import threading
import time
import types

import numpy as np


class _FakeLib:
    """The batch calls of the library that touch no result, on the host."""

    def cfd_batch_create(self, ctx, precision, capacity, out):
        out._obj.value = 1
        return 0

    def cfd_batch_destroy(self, h):
        return 0

    def cfd_batch_remove(self, h, slot):
        return 0

    def cfd_batch_add_staged(self, h, staged, out):
        out._obj.value = 0
        return 0


def _ctx():
    def check(status, where):
        assert status == 0, where
    return types.SimpleNamespace(lib=_FakeLib(), h=1, check=check, _children=set())


def test_batches_of_other_threads_do_not_disturb_the_bound(pkg):
    from cfd_gb300 import runtime
    errors, stop = [], threading.Event()

    def guarded(work):
        def run():
            try:
                while not stop.is_set():
                    work()
            except BaseException as e:
                errors.append(e)
                stop.set()
        return run

    def come_and_go():
        ctx = _ctx()
        bs = [runtime.Batch(ctx) for _ in range(8)]
        for b in bs:
            b.add_staged(types.SimpleNamespace(take=lambda: None, rows=1000))
            b.remove(0)
            b.close()
        ctx._children.clear()

    was = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        ts = [threading.Thread(target=guarded(w))
              for w in (come_and_go, come_and_go, runtime._results.trim, lambda: runtime._results._limit())]
        [t.start() for t in ts]
        end = time.time() + 5.0
        while time.time() < end and not stop.is_set():
            time.sleep(0.05)
        stop.set()
        [t.join() for t in ts]
    finally:
        sys.setswitchinterval(was)
    assert not errors, errors[0]
    assert runtime._results._limit() == 0


def test_the_bound_follows_the_largest_open_batch(pkg):
    from cfd_gb300 import runtime
    ctx = _ctx()
    a, b = runtime.Batch(ctx), runtime.Batch(ctx)
    a.add_staged(types.SimpleNamespace(take=lambda: None, rows=1000))
    b.add_staged(types.SimpleNamespace(take=lambda: None, rows=300))
    assert runtime._results._limit() == 2 * 1000 * 9 * 8
    a.remove(0)
    assert runtime._results._limit() == 2 * 300 * 9 * 8
    b.close()
    assert runtime._results._limit() == 0
    a.close()


def test_a_result_never_sits_on_a_block_twice_the_next_power_of_two(pkg):
    from cfd_gb300 import runtime
    p = runtime._HostBlocks(lambda: 1 << 20)
    large = p.array(20, 9)                      # 180 values: a block of 256
    at = large.ctypes.data
    del large
    small = p.array(10, 9)                      # 90 values: one of 128, not the free 256
    assert small.ctypes.data != at and small.base.mem.size == 128
    assert small.flags.writeable and not small.flags.owndata
    grown = small.copy()
    grown.resize((11, 9))                       # a copy owns its data
    assert np.array_equal(grown[:10], small)
