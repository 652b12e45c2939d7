"""Host memory of a batch's results: reused only when nothing refers to it,
bounded, and safe to drop from any thread."""
from __future__ import annotations

import threading

import numpy as np


def _pool(limit):
    from cfd_gb300 import runtime
    return runtime._HostBlocks(lambda: limit)


def test_a_block_is_reused_only_after_its_last_view():
    p = _pool(10_000)
    a = p.array(10, 9)
    at = a.ctypes.data
    assert a.shape == (10, 9) and a.dtype == np.float64 and a.flags.writeable and a.flags.c_contiguous
    view = a[3:].T
    del a
    b = p.array(10, 9)
    assert b.ctypes.data != at          # the view still holds the block
    del view
    c = p.array(10, 9)
    assert c.ctypes.data == at
    assert p.array(10, 9).ctypes.data not in (at, b.ctypes.data)
    del c
    d = p.array(8, 13)                          # 104 of the block's 128 values
    assert d.ctypes.data == at and d.shape == (8, 13)
    assert p.array(15, 9).ctypes.data != at     # 135 values: a larger block


def test_at_most_the_limit_is_kept():
    from cfd_gb300 import runtime
    limit = [2 * 1024]
    p = runtime._HostBlocks(lambda: limit[0])
    arrays = [p.array(10, 9) for _ in range(5)]
    del arrays
    assert p._held == 2 * 1024
    limit[0] = 1024
    p.trim()
    assert p._held == 1024
    limit[0] = 0
    p.trim()
    assert p._held == 0 and p.array(10, 9).shape == (10, 9)


def test_many_threads():
    p, bad = _pool(1 << 20), []

    def work(k):
        for i in range(300):
            a = p.array(16, 9)
            a[:] = k
            if not (a == k).all():
                bad.append((k, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad and 0 <= p._held <= 1 << 20
