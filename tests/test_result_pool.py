"""Result arrays in page-locked memory (gpu.ResultPool): blocks are used again
once nothing refers to them, never while an array does, and the pool keeps to
its bounds.  The allocator is faked, so this runs without a GPU."""

import ctypes
import gc
import threading

import numpy as np
import pytest


@pytest.fixture
def pool(monkeypatch):
    from argent_b200 import gpu as G

    live = {}

    class Lib:
        def argent_pinned_alloc(self, n, out):
            if getattr(self, "fail", False):
                return 1
            buf = ctypes.create_string_buffer(n)
            p = ctypes.addressof(buf)
            live[p] = buf
            ctypes.cast(out, ctypes.POINTER(ctypes.c_void_p))[0] = p
            return 0

        def argent_pinned_free(self, p):
            del live[p]

    lib = Lib()
    monkeypatch.setattr(G.N, "gpu", lambda: lib)
    p = G.ResultPool()
    p.live, p.lib = live, lib
    return p


def test_blocks_are_reused_after_their_last_view(pool):
    a = pool.array((300, 200, 3), np.float32)
    assert a.shape == (300, 200, 3) and a.dtype == np.float32 and a.flags.writeable and len(pool.live) == 1
    a[:] = 7.0
    view, at = a[10:20, :, 1], a.ctypes.data
    b = pool.array((300, 200, 3), np.float32)
    assert b.ctypes.data != at
    del a
    gc.collect()
    c = pool.array((300, 200, 3), np.float32)  # the view still holds the first block
    assert c.ctypes.data != at and (view == 7.0).all()
    del view
    gc.collect()
    d = pool.array((299, 200, 3), np.float32)  # a nearby size takes it
    assert d.ctypes.data == at and len(pool.live) == 3


def test_bounds_and_fallbacks(pool):
    small = pool.array(100, np.uint8)
    assert small.flags.owndata and pool.total == 0
    pool.LIMIT, pool.IDLE = 3 << 20, 1 << 20
    held = [pool.array(1 << 20, np.uint8) for _ in range(4)]
    assert pool.total <= pool.LIMIT and sum(x.flags.owndata for x in held) == 1
    del held
    gc.collect()
    assert pool.idle <= pool.IDLE and pool.total == pool.idle == sum(len(b) for b in pool.live.values())
    other = pool.array((5 << 20) // 2, np.uint8)  # waiting blocks make room
    assert not other.flags.owndata and pool.total <= pool.LIMIT
    pool.lib.fail = True
    assert pool.array(1 << 18, np.uint8).flags.owndata
    assert pool.array((0, 4), np.float32).shape == (0, 4)


def test_waiting_blocks_of_old_sizes_make_room(pool):
    pool.IDLE = 3 << 20
    held = [pool.array(1 << 20, np.uint8) for _ in range(3)]
    del held
    gc.collect()
    assert pool.idle == pool.IDLE
    a = pool.array(3 << 19, np.uint8)
    del a
    gc.collect()
    assert pool.idle <= pool.IDLE and pool.total == pool.idle == sum(len(b) for b in pool.live.values())
    pool.lib.fail = True  # nothing can be page-locked anew: the block was kept
    assert not pool.array(3 << 19, np.uint8).flags.owndata


def test_threads(pool):
    def work(k):
        for i in range(50):
            a = pool.array(70_000 + 1000 * (i % 5), np.uint8)
            a[:] = k
            assert (a == k).all()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    gc.collect()
    assert pool.total == pool.idle == sum(len(b) for b in pool.live.values())
