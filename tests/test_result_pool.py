"""The pool that large results lie in: pieces come back when their arrays are dropped, there are never more than it may hold, and
arrays outlive the engine. A stand-in for pinned memory, so that this runs without a GPU."""
import ctypes
import gc
import threading

import numpy as np

import synth

pkg = synth.pkg
N = 1 << 16                     # floats: 256 KB


class FakeLib:
    """g5b_host_alloc / g5b_host_free on ordinary memory, counted."""

    def __init__(self, fails=0):
        self.live, self.allocs, self.fails = {}, 0, fails

    def g5b_host_alloc(self, size):
        if self.fails > 0:
            self.fails -= 1
            return None
        buf = ctypes.create_string_buffer(size)
        self.allocs += 1
        self.live[ctypes.addressof(buf)] = buf
        return ctypes.addressof(buf)

    def g5b_host_free(self, ptr):
        del self.live[ptr]


def test_pieces_are_reused_and_bounded():
    lib = FakeLib()
    pool = pkg._ResultPool(lib)
    for _ in range(10):
        a = pool.array((2, N // 2))
        assert a.shape == (2, N // 2) and a.dtype == np.float32 and a.flags.writeable and a.flags.c_contiguous
        a[:] = 1.0
    assert lib.allocs <= 2                                    # one in hand while the next is made
    held = [pool.array((N,)) for _ in range(20)]              # the caller keeps them all: the rest are ordinary arrays
    assert lib.allocs <= pool.KEEP
    for i, h in enumerate(held):
        h[:] = i
    assert all((h == i).all() for i, h in enumerate(held))    # nobody shares memory
    assert pool.array((16,)).base is None                     # small results are ordinary ones
    view = pool.array((N,))[5:]
    del held, a, h
    gc.collect()
    view[:] = 3.0                                             # a view keeps its piece
    others = [pool.array((N,)) for _ in range(pool.KEEP)]
    for o in others:
        o[:] = 0.0
    assert (view == 3.0).all()
    pool.close()
    assert pool.array((N,)).base is None
    del others, o, view
    gc.collect()
    assert not lib.live


def test_threads_share_a_pool():
    pool, errors = pkg._ResultPool(FakeLib()), []

    def work(k):
        for i in range(300):
            a = pool.array((N,))
            a[:64] = k * 1000 + i
            if not (a[:64] == k * 1000 + i).all():
                errors.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors


def test_pieces_that_could_not_be_had_are_not_counted():
    """Memory that cannot be pinned now may be there later: as many failures as a size may have pieces do not close it."""
    lib = FakeLib(fails=pkg._ResultPool.KEEP + 1)
    pool = pkg._ResultPool(lib)
    pool.reserve(4 * N, 2)
    for _ in range(pool.KEEP - 1):
        assert pool.array((N,)).base is None                  # an ordinary array meanwhile
    assert pool.bytes == 0 and lib.fails == 0
    held = [pool.array((N,)) for _ in range(pool.KEEP + 1)]
    assert lib.allocs == len(lib.live) == pool.KEEP and pool.bytes == pool.KEEP * 4 * N
    del held
    gc.collect()
    pool.close()
    assert not lib.live
