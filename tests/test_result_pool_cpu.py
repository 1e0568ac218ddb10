"""The page-locked memory under a cache's result arrays: bounded, reused only when no array is left over it, freed in the end."""
import ctypes
import gc

import numpy as np

from fastllm_b200 import models


class FakeLib:
    def __init__(self, refuse=False):
        self.live, self.refuse = {}, refuse

    def fl_host_alloc(self, size, out):
        if self.refuse:
            return -2
        buf = ctypes.create_string_buffer(size)
        out._obj.value = ctypes.addressof(buf)
        self.live[out._obj.value] = buf
        return 0

    def fl_host_free(self, p):
        del self.live[p.value]
        return 0


SHAPE = (4, 8192)


def at(a):
    return a.__array_interface__["data"][0]


def test_blocks_are_reused_only_when_free():
    lib = FakeLib()
    pool = models._ResultPool(lib)
    a = pool.empty(SHAPE)
    a[:] = 1.0
    row, where = a[2], at(a)
    del a
    b = pool.empty(SHAPE)                       # a row of the first result is still held
    assert at(b) != where and len(lib.live) == 2
    c = pool.empty(SHAPE)                       # both blocks are taken: plain memory
    assert at(c) not in lib.live and (row == 1.0).all()
    del row
    gc.collect()
    d = pool.empty((3, 8192))
    assert at(d) == where and d.shape == (3, 8192) and d.dtype == np.float32 and d.flags.writeable and len(lib.live) == 2


def test_sizes_and_refusals():
    lib = FakeLib()
    pool = models._ResultPool(lib)
    assert at(pool.empty((1, 16))) not in lib.live                # small results: a copy is as good
    a = pool.empty(SHAPE)
    del a
    b = pool.empty((8, 8192))                                     # the free block is too small: exchanged, not added to
    assert at(b) in lib.live and len(lib.live) == 1
    assert models._ResultPool(FakeLib(refuse=True)).empty(SHAPE).shape == SHAPE


def test_freed_with_the_pool_or_the_last_array():
    lib = FakeLib()
    pool = models._ResultPool(lib)
    a, b = pool.empty(SHAPE), pool.empty(SHAPE)
    del b
    pool.close()
    assert len(lib.live) == 1
    a[:] = 2.0
    del a
    gc.collect()
    assert not lib.live


class CountingLib(FakeLib):
    def __init__(self):
        super().__init__()
        self.taken = []

    def fl_host_alloc(self, size, out):
        self.taken.append(size)
        return super().fl_host_alloc(size, out)


def test_growing_calls_hardly_ever_page_lock():
    """page-locking a block takes milliseconds: a batch that grows finds its blocks there, and longer and longer results exchange them a few times"""
    lib = CountingLib()
    pool = models._ResultPool(lib)
    pool.reserve((64, 8192))
    assert lib.taken == [2 * 64 * 8192 * 4]                     # both pieces at once
    for b in range(1, 65):
        keep = pool.empty((b, 8192))                            # noqa: F841  (held until the next one is there, as by a program's loop)
    assert len(lib.taken) == 1
    for rows in range(100, 301):
        keep = pool.empty((rows, 8192))                         # noqa: F841
    assert len(lib.taken) <= 1 + 2 * 3 and len(lib.live) == 2


def test_a_block_that_fits_is_taken_before_one_is_exchanged():
    lib = CountingLib()
    pool = models._ResultPool(lib)
    large, small = pool.empty((16, 8192)), pool.empty((4, 8192))
    where = at(large)
    del large
    del small                                                   # (in this order: the small one was given back last)
    assert at(pool.empty((16, 8192))) == where and len(lib.taken) == 2


def test_results_beyond_a_limit_are_plain():
    lib = CountingLib()
    pool = models._ResultPool(lib)
    rows = pool.MOST // (4 * 8192)
    pool.reserve((rows + 1, 8192))
    assert not lib.taken and at(pool.empty((rows + 1, 8192))) not in lib.live
    a = pool.empty((rows // 2 + 1, 8192))
    del a
    b = pool.empty((rows, 8192))                                # an exchanged block stays inside the limit
    assert at(b) in lib.live and max(lib.taken) == pool.MOST


def test_pieces_of_one_memory():
    """the pieces that are taken together do not overlap, and their memory goes with the last of them"""
    lib = CountingLib()
    pool = models._ResultPool(lib)
    pool.reserve((5, 8191))
    a, b = pool.empty((5, 8191)), pool.empty((5, 8191))
    a[:], b[:] = 1.0, 2.0
    assert abs(at(a) - at(b)) >= a.nbytes and (a == 1.0).all() and (b == 2.0).all() and len(lib.live) == 1
    assert at(pool.empty((5, 8191))) not in (at(a), at(b))      # both are held
    del a
    c = pool.empty((50, 8191))                                  # the free piece is exchanged, the other one's memory stays
    c[:] = 3.0
    assert len(lib.live) == 2 and (b == 2.0).all()
    pool.close()
    del b
    gc.collect()
    assert len(lib.live) == 1 and (c == 3.0).all()
    del c
    gc.collect()
    assert not lib.live
