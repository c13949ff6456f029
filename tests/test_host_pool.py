"""The pool behind `Engine.step_tokens`' results, with a counting allocator in place of page-locked memory."""
import ctypes
import gc
import threading

import numpy as np

from imp_b200.engine.host_pool import GRAIN, HostPool


class Heap:
    def __init__(self):
        self.blocks, self.made = {}, 0

    def alloc(self, size):
        b = ctypes.create_string_buffer(size)
        self.blocks[ctypes.addressof(b)] = b
        self.made += 1
        return ctypes.addressof(b)

    def free(self, address):
        del self.blocks[address]


def make(limit):
    heap = Heap()
    return heap, HostPool(limit, heap.alloc, heap.free)


def test_a_block_serves_again_only_when_nothing_refers_to_it():
    heap, pool = make(1 << 24)
    a = pool.array((3, 1000))
    assert a.shape == (3, 1000) and a.dtype == np.float32 and a.flags.writeable and a.flags.c_contiguous
    a[:] = 1
    view, address = a[1, 10:20], a.ctypes.data
    del a
    b = pool.array((3, 1000))
    b[:] = 2
    assert b.ctypes.data != address and (view == 1).all() and heap.made == 2
    del view
    assert pool.array((2, 1500)).ctypes.data == address and heap.made == 2


def test_limit_and_other_sizes():
    heap, pool = make(4 * GRAIN)
    held = [pool.array((GRAIN // 4,)) for _ in range(6)]        # two of them in ordinary memory
    assert heap.made == 4 and pool.held == 4 * GRAIN
    for i, a in enumerate(held):
        a[:] = i
    assert [a[5] for a in held] == list(range(6))
    del held, a
    big = pool.array((GRAIN,))                                  # the small blocks make room
    assert pool.held == 4 * GRAIN and len(heap.blocks) == 1 and big.size == GRAIN
    assert pool.array((8 * GRAIN,)).size == 8 * GRAIN and len(heap.blocks) == 1
    assert pool.array((0, 7)).shape == (0, 7)


def test_a_request_beyond_the_limit_leaves_the_free_blocks():
    heap, pool = make(4 * GRAIN)
    small, lent = pool.array((GRAIN // 4,)), pool.array((GRAIN // 2,))
    address = small.ctypes.data
    del small
    assert pool.array((8 * GRAIN,)).size == 8 * GRAIN               # larger than the pool
    assert pool.array((3 * GRAIN // 4,)).size == 3 * GRAIN // 4     # does not fit beside what is lent out
    assert pool.held == 3 * GRAIN and heap.made == 2
    assert pool.array((GRAIN // 4,)).ctypes.data == address and lent.size


def test_close_frees_now_and_later():
    heap, pool = make(1 << 24)
    a, b = pool.array((10,)), pool.array((10,))
    del b
    pool.close()
    assert len(heap.blocks) == 1 and (pool.array((10,)).size == 10) and len(heap.blocks) == 1
    a[:] = 3
    del a
    gc.collect()
    assert not heap.blocks and pool.held == 0


def test_no_page_locked_memory():
    pool = HostPool(1 << 24, lambda size: 0, None)
    assert pool.array((5, 5)).shape == (5, 5) and pool.held == 0


def test_an_engines_pool_allocates_on_the_engines_device(monkeypatch):
    calls = []

    class Library:
        def imp_host_alloc(self, size, out):
            calls.append(None)
            return 1

        def imp_context_host_alloc(self, ctx, size, out):
            calls.append((ctx, size))
            return 1

    monkeypatch.setattr("imp_b200.engine.host_pool.capi.load", Library)
    assert HostPool(1 << 24, context=77).array((GRAIN,)).size == GRAIN and calls == [(77, 4 * GRAIN)]
    assert HostPool(1 << 24).array((5,)).size == 5 and calls[1:] == [None]
    assert HostPool(0, context=77).array((5,)).size == 5 and len(calls) == 2      # no page-locked memory at all


def test_threads():
    heap, pool = make(64 * GRAIN)
    wrong = []

    def work(n):
        for i in range(300):
            a = pool.array((GRAIN // 4 * (1 + i % 3),))
            a[:] = n
            if not (a == n).all():
                wrong.append(n)

    threads = [threading.Thread(target=work, args=(n,)) for n in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong and pool.held == sum(len(b) for b in heap.blocks.values()) <= 64 * GRAIN
