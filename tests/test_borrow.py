"""The context's borrowed device buffers: reuse, bounds, and release at close, on a fake library
(no GPU)."""
import ctypes
import threading

import numpy as np


class FakeLib:
    def __init__(self):
        self.live, self.next, self.lock = {}, 1 << 20, threading.Lock()
        self.mallocs = 0

    def ypdq_malloc_device(self, handle, nbytes, out):
        with self.lock:
            self.mallocs += 1
            self.live[self.next] = nbytes
            out._obj.value = self.next
            self.next += 1 << 24
        return 0

    def ypdq_free_device(self, handle, p):
        with self.lock:
            del self.live[p.value]
        return 0

    def ypdq_ctx_destroy(self, handle):
        return 0


def fake_context(yp):
    ctx = yp.Context.__new__(yp.Context)
    ctx.lib, ctx.handle, ctx.device = FakeLib(), ctypes.c_void_p(1), 0
    ctx._spare, ctx._spare_lock = [], threading.Lock()
    return ctx


def test_buffers_are_reused_bounded_and_released(yp):
    ctx = fake_context(yp)
    a = ctx.borrow(100)
    address = a.address
    ctx.give_back(a)
    assert ctx.borrow(64).address == address and ctx.lib.mallocs == 1  # reused (and dropped: freed)
    assert not ctx.lib.live
    big, small = ctx.borrow(1 << 20), ctx.borrow(10)
    ctx.give_back(big)
    other = ctx.borrow(10)  # a large buffer is not spent on a small need
    assert other.nbytes == 1 << 16
    ctx.give_back(small)
    ctx.give_back(other)
    huge = ctx.borrow((1 << 20) + 1)
    ctx.give_back(huge)  # past the bound: freed
    assert len(ctx._spare) == 3
    many = [ctx.borrow(1 << 18) for _ in range(20)]
    for b in many:
        ctx.give_back(b)
    assert len(ctx._spare) == ctx.SPARE_BUFFERS == len(ctx.lib.live)
    ctx.close()
    assert not ctx.lib.live


def test_threads_never_share_a_borrowed_buffer(yp):
    ctx = fake_context(yp)
    held, errors = set(), []
    lock = threading.Lock()

    def work(seed):
        rng = np.random.default_rng(seed)
        for _ in range(300):
            b = ctx.borrow(int(rng.integers(1, 1 << 20)))
            with lock:
                if b.address in held:
                    errors.append(b.address)
                held.add(b.address)
            with lock:
                held.discard(b.address)
            ctx.give_back(b)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    ctx.close()
    assert not ctx.lib.live
