"""The reference's matcher surface (PDQMatcher) backed by the CUDA scan.

Mirrors src/matching/mod.rs:50-105 (the PDQMatcher trait) in the accelerator style of
src/matching/vulkan.rs: the matcher owns the haystack (a device-resident database) and is
queried with needles. Unlike VulkanMatcher (FindsAllMatches = B0), this matcher returns
every hit with its distance, as CpuMatcher does.
"""
import numpy as np

from . import _lib, core


class CudaVectorDatabase(core.Database):
    """Device-resident haystack; mirror of VulkanVectorDatabase::new (vulkan.rs:46-64)."""

    def __init__(self, ctx, data):
        super().__init__(ctx, rows=data)
        self.num_vectors = self.n_rows


class CudaMatcher:
    """PDQMatcher over a CudaVectorDatabase with a fixed threshold. Calls borrow their device
    buffers from the context, so threads can share a matcher. (The word in which a scan reports
    that it gave up waiting is the context's: one of the threads that wait on it gets the error.)"""

    InputDimension = 32
    NoFalseNegative = True
    NoFalsePositive = True
    FindsAllMatches = True

    def __init__(self, ctx, haystack, threshold, algo=_lib.SCAN_AUTO):
        if not 0 <= int(threshold) <= 256:
            raise ValueError("threshold must be in [0, 256]")
        self.ctx = ctx
        self.haystack = haystack
        self.threshold = int(threshold)
        self.algo = algo

    @staticmethod
    def ident():
        return "CUDA sm_103a exact matcher"

    def _launch(self, work, q, d_hits, capacity):
        """Scan needles q, whose copy lies 64 bytes into `work`, and read the count (its first
        8 bytes), which waits for the scan."""
        d_rows, n = self.haystack.device_rows()
        core.scan_device(self.ctx, d_rows, n, work.at(64), q.shape[0], self.threshold, d_hits,
                         capacity, work, self.algo)
        return int(work.download((1,), np.uint64)[0])

    def _needles(self, needles):
        """Needles [q, 32] u8 and a borrowed buffer with them; the copy runs ahead of the scan
        on the same stream."""
        q = np.ascontiguousarray(needles, np.uint8).reshape(-1, 32)
        work = self.ctx.borrow(64 + q.nbytes)
        if q.shape[0]:
            _lib.check(self.ctx.lib.ypdq_memcpy(self.ctx.handle, work.at(64), _lib.ptr(q), q.nbytes,
                                                _lib.H2D, None))
        return q, work

    def scan(self, needles):
        """True if any haystack row is within the threshold of any needle."""
        q, work = self._needles(needles)
        total = self._launch(work, q, None, 0)
        self.ctx.give_back(work)
        return total > 0

    def find_all(self, needles, capacity=1 << 16):
        """Every hit (index, query, distance), sorted by (index, query)."""
        q, work = self._needles(needles)
        while True:
            d_hits = self.ctx.borrow(max(capacity, 1) * 16)
            total = self._launch(work, q, d_hits, capacity)
            if total <= capacity:
                break
            self.ctx.give_back(d_hits)
            capacity = total
        if total > 1:
            core.sort_hits_device(self.ctx, d_hits, total)
        hits = (d_hits.download((total,), _lib.HIT_DTYPE) if total
                else np.zeros(0, _lib.HIT_DTYPE))
        self.ctx.give_back(d_hits)
        self.ctx.give_back(work)
        return hits

    def find(self, needles, f):
        """Call f(haystack_index, needle_index) for hits in (index, needle) order until it
        returns something other than None, and return that (PDQMatcher::find)."""
        for h in self.find_all(needles):
            r = f(int(h["index"]), int(h["query"]))
            if r is not None:
                return r
        return None
