"""The chunks of ypdq_screen_host grow no faster than the copies can follow (host only): by the
kernels' measured times, chunk c + 1 has arrived when chunk c is done."""
import ctypes

import numpy as np
import pytest

# image bytes; hash us: a chunk's fixed part (one wave, the launches, the scan's start), per image
KINDS = {0: (1 << 20, 45.0, 0.16), 1: (1 << 18, 41.0, 0.079), 2: (3 << 18, 53.0, 0.15)}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("rows,t", [(60_000, 31), (1_000_000, 31), (10_000_000, 31),
                                    (60_000, 48), (1_000_000, 48), (10_000_000, 48)])
def test_chunks_do_not_outgrow_the_copies(yp, kind, rows, t):
    lib = yp._lib.load()
    size, fixed, each = KINDS[kind]
    copy = size / 2.11e5  # us an image at the host link's 211 GB/s
    compute = each + 8.0 * rows / (26.0e6 if t <= 36 else 9.5e6)
    granule = 90 if t <= 36 else 32
    bounds, k = (ctypes.c_int64 * 33)(), ctypes.c_int()
    for n in (200, 600, 1024, 2048):
        assert lib.ypdq_screen_plan(n, kind, 0, rows, t, bounds, ctypes.byref(k)) == yp._lib.OK
        end = np.array([bounds[i] for i in range(k.value + 1)], np.float64)
        for c in range(1, k.value - 1):  # (the last chunk may take a remainder)
            if end[c + 1] - end[c] > granule:
                done = end[1] * copy + end[c] * max(compute, copy) + c * fixed
                assert end[c + 1] * copy <= done, (n, c, np.diff(end))
