"""The SIMT scan loads whole 32-byte rows where the database lies on 32-byte boundaries and 16
bytes at a time where it does not: both on each popcount variant, at the edges of a warp's
rows and of the grid, against the oracle's scalar matcher (exact)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 16, 32, 48])
@pytest.mark.parametrize("threshold", [31, 36, 62, 100])
def test_row_alignment(ctx, yp, oracle, offset, threshold):
    for n_rows in (1, 31, 32, 33, 63, 64, 65, 511, 513, 155_648, 311_297, 320_000):
        rows = oracle.synth_rows(n_rows, n_rows).copy()
        queries = yp.synth.rows_128(5, seed=n_rows)
        yp.synth.plant(rows, queries, min(n_rows, 200), 0, 64, seed=n_rows)
        d_rows = ctx.alloc(n_rows * 32 + 64)
        d_rows.upload(rows, offset=offset)
        d_q, d_hits, d_count = ctx.to_device(queries), ctx.alloc(16 << 16), ctx.alloc(8)
        at = ctypes.c_void_p(d_rows.ptr.value + offset)
        yp.core.scan_device(ctx, at, n_rows, d_q, 5, threshold, d_hits, 1 << 16,
                            d_count, yp._lib.SCAN_SIMT)
        n = int(d_count.download((1,), np.uint64)[0])
        yp.core.sort_hits_device(ctx, d_hits, n)
        ctx.sync()
        want = oracle.find_all(rows, queries, threshold)
        assert np.array_equal(d_hits.download((n,), yp.HIT_DTYPE), want.astype(yp.HIT_DTYPE))
