"""Scans at t <= 36 that run as several launches: more than 128 queries as launches of 128 with
three database rows per column, and such launches after a pass of 720, on databases large enough
that the launcher chooses them. Exact against the oracle's scalar matcher."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TC, TC_FP4 = 3, 4
# queries, rows: two launches, the last one full and with one query; three, the last partial;
# a pass of 720 and a launch
CASES = [(256, 500_040), (129, 500_041), (300, 2_300_042), (848, 500_041)]


def extremes(yp, oracle, n_q, n_rows):
    """Rows that put every field of a column at its extreme for queries of the first and the last
    launch: equal and complementary to them, differing only in the two prefix bits that the bound
    leaves out, runs of hits in one tile, and the last, partial tile."""
    rows = oracle.synth_rows(n_rows, n_q).copy()
    q = yp.synth.rows_128(n_q, seed=n_q + 1)
    yp.synth.plant(rows, q, 400, 0, 40, seed=n_q + 2)
    last = (n_q - 1) // 128 * 128  # the last launch's first query
    for at, (a, b) in ((30, (0, n_q - 1)), (750, (last, 127)), (n_rows - 40, (n_q - 1, last))):
        rows[at], rows[at + 1], rows[at + 2] = q[a], q[b], ~q[n_q // 2]
        rows[at + 3], rows[at + 4], rows[at + 5] = ~q[a], ~q[b], q[n_q // 2]
        rows[at + 10, :16], rows[at + 10, 16:] = q[b, :16], ~q[b, 16:]
        rows[at + 11, :16], rows[at + 11, 16:] = ~q[b, :16], q[b, 16:]
        for i in range(3):
            rows[at + 20 + i] = q[(a + i) % n_q]
            rows[at + 20 + i, 15] ^= np.uint8(0xC0)
    rows[1440:1536] = q[np.arange(96) % n_q]
    rows[2160:2256] = q[n_q - 1 - np.arange(96) % n_q]
    rows[n_rows - 1], rows[n_rows - 3] = q[0], q[n_q - 1]
    return rows, q


@pytest.mark.parametrize("n_q,n_rows", CASES)
def test_launches_match_oracle(ctx, yp, oracle, n_q, n_rows):
    rows, q = extremes(yp, oracle, n_q, n_rows)
    for t in (0, 2, 31, 36):
        want = oracle.find_all(rows, q, t).astype(yp.HIT_DTYPE)
        for algo in (TC, TC_FP4):
            got = yp.scan(ctx, rows, q, t, algo=algo, capacity=1 << 18)
            assert np.array_equal(got, want), (t, algo, len(got), len(want))


@pytest.mark.parametrize("n_q,n_rows", CASES)
def test_timeout_of_the_first_launch(ctx, yp, oracle, n_q, n_rows):
    """The first of several launches waits for copies that nobody issues (1 ms limit); those after
    it run. The sync reports the timeout, and the next scan on the context is complete."""
    lib = ctx.lib
    rows, q = extremes(yp, oracle, n_q, n_rows)
    d_rows, d_q = ctx.to_device(rows), ctx.to_device(q)
    cap = 1 << 18
    d_hits, d_cnt = ctx.alloc(cap * 16), ctx.alloc(8)
    assert lib.ypdq_set_scan_wait_limit(1_000_000) == 0
    try:
        assert lib.ypdq_debug_stall_scans(1) == 0
        yp.core.scan_device(ctx, d_rows, n_rows, d_q, n_q, 31, d_hits, cap, d_cnt, TC)
        with pytest.raises(yp.YpdqError) as err:
            ctx.sync()
        assert err.value.status == yp._lib.ERR_TIMEOUT
    finally:
        lib.ypdq_debug_stall_scans(0)
        lib.ypdq_set_scan_wait_limit(0)
    want = oracle.find_all(rows, q, 31).astype(yp.HIT_DTYPE)
    assert np.array_equal(yp.scan(ctx, rows, q, 31, algo=TC, capacity=cap), want)
