"""The launcher's split of a scan at t <= 36 into triple passes and launches of 128 queries:
query counts on both sides of each switch, on databases on both sides of it, against the
oracle's scalar matcher (exact, so no tolerance). Hits of every part, and rows that hit
queries of several parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {60_000: (128, 129, 256, 385, 720, 721), 500_000: (129, 256, 257, 512, 848, 849),
         2_500_000: (256, 257, 384, 385), 4_200_000: (1023, 1104, 1105)}


@pytest.mark.parametrize("n_rows", sorted(SIZES))
def test_split_scan_matches_oracle(ctx, yp, oracle, n_rows):
    base = oracle.synth_rows(n_rows, n_rows)
    for nq in SIZES[n_rows]:
        queries = yp.synth.rows_128(nq, seed=nq)
        queries[nq // 2] = queries[0]  # one row hits the first and a later part
        rows = base.copy()
        yp.synth.plant(rows, queries, 300, 0, 40, seed=nq)
        rows[n_rows - 1] = queries[nq - 1]
        got = yp.scan(ctx, rows, queries, 31)
        want = oracle.find_all(rows, queries, 31)
        assert np.array_equal(got, want.astype(yp.HIT_DTYPE)), (n_rows, nq)
        assert len(got) > 100
