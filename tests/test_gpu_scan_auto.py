"""YPDQ_SCAN_AUTO on both sides of each line of its rule by query count, threshold and database
size: the hits are the oracle's scalar matcher's on either side (exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {199_999: (9, 10, 32, 33), 200_000: (6, 7, 16, 17, 32, 33), 200_001: (6, 7, 16, 17, 32),
         1_500_000: (9, 16, 17), 1_500_001: (9, 10, 16), 2_000_000: (8, 9), 2_000_001: (6, 7, 8)}


@pytest.mark.parametrize("n_rows", sorted(SIZES))
@pytest.mark.parametrize("threshold", [34, 36])
def test_auto_matches_oracle(ctx, yp, oracle, n_rows, threshold):
    rows = oracle.synth_rows(n_rows, n_rows)
    for nq in SIZES[n_rows]:
        queries = yp.synth.rows_128(nq, seed=nq)
        db = rows.copy()
        yp.synth.plant(db, queries, 200, 0, 40, seed=nq)
        db[n_rows - 1] = queries[nq - 1]
        got = yp.scan(ctx, db, queries, threshold)
        want = oracle.find_all(db, queries, threshold)
        assert np.array_equal(got, want.astype(yp.HIT_DTYPE)), (n_rows, nq)
        assert len(got) > 100
