"""Threads that share one matcher: each gets its own needles' hits, with lists of every sort
(none, few, hundreds, thousands) and calls that overflow their first capacity."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_share_a_matcher(ctx, yp, oracle):
    rows = oracle.synth_rows(200_000, 3).copy()
    needles = [yp.synth.rows_128(8, seed=100 + i) for i in range(6)]
    for q, count in zip(needles, (0, 1, 40, 300, 700, 5000)):
        yp.synth.plant(rows, q, count, 0, 25, seed=count + 7)
    want = [oracle.find_all(rows, q, 31).astype(yp.HIT_DTYPE) for q in needles]
    assert len(want[0]) == 0 and len(want[5]) > 2560
    m = yp.CudaMatcher(ctx, yp.CudaVectorDatabase(ctx, rows), 31)
    errors = []

    def work(i):
        try:
            for k in range(60):
                j = (i + k) % 6
                hits = m.find_all(needles[j], capacity=(1 << 16, 100)[k % 2])
                if not np.array_equal(hits, want[j]) or m.scan(needles[j]) != (len(want[j]) > 0):
                    errors.append((i, k, j, len(hits), len(want[j])))
        except Exception as e:
            errors.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]
