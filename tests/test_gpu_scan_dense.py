"""Databases with runs of identical (or nearly identical) rows against as many identical queries:
one look at a warp's accumulator columns finds up to 32 x 32 candidates, more than its queue
holds (96). Exactly a queue's worth, one more, and all of them, each after a partly filled queue,
in the three scans that queue candidates, against the oracle's scalar matcher (exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# a look covers `rows` consecutive rows x `queries` consecutive queries: three rows per column
# (8 columns x 32 lanes), three queries per column, FP8 pairs of queries
FORMS = {"rows3": (4, 24, 32, (128, 100)), "triples": (4, 32, 24, (720, 743)),
         "pairs": (5, 32, 32, (512, 500))}


def near(base, n, flips, rng, yp):
    return np.stack([yp.synth.flip_bits(base, flips, rng) for _ in range(n)])


def as_set(h):
    return set(zip(h["index"].tolist(), h["query"].tolist(), h["distance"].tolist()))


@pytest.mark.parametrize("t", [0, 36])
@pytest.mark.parametrize("form,n_q", [(f, n) for f in FORMS for n in FORMS[f][3]])
def test_more_candidates_than_a_queue(ctx, yp, oracle, form, n_q, t):
    algo, w_rows, w_q, _ = FORMS[form]
    rng = np.random.default_rng(n_q + t)
    common, other = yp.synth.rows_128(2, seed=n_q)
    # in every look one query is `other`, the rest `common`; so a common rows and b other rows
    # in a look's rows make (w_q - 1) a + b candidates
    last = np.arange(n_q) % w_q == w_q - 1
    queries = np.where(last[:, None], near(other, n_q, t // 2, rng, yp),
                       near(common, n_q, t // 2, rng, yp))
    rows = yp.synth.rows_128(3001, seed=n_q + 1)
    full = 96 // (w_q - 1)
    rest = 96 - full * (w_q - 1)
    looks = [(1, 0), (full, rest), (1, 1), (full, rest + 1), (2, 0), (w_rows, 0), (0, 3),
             (w_rows - 1, 1), (full, rest), (full, rest), (0, w_rows), (1, 0)]
    for i, (a, b) in enumerate(looks):
        at = w_rows * (i + 2)
        rows[at:at + a] = near(common, max(a, 1), t // 2, rng, yp)[:a]
        rows[at + a:at + a + b] = near(other, max(b, 1), t // 2, rng, yp)[:b]
    rows[-1] = rows[w_rows * 2]
    want = oracle.find_all(rows, queries, t)
    assert len(want) >= sum(a for a, _ in looks) * int((~last).sum())
    got = yp.scan(ctx, rows, queries, t, algo=algo, capacity=1 << 17)
    assert np.array_equal(got, want.astype(yp.HIT_DTYPE))
    # a hit buffer that ends inside a flush: the count stays exact, what is stored are hits
    d_rows, d_q = ctx.to_device(rows), ctx.to_device(queries)
    for cap in (0, 97, 1000):
        d_hits, d_cnt = ctx.alloc(cap * 16 + 32), ctx.alloc(8)
        guard = np.full(32, 0xCD, np.uint8)
        d_hits.upload(guard, offset=cap * 16)
        yp.core.scan_device(ctx, d_rows, len(rows), d_q, n_q, t, d_hits, cap, d_cnt, algo)
        assert int(d_cnt.download((1,), np.uint64)[0]) == len(want)
        stored = as_set(d_hits.download((cap,), yp.HIT_DTYPE))
        assert len(stored) == cap and stored <= as_set(want)
        assert np.array_equal(d_hits.download((32,), np.uint8, offset=cap * 16), guard)
