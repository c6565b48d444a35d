"""The sort of hits at the edges of its rules: ranks, tiles whose runs are placed at once
(256, 1,024 and 4,096 hits a run, the last run short, one hit or full), and pairwise merges.
Equal hits all have to appear, in any order among themselves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2559, 2560, 2561, 2816, 2817, 16384, 16385, 17408, 17409, 32768, 32769, 36864, 36865,
         98303, 98304, 98305]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["random", "equal", "sorted"])
def test_sort_rules(ctx, yp, n, kind):
    rng = np.random.default_rng(n)
    h = np.zeros(n, yp.HIT_DTYPE)
    if kind == "random":
        h["index"] = rng.integers(0, n // 2, n, dtype=np.uint64) << np.uint64(33)
        h["query"] = rng.integers(0, 3, n, dtype=np.uint64).astype(np.uint32) + np.uint32(0x7FFFFFFF)
    elif kind == "sorted":
        h["index"] = np.arange(n)
    h["distance"] = np.arange(n) % 257
    d = ctx.alloc((n + 2) * 16)
    guard = np.full(32, 0xCD, np.uint8)
    d.upload(guard, offset=16 * n)
    d.upload(h)
    yp.core.sort_hits_device(ctx, d, n)
    ctx.sync()
    got = d.download((n,), yp.HIT_DTYPE)
    whole = ("distance", "query", "index")
    assert np.array_equal(got[["index", "query"]], np.sort(h[["index", "query"]]))
    assert np.array_equal(got[np.lexsort([got[f] for f in whole])], h[np.lexsort([h[f] for f in whole])])
    assert np.array_equal(d.download((32,), np.uint8, offset=16 * n), guard)
