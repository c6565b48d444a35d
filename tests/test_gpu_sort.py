"""The merge sort of hits by (index, query) at the edges of its tiles and passes: a thread's
eight hits, the 2,048- and 8,192-hit tiles, one and several merge passes, runs without a
partner, runs of equal indices, sorted and reversed input."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 255, 2047, 2048, 2049, 8191, 8192, 8193, 10240, 16384, 16385, 24577,
         65536, 100001, 1 << 20]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["random", "ties", "reversed", "interleaved"])
def test_sort_hits_sizes(ctx, yp, n, kind):
    rng = np.random.default_rng(n)
    h = np.zeros(n, yp.HIT_DTYPE)
    if kind == "random":
        h["index"] = rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2) + np.uint64(1)
        h["query"] = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    elif kind == "ties":  # distinct (index, query) pairs, few indices
        h["index"] = rng.permutation(n) % 5
        h["query"] = np.arange(n)
        h = h[rng.permutation(n)]
    elif kind == "reversed":
        h["index"] = np.arange(n)[::-1]
    else:  # every other hit from the far half
        h["index"] = np.arange(n) // 2 + (np.arange(n) % 2) * n
    h["distance"] = rng.integers(0, 257, n)
    d = ctx.alloc((n + 2) * 16)
    guard = np.full(2, 0xAB, np.uint8).repeat(16)
    d.upload(guard, offset=16 * n)
    d.upload(h)
    yp.core.sort_hits_device(ctx, d, n)
    ctx.sync()
    got = d.download((n,), yp.HIT_DTYPE)
    order = np.lexsort((h["query"], h["index"]))
    assert np.array_equal(got, h[order])
    assert np.array_equal(d.download((32,), np.uint8, offset=16 * n), guard)


def test_sort_hits_unaligned(ctx, yp):
    """Hits 8 bytes off a 16-byte boundary, as before."""
    rng = np.random.default_rng(1)
    n = 20000
    h = np.zeros(n, yp.HIT_DTYPE)
    h["index"] = rng.permutation(n)
    d = ctx.alloc(n * 16 + 8)
    d.upload(h, offset=8)
    yp.core.sort_hits_device(ctx, d.at(8), n)
    ctx.sync()
    assert np.array_equal(d.download((n,), yp.HIT_DTYPE, offset=8), np.sort(h, order="index"))
