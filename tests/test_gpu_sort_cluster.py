"""The in-place sort of 257 to 512 hits by one cluster: the edges of its range, of a CTA's 64
hits and of a warp's share of the comparisons; all hits equal, in order, and random."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 257, 263, 264, 319, 320, 321, 449, 505, 511, 512, 513])
@pytest.mark.parametrize("kind", ["random", "equal", "sorted"])
def test_sort_cluster(ctx, yp, n, kind):
    rng = np.random.default_rng(n)
    h = np.zeros(n, yp.HIT_DTYPE)
    if kind == "random":
        h["index"] = rng.integers(0, n // 2, n, dtype=np.uint64) << np.uint64(40)
        h["query"] = rng.integers(0, 3, n, dtype=np.uint64).astype(np.uint32)
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
    assert np.array_equal(got, h[np.lexsort((np.arange(n), h["query"], h["index"]))])
    assert np.array_equal(d.download((32,), np.uint8, offset=16 * n), guard)
