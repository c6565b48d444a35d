"""The persistent hash kernel sums the taps of two row groups side by side for byte input. Images
whose energy sits where a group, a pair or the image begins and ends, and constant ones, are
bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PIXELS = [(0, 0), (1, 2), (2, 5), (4, 6), (5, 6), (8, 8), (9, 10), (12, 3), (13, 510), (506, 509),
          (507, 2), (508, 510), (509, 509), (510, 510), (511, 511)]


@pytest.mark.parametrize("kind,n", [("u8", 117), ("rgb8", 85), ("rgba8", 85)])
def test_edges_of_groups(ctx, yp, oracle, kind, n):
    channels = {"u8": (), "rgb8": (3,), "rgba8": (4,)}[kind]
    few = np.zeros((len(PIXELS) + 2, 512, 512) + channels, np.uint8)
    for i, (r, c) in enumerate(PIXELS):
        few[i, r, c] = 255
        few[i, r, (c + 4) % 512] = 3
    few[-2], few[-1] = 255, 77
    imgs = few[np.arange(n) % len(few)]
    got = yp.hash_batch(ctx, imgs, want_pdqf=True, want_buf1=True)
    plain = oracle.luma(few) if channels else few.astype(np.float32)
    h, q, t, p = oracle.hash_batch(plain, want_pdqf=True)
    for i in range(n):
        k = i % len(few)
        assert np.array_equal(got["hashes"][i], h[k])
        assert np.array_equal(got["quality"][i], q[k])
        assert np.array_equal(got["pdqf"][i, 0], p[k])
    for k in range(len(few)):
        assert np.array_equal(got["buf1"][n - len(few) + k], oracle.compress(plain[(n + k) % len(few)]))
