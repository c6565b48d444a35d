"""The rank-127 selection behind every threshold, where its rounds end differently: keys that
differ early, only in their last bits or not at all, ties around the rank, both zeros,
subnormals and infinities. Exact: the threshold is one of the 256 values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrices(kind, n, rng):
    if kind == "random":
        return rng.standard_normal((n, 256)).astype(np.float32) * 50
    if kind == "equal":
        return np.full((n, 256), 1.5, np.float32)
    if kind == "last_bits":  # 1 + k ulp, in any order
        return (np.float32(1).view(np.int32) + rng.permuted(
            np.tile(np.arange(256, dtype=np.int32), (n, 1)), axis=1)).view(np.float32)
    if kind == "ties":  # the rank lies inside, at an end of, or beside a run of equal values
        m = np.sort(rng.standard_normal((n, 256)).astype(np.float32), axis=1)
        for i in range(n):
            a = 120 + i % 9
            m[i, a:a + 1 + i % 16] = m[i, a]
        return rng.permuted(m, axis=1)
    if kind == "zeros":
        return rng.choice(np.array([-0.0, 0.0, -1e-42, 1e-42], np.float32), (n, 256))
    return rng.choice(np.array([-np.inf, np.inf, -1, 1, 3e38], np.float32), (n, 256))


@pytest.mark.parametrize("kind", ["random", "equal", "last_bits", "ties", "zeros", "infinities"])
def test_rank127(ctx, yp, kind):
    n = 48
    p = matrices(kind, n, np.random.default_rng(11)).reshape(n, 16, 16)
    got = yp.core.dihedrals_batch(ctx, p, np.zeros(n, np.float32))
    for s in range(1, 4):
        v = got["pdqf"][:, s].reshape(n, 256)
        thr = np.sort(v, axis=1)[:, 127]
        for slot in (s, s + 4):
            assert np.array_equal(got["thresholds"][:, slot], thr)
            bits = got["pdqf"][:, slot].reshape(n, 256) > thr[:, None]
            packed = np.packbits(bits, axis=1, bitorder="little")[:, ::-1]
            assert np.array_equal(got["hashes"][:, slot], packed)


def test_non_finite_images_on_both_kernels(ctx, yp):
    """A NaN or infinite pixel spreads over the PDQF; whatever comes of it does not depend on
    the batch size (few images take another kernel)."""
    rng = np.random.default_rng(12)
    imgs = np.tile(rng.random((6, 512, 512), dtype=np.float32) * 255, (22, 1, 1))
    for i, bad in enumerate([np.nan, np.inf, -np.inf, 3e38, 1e38, np.nan]):
        imgs[i::6, 17 * i + 40, 70 * i + 5] = bad
    imgs[5::6] = np.nan
    few, many = yp.core.hash_batch(ctx, imgs[:6]), yp.core.hash_batch(ctx, imgs)
    for key in ("hashes", "quality", "thresholds"):
        assert np.array_equal(np.tile(few[key], (22,) + (1,) * (few[key].ndim - 1)), many[key],
                              equal_nan=key != "hashes")
