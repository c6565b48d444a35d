"""Parity of the small-batch hash kernel (one image per cluster of CTAs) with the oracle.

Batch sizes on both sides of each input kind's switch to the persistent kernel, and the
smallest. FP32 results are bit-exact, so the tolerance is zero.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("f32", n) for n in (1, 2, 56, 57, 88, 89)] + \
        [("u8", n) for n in (1, 104, 105, 208, 209)] + \
        [("rgb8", n) for n in (1, 72, 73, 184, 185)] + [("rgba8", n) for n in (1, 72, 73, 176, 177)]


def images_of(yp, kind, n):
    if kind in ("rgb8", "rgba8"):
        few = yp.synth.color_images(min(n, 6), seed=n, channels=3 if kind == "rgb8" else 4)
        rng = np.random.default_rng(n)
        imgs = rng.integers(0, 256, (n,) + few.shape[1:], dtype=np.uint8)
        imgs[-len(few):] = few
        return imgs
    imgs, _ = yp.synth.mixed_images(min(n, 12), seed=n)
    imgs = imgs[np.arange(n) % len(imgs)] + (np.arange(n, dtype=np.float32) // 12)[:, None, None]
    return yp.synth.to_u8(imgs) if kind == "u8" else imgs


@pytest.mark.parametrize("kind,n", CASES)
def test_split_kernel_matches_oracle(ctx, yp, oracle, kind, n):
    imgs = images_of(yp, kind, n)
    got = yp.hash_batch(ctx, imgs, want_pdqf=True, pdqf_slots=8, want_buf1=True)
    plain = oracle.luma(imgs) if imgs.ndim == 4 else imgs.astype(np.float32)
    h, q, t, p = oracle.hash_batch(plain, want_pdqf=True)
    assert np.array_equal(got["hashes"], h)
    assert np.array_equal(got["quality"], q)
    assert np.array_equal(got["thresholds"], t)
    assert np.array_equal(got["pdqf"][:, 0], p)
    for i in {0, n - 1}:
        assert np.array_equal(got["buf1"][i], oracle.compress(plain[i]))
        dh, _, _, dp = oracle.dihedrals(p[i], t[i, 0], "exact")
        assert np.array_equal(got["pdqf"][i, 1:], dp)
        assert np.array_equal(got["hashes"][i, 1:], dh)


@pytest.mark.parametrize("semantics", ["avx2", "scalar"])
def test_split_kernel_semantics(ctx, yp, oracle, semantics):
    imgs, _ = yp.synth.mixed_images(5, seed=3)
    got = yp.hash_batch(ctx, imgs, semantics=semantics)
    h, q, t, _ = oracle.hash_batch(imgs, semantics=semantics)
    assert np.array_equal(got["hashes"], h)
    assert np.array_equal(got["quality"], q)
    assert np.array_equal(got["thresholds"], t)


def test_split_kernel_degenerate_images(ctx, yp, oracle):
    """Constant, black and single-pixel images: equal values around the median, zero
    gradients, subnormal residues."""
    imgs = np.zeros((5, 512, 512), np.float32)
    imgs[1] = 255.0
    imgs[2] = 77.0
    imgs[3, 200, 300] = 255.0
    imgs[4, :, 505:] = 1e-30
    got = yp.hash_batch(ctx, imgs, want_pdqf=True)
    h, q, t, p = oracle.hash_batch(imgs, want_pdqf=True)
    assert np.array_equal(got["hashes"], h)
    assert np.array_equal(got["quality"], q)
    assert np.array_equal(got["thresholds"], t)
    assert np.array_equal(got["pdqf"][:, 0], p)
