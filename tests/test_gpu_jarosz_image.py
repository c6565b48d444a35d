"""Parity of the one-kernel Jarosz path (csrc/jarosz.cu) with the oracle: u8 from one image,
f32 and RGB from 32 images on, and the planes just below. Bit-exact, so the tolerance is zero.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JAROSZ = 0x200


def images_of(yp, kind, n):
    rng = np.random.default_rng(n)
    if kind in ("rgb8", "rgba8"):
        imgs = rng.integers(0, 256, (n, 512, 512, 3 if kind == "rgb8" else 4), dtype=np.uint8)
        imgs[:2] = yp.synth.color_images(2, seed=n, channels=imgs.shape[3])
        imgs[2] = 0
        return imgs
    imgs, _ = yp.synth.mixed_images(min(n, 8), seed=n)
    imgs = imgs[np.arange(n) % len(imgs)] + (np.arange(n, dtype=np.float32) // 8)[:, None, None]
    if kind == "u8":
        return yp.synth.to_u8(imgs)
    imgs[1] = 0.0
    imgs[1, 511, 511] = 1e-38  # sums below 2^-120
    imgs[2] *= 1e33
    imgs[3] = rng.normal(0, 100, (512, 512)).astype(np.float32)
    return imgs


@pytest.mark.parametrize("kind,n", [("u8", 1), ("u8", 5), ("f32", 31), ("f32", 32), ("f32", 33),
                                    ("rgb8", 31), ("rgb8", 32), ("rgba8", 32)])
def test_image_kernel_matches_oracle(ctx, yp, oracle, kind, n):
    imgs = images_of(yp, kind, n)
    got = yp.hash_batch(ctx, imgs, dct=JAROSZ, semantics="scalar", want_pdqf=True, want_buf1=True)
    plain = oracle.luma(imgs) if imgs.ndim == 4 else imgs.astype(np.float32)
    h, q, t, p, b = oracle.hash_batch_reference(plain, semantics="scalar")
    assert np.array_equal(got["buf1"], b)
    assert np.array_equal(got["pdqf"][:, 0], p)
    assert np.array_equal(got["hashes"], h)
    assert np.array_equal(got["quality"], q)
    assert np.array_equal(got["thresholds"], t)
