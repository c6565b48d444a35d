"""The Jarosz filter on infinite, NaN and very large pixels: the one-kernel path (32 images) gives
the same compressed image and DCT, bit for bit but for a NaN's payload, as the planes do for the
same images (fewer than 32), which follow the reference's filter step by step; and the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JAROSZ = 0x200


def test_both_paths_and_the_oracle(ctx, yp, oracle):
    rng = np.random.default_rng(21)
    imgs = rng.random((8, 512, 512), dtype=np.float32) * 255
    places = [(0, 0), (1, 511), (2, 3), (255, 256), (509, 510), (511, 511), (33, 64), (100, 130)]
    values = [np.inf, -np.inf, np.nan, np.inf, np.nan, -np.inf, 3e38, -3e38]
    for img, (r, c), v in zip(imgs, places, values):
        img[r, c] = v
    imgs[3, 255, 258] = -np.inf  # both signs in one window
    imgs[6, 33, 65] = 3e38       # a finite sum that overflows
    few = yp.hash_batch(ctx, imgs, dct=JAROSZ, want_pdqf=True, want_buf1=True)
    many = yp.hash_batch(ctx, np.tile(imgs, (4, 1, 1)), dct=JAROSZ, want_pdqf=True, want_buf1=True)
    _, _, _, p, b = oracle.hash_batch_reference(imgs)
    for got in (few, {k: v[24:] for k, v in many.items()}):
        assert np.array_equal(got["buf1"], b, equal_nan=True)
        assert np.array_equal(got["pdqf"][:, 0], p, equal_nan=True)
    for key in ("hashes", "quality", "thresholds"):
        assert np.array_equal(np.tile(few[key], (4,) + (1,) * (few[key].ndim - 1)), many[key],
                              equal_nan=key != "hashes")


@pytest.mark.parametrize("kind", ["rgb8", "rgba8", "f32"])
@pytest.mark.parametrize("extra", [0, 1, "sm+1"])
def test_waves_of_other_inputs(ctx, yp, kind, extra):
    """The rules by the number of waves, for the inputs besides u8: more than a wave of CTAs, with
    parts by block index and with staggered starts."""
    n = 3 * ctx.num_sms + {"sm+1": ctx.num_sms + 1}.get(extra, extra)
    rng = np.random.default_rng(5)
    shape = (7, 512, 512) + {"rgb8": (3,), "rgba8": (4,), "f32": ()}[kind]
    few = (rng.normal(100, 60, shape).astype(np.float32) if kind == "f32"
           else rng.integers(0, 256, shape, dtype=np.uint8))
    size = few[0].nbytes
    d_img = ctx.alloc(n * size)
    for i in range(0, n, 7):
        d_img.upload(few[:n - i], offset=i * size)
    d_h, d_t = ctx.alloc(n * 256), ctx.alloc(n * 32)
    code = {"f32": 0, "rgb8": 2, "rgba8": 3}[kind]
    yp.core.hash_batch_device(ctx, d_img, n, code, d_hashes=d_h, d_thresholds=d_t, dct=JAROSZ)
    ctx.sync()
    h, t = d_h.download((n, 8, 32), np.uint8), d_t.download((n, 8), np.float32)
    one = yp.core.hash_batch(ctx, few, dct=JAROSZ)
    assert np.array_equal(h, one["hashes"][np.arange(n) % 7])
    assert np.array_equal(t, one["thresholds"][np.arange(n) % 7])
