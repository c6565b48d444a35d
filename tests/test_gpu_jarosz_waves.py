"""The Jarosz kernel turns its warps' parts, and delays CTAs, by how many waves a batch makes:
batch sizes on both sides of each rule give the hashes that each image has by itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JAROSZ = 0x200


@pytest.mark.parametrize("sms3,extra", [(1, 0), (1, 1), (1, "sm"), (1, "sm+1"), (3, 0), (3, 1)])
def test_waves(ctx, yp, sms3, extra):
    sms = ctx.num_sms
    n = 3 * sms * sms3 + {"sm": sms, "sm+1": sms + 1}.get(extra, extra)
    few = np.random.default_rng(4).integers(0, 256, (7, 512, 512), dtype=np.uint8)
    d_img = ctx.alloc(n << 18)
    for i in range(0, n, 7):
        d_img.upload(few[:n - i], offset=i << 18)
    d_h, d_t = ctx.alloc(n * 256), ctx.alloc(n * 32)
    yp.core.hash_batch_device(ctx, d_img, n, yp._lib.INPUT_U8, d_hashes=d_h, d_thresholds=d_t,
                              dct=JAROSZ)
    ctx.sync()
    h, t = d_h.download((n, 8, 32), np.uint8), d_t.download((n, 8), np.float32)
    one = yp.core.hash_batch(ctx, few, dct=JAROSZ)
    assert np.array_equal(h, one["hashes"][np.arange(n) % 7])
    assert np.array_equal(t, one["thresholds"][np.arange(n) % 7])
