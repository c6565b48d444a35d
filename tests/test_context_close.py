"""A context whose construction fails half-way gives its handle back (fake library, no GPU)."""
import gc

import pytest


class FakeLib:
    destroyed = 0

    def ypdq_ctx_create(self, device, out):
        out._obj.value = 1
        return 0

    def ypdq_device_info(self, handle, sms, ctas):
        return 1

    def ypdq_last_error(self):
        return b"no device info"

    def ypdq_ctx_destroy(self, handle):
        self.destroyed += 1
        return 0


def test_failed_construction_destroys_the_context(yp, monkeypatch):
    fake = FakeLib()
    monkeypatch.setattr(yp._lib, "load", lambda *a: fake)
    with pytest.raises(Exception) as err:
        yp.Context(0)
    del err
    gc.collect()
    assert fake.destroyed == 1
