"""Host paths against a stand-in for the CUDA runtime (tests/fake_cudart.c, no GPU)."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

CREATE = r"""
import ctypes, sys
fake, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2])
lib.ypdq_ctx_destroy.argtypes = [ctypes.c_void_p]
OK, UNSUPPORTED = 0, int(sys.argv[3])

def create(fail_at):
    fake.fake_reset(fail_at)
    h = ctypes.c_void_p()
    return lib.ypdq_ctx_create(0, ctypes.byref(h)), h

st, h = create(0)
made = fake.fake_made()
assert st == OK and made > 30 and fake.fake_live() == made, (st, made, fake.fake_live())
lib.ypdq_ctx_destroy(h)
assert fake.fake_live() == 0
kinds = set()
for k in range(1, made + 1):
    st, h = create(k)
    kind = chr(fake.fake_failed_kind())
    kinds.add(kind)
    if kind == "p":
        assert st == OK and h.value
        lib.ypdq_ctx_destroy(h)
    else:
        assert st != OK and h.value is None
    assert fake.fake_live() == 0, (k, kind, fake.fake_live())
assert kinds == set("hsep"), kinds
fake.fake_attribute(0)  # no shared memory, registers or threads: no hash kernel fits
st, h = create(0)
assert st == UNSUPPORTED and h.value is None and fake.fake_live() == 0, (st, fake.fake_live())
assert fake.fake_wrong_frees() == 0
print("ok")
"""


@pytest.fixture(scope="module")
def fake_cudart(tmp_path_factory):
    cc = shutil.which("gcc") or shutil.which("cc")
    include = "/usr/local/cuda/include"
    if cc is None or not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        pytest.skip("no C compiler or CUDA headers")
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run([cc, "-O1", "-shared", "-fPIC", "-I", include, "-o", so,
                    os.path.join(ROOT, "tests", "fake_cudart.c")], check=True)
    return so


def run_with(fake, script, *args):
    r = subprocess.run([sys.executable, "-c", script, fake, *args], capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, LD_PRELOAD=fake))
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr


def test_failed_creation_leaves_nothing(yp, fake_cudart):
    """ypdq_ctx_create with one of its calls refused: nothing created stays behind, and a device
    without memory pools is no reason to refuse."""
    yp._lib.load()
    run_with(fake_cudart, CREATE, yp._lib.LIB_PATH, str(yp._lib.ERR_UNSUPPORTED))


SCREEN = r"""
import ctypes, sys
import numpy as np
fake, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2])
fake.fake_most_pinned.restype = ctypes.c_size_t
u64, vp = ctypes.c_uint64, ctypes.c_void_p
lib.ypdq_screen_host.argtypes = [vp, vp, vp, ctypes.c_int64, ctypes.c_int, ctypes.c_int,
                                 ctypes.c_int, ctypes.c_uint32, vp, u64, vp, vp, vp]
lib.ypdq_db_wrap.argtypes = [vp, vp, u64, vp]
ctx, db, total = vp(), vp(), u64(7)
assert lib.ypdq_ctx_create(0, ctypes.byref(ctx)) == 0
assert lib.ypdq_db_wrap(ctx, vp(1 << 20), 1000, ctypes.byref(db)) == 0
capacity = 1000
hits = np.zeros(capacity * 16, np.uint8)
images = np.empty((8192, 512, 512), np.uint8)  # never touched
for n in (1, 200, 1024, 2048, 8192):
    fake.fake_reset(0)
    for want_hashes, want_quality in ((1, 1), (1, 0), (0, 1), (0, 0)):
        hashes, quality = np.full((n, 256), 0xAA, np.uint8), np.full((n, 8), 3, np.float32)
        st = lib.ypdq_screen_host(ctx, db, images.ctypes.data, n, 1, 0, 0, 31, hits.ctypes.data,
                                  capacity, ctypes.addressof(total),
                                  hashes.ctypes.data if want_hashes else None,
                                  quality.ctypes.data if want_quality else None)
        assert st == 0 and total.value == 0, (st, total.value)
        assert (hashes == (0 if want_hashes else 0xAA)).all()
        assert (quality == (0 if want_quality else 3)).all()
    assert fake.fake_most_pinned() <= 64 + 16 * capacity + (512 << 10), (n, fake.fake_most_pinned())
print("ok")
"""


def test_screening_pins_no_memory_per_image(yp, fake_cudart):
    """What ypdq_screen_host keeps page-locked grows with the hit capacity alone: the hashes and
    qualities of many images go straight to the caller, and arrive in every combination."""
    yp._lib.load()
    run_with(fake_cudart, SCREEN, yp._lib.LIB_PATH)
