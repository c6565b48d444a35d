"""ypdq_ctx_create on a machine that refuses one of its calls, with a stand-in for the CUDA
runtime (tests/fake_cudart.c, no GPU): nothing created stays behind, and a device without memory
pools is no reason to refuse."""
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
    yp._lib.load()
    run_with(fake_cudart, CREATE, yp._lib.LIB_PATH, str(yp._lib.ERR_UNSUPPORTED))
