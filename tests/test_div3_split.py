"""The two-operation x / 3 of the Jarosz kernel's byte images (div3, csrc/jarosz.cu) equals
IEEE division for every float from 2^-120 on (tests/div3_split_exhaustive.c); the sums it
divides are 0 or larger than that."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_div3_split_exhaustive(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    exe = str(tmp_path / "div3_split_exhaustive")
    subprocess.run([cc, "-O2", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "div3_split_exhaustive.c"), "-lm", "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
