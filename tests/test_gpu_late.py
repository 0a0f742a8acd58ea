"""A CTA whose wait gave up tells the others: the teams of the slice-form CG,
driven by a small program of their own (tests/cpp/late_test.cu).  The solve
itself can only reach this after a wait of two seconds has run out."""
import os
import subprocess

import pytest

from monolish_b200 import build

pytestmark = pytest.mark.gpu


def test_every_cta_learns_of_a_late_one(cuda, tmp_path):
    exe = str(tmp_path / "late_test")
    subprocess.run([build.NVCC, *build.ARCH, "-O2", "-std=c++17", "-I", build.CSRC, "-I",
                    os.path.join(build.ROOT, "include"), "-o", exe,
                    os.path.join(build.ROOT, "tests", "cpp", "late_test.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    lines = [line.split() for line in r.stdout.splitlines()]
    assert r.returncode == 0 and len(lines) == 10, r.stdout
    assert all(ok == "1" for _, _, ok in lines), r.stdout
