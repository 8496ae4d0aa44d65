"""Pages of a fresh host array brought in by a few threads: each page once, none outside the array, and none
from a thread on another memory node than the caller's, where it would land (pages_check.cpp)."""
import os
import subprocess

import pytest

from test_cpu_fixed import HERE, ROOT, _cxx


@pytest.mark.parametrize("helpers", ["near", "far"])
def test_pages_land_with_the_caller(tmp_path, helpers):
    cxx, _ = _cxx()
    exe = str(tmp_path / "pages")
    cmd = [cxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "-2d-3d-_gb300", "csrc"), "-Wl,--wrap=madvise",
           "-Wl,--wrap=getcpu", "-o", exe, os.path.join(HERE, "pages_check.cpp")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, helpers], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
