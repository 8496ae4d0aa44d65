"""The largest lattices whose kernels take 32-bit indices: no index, used or selected away, leaves
32 bits (index_range_check.cpp under the undefined-behaviour sanitizer)."""
import os
import subprocess

from test_cpu_fixed import HERE, ROOT, _cxx


def test_largest_narrow_lattices_stay_in_32_bits(tmp_path):
    cxx, cuda_inc = _cxx()
    exe = str(tmp_path / "index_range")
    cmd = [cxx, "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I",
           os.path.join(ROOT, "-2d-3d-_gb300", "csrc"), "-I", os.path.join(ROOT, "include"), "-I", cuda_inc, "-o", exe,
           os.path.join(HERE, "index_range_check.cpp")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
