"""The reciprocal of the fixed arithmetic over its whole range (1/2, 4), its ends among it, against
long double (fixed_recip_check.cpp).

The result is a q60 number of at least 1/4.  The last product of the iteration and its shift each
round by less than one unit of 2^-60, and what the second step leaves of a first residual below 2^-44
is below 2^-88 of the result: 2 * 2^-60 / (1/4) = 2^-57 covers it."""
import os
import subprocess

from test_cpu_fixed import HERE, ROOT, _cxx


def test_reciprocal_to_the_ends_of_its_range(tmp_path):
    cxx, cuda_inc = _cxx()
    exe = str(tmp_path / "recip")
    cmd = [cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "-2d-3d-_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
           "-I", cuda_inc, "-o", exe, os.path.join(HERE, "fixed_recip_check.cpp")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    errors = [float(x) for x in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()]
    assert len(errors) == 3 and max(errors) < 2.0 ** -57, errors
