"""The steady-state FP32 flow collision adds the force to the momentum and nothing else: over 400,000
random states the mean relative gain beyond it stays below 2^-28 (steady_momentum_check.cpp).

One constant that is half an FP32 unit off 1 gives every state the same gain of up to 2^-25 in each
step.  What rounding leaves is of either sign: 20 to 30 roundings of 2^-25 of a population, and a
population is of the momentum's own size, give each state about 2^-22, so the mean of 400,000
about 4e-10, a ninth of the bound.  Mass likewise, absolute (populations of about 1e-2)."""
import os
import subprocess

from test_cpu_fixed import HERE, ROOT, _cxx


def test_collision_conserves_momentum_in_the_mean(tmp_path):
    cxx, cuda_inc = _cxx()
    exe = str(tmp_path / "momentum")
    cmd = [cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "-2d-3d-_gb300", "csrc"), "-I",
           os.path.join(ROOT, "include"), "-I", cuda_inc, "-o", exe, os.path.join(HERE, "steady_momentum_check.cpp")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [line.split() for line in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 16
    for dim, tau, force, gain, mass in rows:
        assert abs(float(gain)) < 2.0 ** -28 and abs(float(mass)) < 2.0 ** -28, (dim, tau, force, gain, mass)
