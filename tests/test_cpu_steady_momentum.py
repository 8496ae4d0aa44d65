"""The steady-state FP32 flow collision conserves momentum at least as well as the moment-space form that it
stands for: over 400,000 random states the mean relative gain of either (steady_momentum_check.cpp).

A constant that is half an FP32 unit off gives every state the same gain of up to 2^-25 in each step, and
a step's worth of it adds up over a run.  What rounding leaves else is of either sign: 20 to 30 roundings
of 2^-25 of a population, and a population is of the momentum's own size, give each state about 2^-22, so
the mean of 400,000 about 4e-10, which is allowed on top.  Mass: below that, absolute."""
import os
import subprocess

from test_cpu_fixed import HERE, ROOT, _cxx

MEAN = 4e-10


def test_collision_gains_no_more_momentum_than_the_moment_form(tmp_path):
    cxx, cuda_inc = _cxx()
    exe = str(tmp_path / "momentum")
    cmd = [cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "-2d-3d-_gb300", "csrc"), "-I",
           os.path.join(ROOT, "include"), "-I", cuda_inc, "-o", exe, os.path.join(HERE, "steady_momentum_check.cpp")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [line.split() for line in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 8
    for dim, tau, moment, steady, mass in rows:
        assert abs(float(steady)) < abs(float(moment)) + MEAN and abs(float(mass)) < MEAN, (dim, tau, moment, steady, mass)
