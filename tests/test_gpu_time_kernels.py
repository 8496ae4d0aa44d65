"""lbm_time_kernels times the launches that lbm_step makes: one per step on 2D lattices that take the
one-launch form (all of it in the first figure), two on the others; its steps are ordinary steps."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Lattice
from lbmgpu.abi import rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nx,ny,wide,launches", [
    ("fp32", 64, 40, 0, 1), ("fp32", 401, 300, 0, 1), ("fp32", 401, 777, 0, 2), ("fp32", 64, 40, 1, 2),
    ("fp16", 64, 40, 0, 1), ("fp16", 401, 300, 0, 2), ("fp64x", 64, 48, 0, 1), ("fp64x", 256, 128, 0, 2),
    ("fp64x", 64, 48, 1, 2), ("fp64", 64, 48, 0, 2)])
def test_times_what_runs(gpu_lib, precision, nx, ny, wide, launches):
    p = rb_params(dim=2, nx=nx, ny=ny, nz=1, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision)
    a, b = Lattice(p), Lattice(p)
    for lat in (a, b):
        lat.set_option(LBM_OPT_WIDE_INDEX, wide)
        lat.initial()
        lat.step(3)
    flow, thermal = a.time_kernels(3)
    assert flow > 0.0 and (thermal == 0.0) == (launches == 1)
    a.step(5)
    b.step(8)
    assert a.itc == b.itc == 11
    for k in ("f", "g", "T", "u", "v"):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
