"""The one-launch 2D step of the fixed arithmetic (small lattices) against the two kernels with 64-bit
indices, bit for bit: lattices that one block covers, that end on, before and after the edge of a
block, periodic and walled; calls that leave an odd number of steps, and a load in between."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Lattice
from lbmgpu.abi import LBM_BCT_CONST, LBM_CELL_SIDE, rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["periodic", "walls", "side"])
@pytest.mark.parametrize("nx,ny", [(5, 5), (30, 6), (31, 7), (32, 5), (33, 8), (60, 9), (61, 48), (128, 64)])
def test_tiles_equal_two_kernels(gpu_lib, kind, nx, ny):
    p = rb_params(dim=2, nx=nx, ny=ny, nz=1, Ra=1e5, U=0.05, noise_amp=1e-2, precision="fp64x",
                  periodic_x=kind == "periodic")
    if kind == "side":
        p.cell = LBM_CELL_SIDE
        p.bc_thermal[0], p.bc_thermal[1] = LBM_BCT_CONST, 1
    a, b = Lattice(p), Lattice(p)
    b.set_option(LBM_OPT_WIDE_INDEX, 1)
    for lat in (a, b):
        lat.initial()
        for n in (1, 2, 38):
            lat.step(n)
            lat.calNuRe()
        lat.set_state("g", lat.get_state("g"))
        lat.step(7)
    for k in ("f", "g", "T", "u", "v", "rho", "Bx_prev", "By_prev", "Fy"):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
    a.close()
    b.close()
