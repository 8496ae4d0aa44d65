"""The step with two cells per thread (32 apart, packed FP32 arithmetic) against one cell per
thread (64-bit indices force it), bit for bit: rows shorter than, equal to and longer than the
distance of the two cells, lattices that end inside a warp, walls and periodic faces."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_PAIRS, LBM_OPT_WIDE_INDEX, Lattice
from lbmgpu.abi import LBM_BCT_CONST, LBM_CELL_SIDE, rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("dim,nx,ny,nz,kind", [
    (2, 5, 5, 1, "periodic"), (2, 31, 6, 1, "walls"), (2, 32, 7, 1, "periodic"), (2, 33, 65, 1, "side"),
    (2, 130, 33, 1, "walls"), (3, 5, 5, 2, "walls"), (3, 7, 6, 5, "periodic"), (3, 32, 5, 3, "side"),
    (3, 33, 9, 4, "periodic"), (3, 64, 5, 5, "walls"), (3, 65, 7, 9, "side")])
def test_duo_equals_one_cell(gpu_lib, precision, dim, nx, ny, nz, kind):
    p = rb_params(dim=dim, nx=nx, ny=ny, nz=nz, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision,
                  periodic_x=kind == "periodic")
    if kind == "periodic" and dim == 3:
        p.bc_flow[2], p.bc_thermal[2] = 1, 2
    if kind == "side":
        p.cell = LBM_CELL_SIDE
        p.bc_thermal[0], p.bc_thermal[1] = LBM_BCT_CONST, 1
    a, b = Lattice(p), Lattice(p)
    b.set_option(LBM_OPT_WIDE_INDEX, 1)
    for lat in (a, b):
        lat.set_option(LBM_OPT_PAIRS, 0)
        lat.initial()
        lat.step(37)
    for k in ("f", "g", "T", "u", "v", "Bx_prev", "By_prev") + (("w", "Bz_prev") if dim == 3 else ("Fy",)):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
    a.close()
    b.close()
