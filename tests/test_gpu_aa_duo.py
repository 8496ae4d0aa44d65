"""The in-place sweeps with two cells per thread (walls on every face) against one cell per thread
(64-bit indices force it), bit for bit: rows around the distance of the two cells, lattices that
end inside a warp, constant-temperature floors and side walls, populations loaded mid-run."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Lattice
from lbmgpu.abi import LBM_BCT_CONST, LBM_CELL_SIDE, rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("dim,nx,ny,nz,side", [
    (2, 5, 5, 1, False), (2, 33, 6, 1, True), (2, 130, 9, 1, False), (3, 6, 5, 3, True), (3, 32, 5, 4, False),
    (3, 65, 7, 5, False)])
def test_aa_duo_equals_one_cell(gpu_lib, precision, dim, nx, ny, nz, side):
    p = rb_params(dim=dim, nx=nx, ny=ny, nz=nz, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision, pattern="AA",
                  periodic_x=False)
    if side:
        p.cell = LBM_CELL_SIDE
        p.bc_thermal[0], p.bc_thermal[1] = LBM_BCT_CONST, 1
    a, b = Lattice(p), Lattice(p)
    b.set_option(LBM_OPT_WIDE_INDEX, 1)
    for lat in (a, b):
        lat.initial()
        for n in (1, 2, 37):
            lat.step(n)
        lat.set_state("g", lat.get_state("g"))  # the two arrays run one layout apart from here
        lat.step(6)
    for k in ("f", "g", "T", "u", "v", "Bx_prev", "By_prev") + (("w", "Bz_prev") if dim == 3 else ("Fy",)):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
    a.close()
    b.close()
