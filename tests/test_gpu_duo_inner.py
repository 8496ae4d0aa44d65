"""Warps of the two-cells-per-thread step that lie off every face, on rows with an x face and on
face rows take different pulls; rows long enough for all three, against one cell per thread
(64-bit indices force it), bit for bit."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Lattice
from lbmgpu.abi import rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("pattern,periodic", [("AB", True), ("AB", False), ("AA", False)])
@pytest.mark.parametrize("dim,nx,ny,nz", [(2, 66, 9, 1), (2, 193, 7, 1), (3, 128, 6, 5), (3, 200, 7, 6)])
def test_inner_warps_equal_one_cell(gpu_lib, precision, pattern, periodic, dim, nx, ny, nz):
    p = rb_params(dim=dim, nx=nx, ny=ny, nz=nz, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision,
                  pattern=pattern, periodic_x=periodic)
    a, b = Lattice(p), Lattice(p)
    b.set_option(LBM_OPT_WIDE_INDEX, 1)
    for lat in (a, b):
        lat.initial()
        lat.step(37)
    for k in ("f", "g", "T", "u", "v", "Bx_prev", "By_prev") + (("w", "Bz_prev") if dim == 3 else ("Fy",)):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
    a.close()
    b.close()
