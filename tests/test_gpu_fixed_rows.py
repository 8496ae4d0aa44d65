"""The fixed arithmetic's kernels with 32-bit indices (boundary rules as selects on the load index)
against its interior and face kernels (64-bit indices force those), bit for bit: row lengths at
the edges of a warp and of a block, lattices that end inside a block, walls and periodic faces."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Lattice
from lbmgpu.abi import rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nx,ny,nz,periodic", [
    (2, 5, 5, 1, True), (2, 31, 6, 1, False), (2, 33, 7, 1, True), (2, 64, 9, 1, True), (2, 97, 5, 1, False),
    (2, 129, 13, 1, True), (2, 1025, 1024, 1, False), (3, 5, 5, 2, False), (3, 32, 5, 3, True), (3, 65, 7, 5, False),
    (3, 96, 8, 4, True), (3, 130, 6, 5, False), (3, 105, 100, 101, True)])
def test_index_kernels_equal_interior_and_face_kernels(gpu_lib, dim, nx, ny, nz, periodic):
    p = rb_params(dim=dim, nx=nx, ny=ny, nz=nz, Ra=1e5, noise_amp=1e-2, precision="fp64x", periodic_x=periodic)
    if dim == 3 and periodic:
        p.bc_flow[2], p.bc_thermal[2] = 1, 2
    a, b = Lattice(p), Lattice(p)
    b.set_option(LBM_OPT_WIDE_INDEX, 1)
    for lat in (a, b):
        lat.initial()
        lat.step(37)
    for k in ("f", "g", "T", "u", "v", "Bx_prev", "By_prev") + (("w", "Bz_prev") if dim == 3 else ("Fy",)):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
    a.close()
    b.close()
