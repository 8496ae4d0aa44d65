"""2D lattices past the sizes whose step is one launch, so that the two kernels with 32-bit indices run:
FP32 and FP16 with two cells per thread, FP64 accuracy with selects on the load index; against 64-bit
indices (one cell per thread; interior and face kernels), bit for bit.  lbm_time_kernels says which
form a lattice takes, so a size that stops reaching these kernels fails."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Lattice
from lbmgpu.abi import LBM_BCT_CONST, LBM_CELL_SIDE, rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["periodic", "walls", "side"])
@pytest.mark.parametrize("precision,nx,ny", [
    ("fp32", 401, 777), ("fp32", 31, 3701), ("fp32", 33, 3701), ("fp32", 1026, 301), ("fp16", 401, 777),
    ("fp16", 31, 1901), ("fp16", 130, 533), ("fp64x", 257, 130), ("fp64x", 33, 501), ("fp64x", 31, 701),
    ("fp64x", 1000, 64)])
def test_two_kernels_equal_wide(gpu_lib, precision, nx, ny, kind):
    p = rb_params(dim=2, nx=nx, ny=ny, nz=1, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision,
                  periodic_x=kind == "periodic")
    if kind == "side":
        p.cell = LBM_CELL_SIDE
        p.bc_thermal[0], p.bc_thermal[1] = LBM_BCT_CONST, 1
    a, b = Lattice(p), Lattice(p)
    b.set_option(LBM_OPT_WIDE_INDEX, 1)
    for lat in (a, b):
        lat.initial()
        lat.step(37)
    for k in ("f", "g", "T", "u", "v", "Bx_prev", "By_prev", "Fy"):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
    assert a.time_kernels(1)[1] > 0.0
