"""LBM_OPT_ROWS given without LBM_OPT_PAIRS: the same values as without it in every storage form and
dimension, whatever launches it selects."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_ROWS, Lattice
from lbmgpu.abi import rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("dim,nx,ny,nz", [(2, 66, 19, 1), (2, 67, 19, 1), (3, 34, 9, 7)])
def test_rows_alone(gpu_lib, precision, dim, nx, ny, nz):
    p = rb_params(dim=dim, nx=nx, ny=ny, nz=nz, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision, periodic_x=True)
    a, b = Lattice(p), Lattice(p)
    a.set_option(LBM_OPT_ROWS, 1)
    for lat in (a, b):
        lat.initial()
        lat.step(37)
    for k in ("f", "g", "T", "u", "v"):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
