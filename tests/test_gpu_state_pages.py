"""Fields read into host arrays below, at and above the sizes whose pages are brought in by one and
by several threads, at addresses off the page boundary, with their neighbours left alone."""
import ctypes as C

import numpy as np
import pytest

from lbmgpu import Lattice
from lbmgpu.abi import FIELDS, rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 8), (1000, 500), (1024, 520), (2050, 1025)])
@pytest.mark.parametrize("offset", [0, 3])
def test_field_into_fresh_array(gpu_lib, nx, ny, offset):
    lat = Lattice(rb_params(dim=2, nx=nx, ny=ny, nz=1, Ra=1e5, U=0.05, noise_amp=0.0))
    lat.initial()
    n = nx * ny
    T = np.random.default_rng(5).random(n)
    lat.set_state("T", T.reshape(ny, nx))
    got = np.zeros(n + 8)  # fresh pages, none of them written yet
    got[:offset], got[offset + n:] = -1.0, -2.0
    p = got[offset:].ctypes.data_as(C.POINTER(C.c_double))
    assert gpu_lib.lbm_get_state(lat._h, FIELDS["T"], p, n) == 0
    assert np.array_equal(got[offset:offset + n], T)
    assert (got[:offset] == -1.0).all() and (got[offset + n:] == -2.0).all()
    lat.close()
