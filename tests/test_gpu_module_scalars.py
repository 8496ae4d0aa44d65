"""Reading scalar fields and diagnostics leaves the module populations of the last read alone, and a
later read of the populations, a state load or a stage of the loop brings them up to date: the
sequence of reads does not change what is read."""
import numpy as np
import pytest

from lbmgpu import Lattice
from lbmgpu.abi import rb_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp64x", "fp32", "fp16"])
@pytest.mark.parametrize("dim,nx,ny,nz,periodic", [(2, 33, 17, 1, True), (3, 20, 9, 7, False), (3, 34, 6, 5, True)])
def test_reads_in_any_order(gpu_lib, precision, dim, nx, ny, nz, periodic):
    p = rb_params(dim=dim, nx=nx, ny=ny, nz=nz, Ra=1e5, noise_amp=1e-2, precision=precision, periodic_x=periodic)
    a, b = Lattice(p), Lattice(p)
    for lat in (a, b):
        lat.initial()
        lat.step(5)
    fields = ["T", "u", "v", "rho", "f", "g"]
    one = {k: a.get_state(k) for k in ["f", "g", "T", "u", "v", "rho"]}
    nu = a.calNuRe()
    assert b.calNuRe() == nu
    for k in fields:
        assert np.array_equal(b.get_state(k), one[k]), k
    for lat in (a, b):
        lat.step(3)
    a.get_state("f")
    for lat in (a, b):  # a load after scalar reads continues from up-to-date populations
        T = lat.get_state("T")
        lat.set_state("T", T)
        lat.step(4)
    for k in fields:
        assert np.array_equal(a.get_state(k), b.get_state(k)), k
    a.close()
    b.close()
