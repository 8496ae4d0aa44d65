"""LBM_OPT_WIDE_INDEX selects the kernels of lattices too large for 32-bit indices.  Those of the plain
FP64 step, of the module arrays' rebuild and of a batch, against the 32-bit ones, bit for bit."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Ensemble, Lattice
from lbmgpu.abi import rb_params

pytestmark = pytest.mark.gpu
SHAPES = [(2, 5, 5, 1, True), (2, 130, 33, 1, False), (3, 6, 5, 2, False), (3, 33, 9, 5, True), (3, 65, 7, 4, False)]


def params(dim, nx, ny, nz, periodic, precision, pattern="AB"):
    p = rb_params(dim=dim, nx=nx, ny=ny, nz=nz, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision, pattern=pattern,
                  periodic_x=periodic)
    if periodic and dim == 3:
        p.bc_flow[2], p.bc_thermal[2] = 1, 2
    return p


def fields(dim):
    return ("f", "g", "T", "u", "v", "rho", "Bx_prev", "By_prev") + (("w", "Bz_prev") if dim == 3 else ("Fy",))


@pytest.mark.parametrize("dim,nx,ny,nz,periodic", SHAPES)
def test_plain_fp64_step(gpu_lib, dim, nx, ny, nz, periodic):
    p = params(dim, nx, ny, nz, periodic, "fp64")
    a, b = Lattice(p), Lattice(p)
    b.set_option(LBM_OPT_WIDE_INDEX, 1)
    for lat in (a, b):
        lat.initial()
        lat.step(37)
    for k in fields(dim):
        assert np.array_equal(a.get_state(k), b.get_state(k)), k


@pytest.mark.parametrize("precision,pattern", [("fp64", "AB"), ("fp64x", "AB"), ("fp32", "AB"), ("fp32", "AA"),
                                               ("fp16", "AB"), ("fp16", "AA")])
@pytest.mark.parametrize("dim,nx,ny,nz,periodic", SHAPES)
def test_rebuild_of_the_module_arrays(gpu_lib, precision, pattern, dim, nx, ny, nz, periodic):
    p = params(dim, nx, ny, nz, periodic, precision, pattern)
    a, b = Lattice(p), Lattice(p)
    for steps in (8, 3):  # either layout of the in-place arrays
        for lat in (a, b):
            lat.set_option(LBM_OPT_WIDE_INDEX, 0)
            lat.initial()
            lat.step(steps)
        b.set_option(LBM_OPT_WIDE_INDEX, 1)
        assert a.calNuRe() == b.calNuRe()
        for k in fields(dim):
            assert np.array_equal(a.get_state(k), b.get_state(k)), k


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_batch(gpu_lib, precision):
    ps = [params(*s, precision) for s in SHAPES]
    lats, ens = [Lattice(p) for p in ps], Ensemble()
    for n, lat in enumerate(lats):
        lat.set_option(LBM_OPT_WIDE_INDEX, n % 2)
        lat.initial()
        lat.step(1)
        ens.add(lat)
    ens.step(35)
    for n, lat in enumerate(lats):  # members change their form while they are in the ensemble
        lat.set_option(LBM_OPT_WIDE_INDEX, 1 - n % 2)
    ens.step(6)
    ens.configure(block=256, tile_cells=1024)
    ens.step(3)
    ens.sync()
    for s, p, lat in zip(SHAPES, ps, lats):
        b = Lattice(p)
        b.initial()
        b.step(45)
        for k in fields(s[0]):
            if k != "rho":
                assert np.array_equal(lat.get_state(k), b.get_state(k)), (s, k)
