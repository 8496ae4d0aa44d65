"""The one-launch 2D step (FP32, FP16; blocks of four and eight rows of 64 cells) against one cell per
thread (64-bit indices force it), bit for bit: lattices that one block covers, that end on, before
and after the edge of a block, periodic and walled, and one whose state does not fit L2.  Members
of a batch are held to the same."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Ensemble, Lattice
from lbmgpu.abi import LBM_BCT_CONST, LBM_CELL_SIDE, rb_params

pytestmark = pytest.mark.gpu
FIELDS = ("f", "g", "T", "u", "v", "Bx_prev", "By_prev", "Fy")


def params(nx, ny, precision, kind):
    p = rb_params(dim=2, nx=nx, ny=ny, nz=1, Ra=1e5, U=0.05, noise_amp=1e-2, precision=precision,
                  periodic_x=kind == "periodic")
    if kind == "side":
        p.cell = LBM_CELL_SIDE
        p.bc_thermal[0], p.bc_thermal[1] = LBM_BCT_CONST, 1
    return p


def alone(p, steps):
    lat = Lattice(p)
    lat.set_option(LBM_OPT_WIDE_INDEX, 1)
    lat.initial()
    lat.step(steps)
    return lat


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("kind", ["periodic", "walls", "side"])
@pytest.mark.parametrize("nx,ny", [(5, 5), (62, 5), (63, 6), (64, 7), (65, 8), (124, 9), (125, 13), (186, 33),
                                   (700, 203)])
def test_tiles_equal_one_cell(gpu_lib, precision, kind, nx, ny):
    p = params(nx, ny, precision, kind)
    a, b = Lattice(p), alone(p, 37)
    a.initial()
    a.step(20)
    a.step(17)
    for k in FIELDS:
        assert np.array_equal(a.get_state(k), b.get_state(k)), k


def test_state_beyond_l2(gpu_lib):
    p = params(2047, 1100, "fp32", "walls")
    a, b = Lattice(p), alone(p, 7)
    a.initial()
    a.step(7)
    for k in FIELDS:
        assert np.array_equal(a.get_state(k), b.get_state(k)), k


def test_batch_members(gpu_lib):
    ps = [params(nx, ny, "fp32", kind) for nx, ny, kind in
          ((5, 5, "walls"), (64, 8, "periodic"), (63, 33, "side"), (130, 65, "walls"), (700, 203, "periodic"))]
    lats, ens = [Lattice(p) for p in ps], Ensemble()
    for lat in lats:
        lat.initial()
        lat.step(1)
        ens.add(lat)
    ens.step(19)
    ens.step(16)
    ens.sync()
    for p, lat in zip(ps, lats):
        b = alone(p, 36)
        for k in FIELDS:
            assert np.array_equal(lat.get_state(k), b.get_state(k)), (p.nx, p.ny, k)
