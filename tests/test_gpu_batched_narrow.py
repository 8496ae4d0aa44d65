"""2D FP32 members of a batch whose one-launch tiles would own little of what they hold: narrower than a
block, a little wider than one, and mixed with members of the other kind, against the same lattices
alone with 64-bit indices (one cell per thread), bit for bit."""
import numpy as np
import pytest

from lbmgpu import LBM_OPT_WIDE_INDEX, Ensemble, Lattice
from lbmgpu.abi import rb_params

pytestmark = pytest.mark.gpu
FIELDS = ("f", "g", "T", "u", "v", "Bx_prev", "By_prev", "Fy")


@pytest.mark.parametrize("shapes", [
    [(8, 4001), (8, 4001), (66, 900)],              # more than two waves of such blocks: two launches a step
    [(5, 7), (70, 20), (33, 64)],                   # few of them: one
    [(8, 8001), (66, 900), (130, 65), (700, 203)],  # both lists in one step
])
def test_narrow_members(gpu_lib, shapes):
    ps = [rb_params(dim=2, nx=nx, ny=ny, nz=1, Ra=1e5, U=0.05, noise_amp=1e-2, precision="fp32", periodic_x=n % 2 == 0)
          for n, (nx, ny) in enumerate(shapes)]
    lats, ens = [Lattice(p) for p in ps], Ensemble()
    for lat in lats:
        lat.initial()
        lat.step(1)
        ens.add(lat)
    ens.step(33)
    ens.step(2)
    ens.sync()
    for p, lat in zip(ps, lats):
        b = Lattice(p)
        b.set_option(LBM_OPT_WIDE_INDEX, 1)
        b.initial()
        b.step(36)
        for k in FIELDS:
            assert np.array_equal(lat.get_state(k), b.get_state(k)), (p.nx, p.ny, k)
