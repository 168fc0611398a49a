"""The quiet stage kernels at the edges of their 32 x 8 tiles and z chunks:
grids smaller than a tile, one to five columns in the last tile (whose halo
origin moves down on non-periodic axes), ragged periodic grids that wrap more
than once within a tile, and chunks shorter than the window.

Tolerance: one iteration from a random state agrees with the oracle to
1e-12 relative L2 per field in FP64 (the derivative sums differ by a few
rounding errors of 1.1e-16 per term, about 1e-15 after five stages), and the
precision form with the plain form to 1e-5 (24-bit rounding, 6e-8 per
operation)."""
import numpy as np
import pytest

import oracle
from sparc2_b200 import Simulation, abi
from sparc2_b200 import workloads as W
from tests import cases

pytestmark = pytest.mark.gpu

MM = W.MM
# nx, ny, nz, periodic, magnetic
SIZES = [(22, 22, 24, True, 0), (33, 25, 31, True, 0), (64, 40, 44, True, 0),
         (33, 22, 24, False, 0), (37, 29, 40, False, 1), (34, 41, 33, False, 1),
         (23, 33, 26, True, 1)]


def case(nx, ny, nz, periodic, magnetic):
    lx, ly = 0.4 * nx * MM, 0.4 * ny * MM
    p = W.base_params(nx, ny, nz, magnetic=magnetic, periodic=periodic, hpml=not periodic,
                      xlength=lx, ylength=ly, timestep=0.5, t_z=1.0, t_xy=1.0, npml=8,
                      blocks=(2, 2, 2))
    if magnetic:
        bg = dict(W.fluxtube_background(nx, ny, nz, lx, ly, -6.0, 1.0, R0_mm=2.0,
                                        periodic=periodic), bx0=None, by0=None, bz0=None)
    else:
        bg = W.quiet_background(nx, ny, nz, -8.0, 1.0)
    src = W.pulse_source(px=0.4 * lx, py=0.5 * ly, pz=-1.0 * MM, sr=1.0 * MM, sz=0.5 * MM,
                         t1=10.0, st=5.0, direction=1 + (nx + ny) % 3)
    return p, bg, src


@pytest.mark.parametrize("size", SIZES)
def test_tile_edges(size):
    p, bg, src = case(*size)
    sim, orc = Simulation(p, bg, src), oracle.Oracle(p, bg, src)
    a0, psi0 = cases.random_state(sim, seed=3)
    for s in (sim, orc):
        s.set_state(a0, psi0)
        s.step(1)
        s.filter_vars(1)
    a, psi = sim.get_state()
    ra, rpsi = orc.get_state()
    for l in range(sim.V):
        assert cases.rel_l2(a[l], ra[l]) <= 1e-12
    assert cases.rel_l2(psi, rpsi) <= 1e-12
    # the chunk extent does not change the result
    for zc in (11, 16):
        b = Simulation(p, bg, src)
        b.set_state(a0, psi0)
        b.set_zchunk(zc)
        b.step(1)
        b.filter_vars(1)
        assert np.array_equal(b.get_state()[0], a)
    # the precision form against the plain form
    p32, bg, src = case(*size)
    p32.precision = abi.SPARC_FP32
    low = Simulation(p32, bg, src)
    low.set_state(a0, psi0)
    low.step(1)
    low.filter_vars(1)
    la, _ = low.get_state()
    for l in range(sim.V):
        assert cases.rel_l2(la[l], a[l]) <= 1e-5
