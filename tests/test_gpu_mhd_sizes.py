"""The MHD stage kernels at the edges of their 32 x 8 tiles: every remainder of
nx by 4 (rows are padded to 16 bytes on the device, and the last tile's halo
box starts further left), one to nine columns in the last tile, grids with and
without interior tiles, halos that wrap.

Tolerance: one iteration from a random state agrees with the oracle to 1e-12
relative L2 per field in FP64 (rounding of about 1e-15 after five stages), and
the precision form with the plain form to 1e-5 (24-bit rounding, 6e-8 per
operation)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from sparc2_b200 import Simulation, abi
from sparc2_b200 import workloads as W
from tests import cases

pytestmark = pytest.mark.gpu

MM = W.MM
# nx, ny, nz, periodic
SIZES = [(22, 22, 24, False), (33, 25, 31, False), (65, 40, 26, False), (97, 41, 33, False),
         (98, 33, 24, False), (99, 30, 26, False), (100, 33, 24, False), (37, 29, 24, True),
         (97, 40, 26, True), (22, 23, 24, True)]


def case(nx, ny, nz, periodic):
    lx, ly = 0.4 * nx * MM, 0.4 * ny * MM
    p = W.base_params(nx, ny, nz, magnetic=2, periodic=periodic, hpml=not periodic, xlength=lx,
                      ylength=ly, timestep=0.5, t_z=1.0, t_xy=1.0, npml=8, blocks=(2, 2, 2))
    bg = W.fluxtube_background(nx, ny, nz, lx, ly, -6.0, 1.0, R0_mm=2.0, periodic=periodic)
    return p, bg, W.psr_source(W.psr_table(p, 20, 7))


def one(sim, a0, psi0):
    sim.set_state(a0, psi0)
    sim.step(2)
    return sim


@pytest.mark.parametrize("size", SIZES)
def test_tile_edges(size):
    p, bg, src = case(*size)
    sim, orc = Simulation(p, bg, src), oracle.Oracle(p, bg, src)
    a0, psi0 = cases.random_state(sim, seed=3)
    one(orc, a0, psi0)
    one(sim, a0, psi0)
    # the norm without allocation reads the padded rows
    norm = C.c_double()
    assert sim.lib.sparc_ke_norm_noalloc(sim.h, C.byref(norm)) == abi.SPARC_OK
    d, _ = sim.diagnostics()
    assert abs(norm.value - d.ke_norm) <= 1e-12 * d.ke_norm
    for s in (sim, orc):
        s.filter_vars(2)
    a, psi = sim.get_state()
    ra, rpsi = orc.get_state()
    for l in range(sim.V):
        assert cases.rel_l2(a[l], ra[l]) <= 1e-12
    assert cases.rel_l2(psi, rpsi) <= 1e-12
    for name in ("rho0", "curlboz", "source_damp"):
        assert cases.rel_l2(sim.coeff(name), orc.coeff(name)) <= 1e-13
    # neither the state nor (multiples of four layers) the norm depends on
    # the chunk extent
    for zc in (11, 16):
        b = Simulation(p, bg, src)
        b.set_zchunk(zc)
        one(b, a0, psi0)
        if zc == 16:
            assert b.diagnostics()[0].ke_norm == d.ke_norm
        b.filter_vars(2)
        assert np.array_equal(b.get_state()[0], a)
    p32, bg, src = case(*size)
    p32.precision = abi.SPARC_FP32
    low = one(Simulation(p32, bg, src), a0, psi0)
    low.filter_vars(2)
    la, _ = low.get_state()
    for l in range(sim.V):
        assert cases.rel_l2(la[l], a[l]) <= 1e-5
