"""The options of an MHD run on rows that are padded on the device (nx odd, or not
a multiple of four in the precision form): velocity damping, the 7-point filter
and sponges in place of CPML, on grids that wrap and that do not, and the
quiet equations with sponges at the same sizes.

Tolerance: three iterations with a filter event each, from a random state, agree
with the oracle to 1e-11 relative L2 per field in FP64 (as the damping test on
other sizes), and the precision form with the plain form to 1e-5 (24-bit
rounding, 6e-8 per operation)."""
import pytest

import oracle
from sparc2_b200 import Simulation, abi
from sparc2_b200 import workloads as W
from sparc2_b200.batch import Batch
from tests import cases

pytestmark = pytest.mark.gpu

MM = W.MM


def case(nx, ny, nz, option, magnetic=2):
    periodic = option.endswith("periodic")
    sponge = option == "sponge"
    lx, ly = 0.4 * nx * MM, 0.4 * ny * MM
    p = W.base_params(nx, ny, nz, magnetic=magnetic, periodic=periodic,
                      hpml=not periodic and not sponge, xlength=lx, ylength=ly, timestep=0.5,
                      t_z=0.5, t_xy=0.5, npml=8, blocks=(2, 2, 2))
    if option.startswith("damping"):
        p.damping = 1
    if option.startswith("filter7"):
        p.filter_mode_xy = p.filter_mode_z = 2
    if sponge:
        p.use_pml = 0
        p.sp_str, p.sp_length = 20.0, 2.0 * MM
    bg = W.fluxtube_background(nx, ny, nz, lx, ly, -6.0, 1.0, R0_mm=2.0, periodic=periodic)
    if magnetic == 1:
        bg = dict(bg, bx0=None, by0=None, bz0=None)
    return p, bg, W.psr_source(W.psr_table(p, 20, 7))


@pytest.mark.parametrize("size", [(41, 37, 40), (99, 30, 26)])
@pytest.mark.parametrize("option", ["damping", "damping-periodic", "filter7",
                                    "filter7-periodic", "sponge"])
def test_options_against_the_oracle(size, option):
    p, bg, src = case(*size, option)
    sim, orc = Simulation(p, bg, src), oracle.Oracle(p, bg, src)
    a0, psi0 = cases.random_state(sim, seed=13)
    for s in (sim, orc):
        s.set_state(a0, psi0)
        s.run(1, 3)
    a, psi = sim.get_state()
    ra, rpsi = orc.get_state()
    for l in range(sim.V):
        assert cases.rel_l2(a[l], ra[l]) <= 1e-11, l
    if sim.n_psi:
        assert cases.rel_l2(psi, rpsi) <= 1e-11
    if p.damping:
        return
    p32, bg, src = case(*size, option)
    p32.precision = abi.SPARC_FP32
    low = Simulation(p32, bg, src)
    low.set_state(a0, psi0)
    low.run(1, 3)
    la, _ = low.get_state()
    for l in range(sim.V):
        assert cases.rel_l2(la[l], a[l]) <= 1e-5, l


@pytest.mark.parametrize("size", [(41, 37, 40), (33, 25, 31)])
def test_quiet_sponges(size):
    p, bg, src = case(*size, "sponge", magnetic=1)
    sim, orc = Simulation(p, bg, src), oracle.Oracle(p, bg, src)
    a0, psi0 = cases.random_state(sim, seed=13)
    for s in (sim, orc):
        s.set_state(a0, psi0)
        s.run(1, 3)
    for x, y in zip(sim.get_state()[0], orc.get_state()[0]):
        assert cases.rel_l2(x, y) <= 1e-11


def test_batch_of_padded_members_with_the_7_point_filter():
    options = ["filter7", "filter7-periodic", "sponge"]

    def make():
        out = []
        for o in options:
            p, bg, src = case(41, 37, 40, o)
            p.precision = abi.SPARC_FP32
            out.append(Simulation(p, bg, src))
        return out

    sims, alone = make(), make()
    for s in alone:
        s.run(1, 4)
    with Batch(3) as b:
        slots = [b.add(s, 1, 4) for s in sims]
        b.run(4)
        for q in slots:
            b.remove(q)
    for s, t in zip(sims, alone):
        for x, y in zip(s.get_state()[0], t.get_state()[0]):
            assert cases.rel_l2(x, y) <= 1e-6
