"""A batch whose magnetic members take different bodies in one persistent block:
the edge tiles of a periodic member (halos that wrap) and all tiles of a member
without tensor maps are copied by cp.async, those of the others by tensor
copies.  Both orders of slots, more edge items than blocks (144 and 160 of 128 x
128 columns on 148 blocks), last chunks of 6, 7 and 27 layers.

Tolerance: a member ends where it ends alone to 1e-6 relative L2 (FP32-level,
as in the other batch tests)."""
import pytest

from sparc2_b200 import Simulation, abi
from sparc2_b200 import workloads as W
from sparc2_b200.batch import Batch
from tests import cases

pytestmark = pytest.mark.gpu

MM = W.MM


def sim_of(nz, periodic):
    n = 128
    lx = W.DX_MM * n * MM
    p = W.base_params(n, n, nz, magnetic=2, periodic=periodic, hpml=not periodic, xlength=lx,
                      ylength=lx, timestep=0.5, t_z=1.0, t_xy=1.0, npml=10, blocks=(2, 2, 2),
                      precision=abi.SPARC_FP32)
    bg = W.fluxtube_background(n, n, nz, lx, lx, 1.0 - (nz - 1) * W.DZ_MM, 1.0,
                               periodic=periodic)
    return Simulation(p, bg, W.psr_source(W.psr_table(p, 20, 3)))


# members in slot order: (nz, periodic, tensor maps)
MIXES = [((150, True, True), (150, False, True)), ((171, False, True), (171, True, True)),
         ((171, True, True), (150, False, True), (151, True, True)),
         ((150, False, False), (171, False, True))]


@pytest.mark.parametrize("mix", MIXES)
def test_members_of_different_bodies(mix, monkeypatch):
    def make():
        out = []
        for nz, periodic, maps in mix:
            monkeypatch.setenv("SPARC_TMA32", "1" if maps else "0")
            out.append(sim_of(nz, periodic))
        return out

    want = []
    for s in make():
        s.run(1, 3)
        want.append((s.get_state(), s.diagnostics()[0].ke_norm))
        s.close()
    sims = make()
    with Batch(len(sims)) as b:
        slots = [b.add(s, 1, 3) for s in sims]
        b.run(3)
        for q in slots:
            b.remove(q)
    for s, ((a0, psi0), ke) in zip(sims, want):
        d, r = s.diagnostics()
        assert r == abi.SPARC_OK and d.iteration == 3
        assert d.ke_norm == pytest.approx(ke, rel=1e-6)
        a, psi = s.get_state()
        for l in range(s.V):
            assert cases.rel_l2(a[l], a0[l]) <= 1e-6
        assert cases.rel_l2(psi, psi0) <= 1e-6
