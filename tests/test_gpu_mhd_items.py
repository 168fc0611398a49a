"""Blocks that take several MHD work items one after another: the mbarriers of
their layer buffers stay live from item to item (an item of an odd number of
layers leaves the two at different parities), also where the next item belongs
to another member of a batch.

Tolerance: a member ends where it ends alone to 1e-6 relative L2 (FP32-level,
as in the other batch tests); the plain form's state does not depend on the
extent (bitwise)."""
import numpy as np
import pytest

from sparc2_b200 import Simulation, abi
from sparc2_b200 import workloads as W
from sparc2_b200.batch import Batch
from tests import cases

pytestmark = pytest.mark.gpu

MM = W.MM


def sim_of(nx, ny, nz, prec):
    lx, ly = W.DX_MM * nx * MM, W.DX_MM * ny * MM
    p = W.base_params(nx, ny, nz, magnetic=2, periodic=False, hpml=True, xlength=lx, ylength=ly,
                      timestep=0.5, t_z=1.0, t_xy=1.0, npml=10, blocks=(2, 2, 2), precision=prec)
    bg = W.fluxtube_background(nx, ny, nz, lx, ly, 1.0 - (nz - 1) * W.DZ_MM, 1.0)
    return Simulation(p, bg, W.psr_source(W.psr_table(p, 20, 3)))


@pytest.mark.parametrize("sizes", [((74, 105), (84, 99)), ((128, 61), (97, 45), (64, 50))])
def test_batch_items_of_odd_layers(sizes):
    ref = []
    for n, nz in sizes:
        s = sim_of(n, n, nz, abi.SPARC_FP32)
        s.run(1, 3)
        ref.append(s.get_state()[0])
    sims = [sim_of(n, n, nz, abi.SPARC_FP32) for n, nz in sizes]
    with Batch(len(sims)) as b:
        b.set_tiles(33, 32)
        slots = [b.add(s, 1, 3) for s in sims]
        b.run(3)
        for q in slots:
            b.remove(q)
    for s, want in zip(sims, ref):
        d, r = s.diagnostics()
        assert r == abi.SPARC_OK and d.iteration == 3
        a, _ = s.get_state()
        for l in range(s.V):
            assert cases.rel_l2(a[l], want[l]) <= 1e-6


def test_set_up_extent_can_be_set_again():
    s = sim_of(40, 40, 48, abi.SPARC_FP64)
    zc = s.zchunk
    assert 4 <= zc <= 48
    s.set_zchunk(24)
    s.set_zchunk(zc)
    assert s.zchunk == zc
    if zc != 5:
        with pytest.raises(abi.SparcError):
            s.set_zchunk(5)


def test_persistent_items_of_odd_layers():
    # 4 x 20 tiles: about 400 items at 11 layers, 240 at 17, on 148 blocks
    got = []
    for zc in (None, 11, 17):
        s = sim_of(97, 160, 45, abi.SPARC_FP64)
        if zc:
            s.set_zchunk(zc)
        a0, psi0 = cases.random_state(s, seed=4, amp=1e-6)
        s.set_state(a0, psi0)
        s.run(1, 2)
        assert s.diagnostics()[1] == abi.SPARC_OK
        got.append(s.get_state()[0])
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
