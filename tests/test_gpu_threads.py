"""Handles of different z extents stepped by several host threads at once: the
dynamic shared memory a stage kernel may take belongs to the kernel, not to the
handle, so no handle may lower it between another one's launches.  Every step
has to be accepted, and each handle ends bitwise where it ends alone."""
import threading

import numpy as np
import pytest

from sparc2_b200 import Simulation, abi
from tests import cases

pytestmark = pytest.mark.gpu

STEPS = 600


def sim_of(name, prec, zc):
    p, bg, src = cases.CASES[name](nz=64)
    p.precision = prec
    s = Simulation(p, bg, src)
    s.set_zchunk(zc)
    return s


@pytest.mark.parametrize("name,prec", [("quiet_periodic", abi.SPARC_FP64),
                                       ("quiet_periodic", abi.SPARC_FP32),
                                       ("mhd_hpml", abi.SPARC_FP32)])
def test_extents_of_other_threads(name, prec):
    extents = (32, 11, 29, 16)
    want = []
    for zc in extents:
        s = sim_of(name, prec, zc)
        for nn in range(1, STEPS + 1):
            s.step(nn)
        want.append(s.get_state()[0])
    sims = [sim_of(name, prec, zc) for zc in extents]
    errors = []

    def work(s):
        try:
            for nn in range(1, STEPS + 1):
                s.step(nn)
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    th = [threading.Thread(target=work, args=(s,)) for s in sims]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
    for s, a in zip(sims, want):
        assert np.array_equal(s.get_state()[0], a)
