"""PULSE = 2 tables as long as the forcing kernels' buffer takes: 4096 pulses in
the plain form, 6144 in the precision form; and one pulse more than a block has
threads.

Tolerance: one iteration from a random state agrees with the oracle to 1e-12
relative L2 per field in FP64 (sums of thousands of terms of one sign pattern,
1.1e-16 each), and to 1e-5 in the precision form (24-bit rounding)."""
import pytest

import oracle
from sparc2_b200 import Simulation, abi
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,pulses,tol", [(abi.SPARC_FP64, 257, 1e-12),
                                             (abi.SPARC_FP64, 4096, 1e-12),
                                             (abi.SPARC_FP32, 6144, 1e-5)])
def test_longest_tables(prec, pulses, tol):
    p, bg, src = cases.thermal_hpml(npulses=pulses)
    orc = oracle.Oracle(p, bg, src)
    p.precision = prec
    sim = Simulation(p, bg, src)
    a0, psi0 = cases.random_state(sim, seed=6, amp=1e-6)
    for s in (sim, orc):
        s.set_state(a0, psi0)
        for nn in (400, 401):   # the pulses' amplitudes are near their peak
            s.step(nn)
    a, _ = sim.get_state()
    ra, _ = orc.get_state()
    for l in range(sim.V):
        assert cases.rel_l2(a[l], ra[l]) <= tol, l
