"""Which extents the z-extent autotuner times (sparc_tune): the set-up extent, so
that tuning does not lose to not tuning, and no launch shape twice.  Away from
any filter cadence each extent takes exactly one untimed and one timed
iteration, so their number can be read off the iterations run."""
import pytest

from sparc2_b200 import Simulation, abi
from tests import cases

pytestmark = pytest.mark.gpu

MHD = (12, 16, 24, 32, 40, 48, 64, 80, 100, 152)
QUIET = (12, 16, 24, 32)


@pytest.mark.parametrize("prec", [abi.SPARC_FP64, abi.SPARC_FP32])
@pytest.mark.parametrize("name,size", [("mhd_hpml", (80, 60, 128)), ("mhd_hpml", (96, 96, 160)),
                                       ("quiet_hpml", (64, 64, 128)),
                                       ("quiet_periodic", (64, 64, 28))])
def test_extents_timed(name, size, prec):
    p, bg, src = cases.CASES[name](*size)
    p.precision = prec
    p.t_z = p.t_xy = 1e6
    s = Simulation(p, bg, src)
    first = s.zchunk
    want = {first} | {min(c, p.nz) for c in (MHD if p.magnetic == 2 else QUIET)}
    if p.magnetic == 2:
        assert first >= 11
    nxt, best = s.tune(1, steps_per_trial=1)
    assert nxt - 1 == 2 * len(want)
    assert best in want and s.zchunk == best
