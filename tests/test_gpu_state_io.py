"""State I/O through the staged copies (arrays of 32 MB and more) and the plain ones:
what is set is read back unchanged in FP64, and in the precision form it is
exactly the rounded, scaled value (one FP32 rounding of scale * value on the
way in, an exact FP64 product on the way out), also with an odd number of
values and with two handles copying at the same time."""
import threading

import numpy as np
import pytest

from sparc2_b200 import Simulation, abi
from sparc2_b200 import workloads as W

pytestmark = pytest.mark.gpu


def sim_of(nx, ny, nz, magnetic, prec):
    p = W.base_params(nx, ny, nz, magnetic=magnetic, periodic=True, blocks=(1, 1, 2), npml=8,
                      precision=prec)
    bg = (W.quiet_background(nx, ny, nz) if magnetic == 0 else
          W.fluxtube_background(nx, ny, nz, p.xlength, p.ylength, periodic=True))
    return Simulation(p, bg), bg


def fields(sim, seed):
    rng = np.random.Generator(np.random.Philox(key=seed))
    return (rng.standard_normal((sim.V,) + sim.shape), rng.standard_normal(sim.n_psi))


@pytest.mark.parametrize("size", [(22, 22, 24, 0), (151, 121, 97, 0), (96, 96, 120, 2)])
def test_fp64_round_trip(size):
    sim, _ = sim_of(*size, abi.SPARC_FP64)
    a, psi = fields(sim, 1)
    sim.set_state(a, psi)
    b, bpsi = sim.get_state()
    assert np.array_equal(a, b) and np.array_equal(psi, bpsi)


@pytest.mark.parametrize("size", [(22, 22, 24, 0), (151, 121, 97, 0), (96, 96, 120, 2)])
def test_fp32_round_trip(size):
    sim, bg = sim_of(*size, abi.SPARC_FP32)
    a, psi = fields(sim, 2)
    sim.set_state(a, psi)
    b, bpsi = sim.get_state()
    assert np.array_equal(bpsi, psi.astype(np.float32).astype(np.float64))
    rho = bg["rho0"][:, 0, 0] / bg["rho0"][0, 0, 0]
    c2 = (bg["cs0"][:, 0, 0] / bg["cs0"][0, 0, 0]) ** 2
    one = np.ones_like(rho)
    for l in range(sim.V):
        s = 1.0 / rho if l == 0 else np.sqrt(rho) if l < 4 else 1.0 / (c2 * rho) if l == 4 else one
        sc = s.astype(np.float32).astype(np.float64)[:, None, None]
        isc = (1.0 / s).astype(np.float32).astype(np.float64)[:, None, None]
        want = (sc * a[l]).astype(np.float32).astype(np.float64) * isc
        # the test's own scales may round differently by one FP32 ulp
        assert np.all(np.abs(b[l] - want) <= 2.5e-7 * np.abs(want))


def test_two_handles_at_once():
    sims = [sim_of(96, 96, 120, 2, p)[0] for p in (abi.SPARC_FP64, abi.SPARC_FP32)]
    want = []
    for k, s in enumerate(sims):
        s.set_state(*fields(s, 5 + k))
        want.append(s.get_state())
    bad = []

    def work(k):
        for _ in range(4):
            got = sims[k].get_state()
            if not all(np.array_equal(x, y) for x, y in zip(got, want[k])):
                bad.append(k)

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
