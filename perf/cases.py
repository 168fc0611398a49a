"""The work that a user of this framework has it do, as measurable cases.

A case is one handle (or one batch of handles) that is built once and then
advanced: `prepare` builds the seeded background, source and starting state
and uploads them, `run` advances the driver loop by the case's iterations and
reads the whole state back, as a program that writes snapshots does.  All of
it goes through sparc2_b200.Simulation and sparc2_b200.batch.Batch.  `exact`
restates the same iterations in plain torch at 64 bits.

Form of a case:
  driver  the reference driver's calls one by one: step, diagnostics read
          back, filter_vars, for each iteration
  run     whole iterations through Simulation.run (captured graphs), then
          the diagnostics
  batch   several FP32 members admitted to a batch, advanced together,
          removed and read back
"""
import math
import random

import numpy as np
import torch

from sparc2_b200 import Simulation, abi
from sparc2_b200 import workloads as W
from sparc2_b200.batch import Batch

MM = W.MM
NPML = 10


def _c(form, nx, ny, nz, iterations, *, magnetic, precision="fp64", periodic=False,
       source="psr", pulses=100, filt=11, damping=False, tune=False):
    return dict(form=form, nx=nx, ny=ny, nz=nz, iterations=iterations, magnetic=magnetic,
                precision=precision, periodic=periodic, source=source, pulses=pulses,
                filt=filt, damping=damping, tune=tune)


def listed():
    cases = {
        # the smallest calls: a driver loop over a test-sized quiet box, where
        # launches and host round trips are most of the time
        "quiet32-driver": _c("driver", 32, 32, 48, 10, magnetic=0, periodic=True,
                             source="pulse"),
        # the quiet-Sun configuration: 64x64x128, periodic, one pulse
        "quiet64-fp64": _c("run", 64, 64, 128, 60, magnetic=0, periodic=True, source="pulse"),
        # a quiet ensemble member of the largest size, precision form
        "quiet256-fp32": _c("run", 256, 256, 300, 40, magnetic=0, periodic=True,
                            precision="fp32", source="pulse"),
        # hydro on a 3-D thermal background with side CPML, odd sizes
        "thermal-odd-fp64": _c("run", 133, 117, 171, 40, magnetic=1, source="psr"),
        # velocity damping (FFT per layer) on a quiet box
        "quiet-damping-fp64": _c("run", 96, 96, 150, 20, magnetic=0, periodic=True,
                                 source="pulse", damping=True),
        # a small magnetic box driven call by call with its diagnostics read
        "tube40-driver": _c("driver", 40, 40, 48, 10, magnetic=2, source="psr", pulses=20),
        # a magnetic box of odd size (no 16-byte rows), plain form
        "tube-odd-fp64": _c("run", 149, 151, 203, 30, magnetic=2, source="psr"),
        # the flux-tube configuration: 256x256x300, CPML on six faces, 200
        # pulses, tuned as a long production run tunes it
        "tube256-fp64": _c("run", 256, 256, 300, 40, magnetic=2, source="psr", pulses=200,
                           tune=True),
        # the same in the precision form
        "tube256-fp32": _c("run", 256, 256, 300, 40, magnetic=2, precision="fp32",
                           source="psr", pulses=200, tune=True),
        # a served solve: odd size, precision form, many pulses
        "tube-odd-fp32": _c("run", 149, 149, 211, 40, magnetic=2, precision="fp32",
                            source="psr", pulses=300),
        # a periodic magnetic box with the random source and the 7-point filter
        "periodic-random-fp32": _c("run", 128, 160, 180, 40, magnetic=2, precision="fp32",
                                   periodic=True, source="random", filt=7),
        # an ensemble of mixed members (quiet and magnetic, odd sizes) in a batch
        "batch6-fp32": dict(form="batch", members=6, pick=3, nmin=64, nmax=128, zmin=128,
                            zmax=200, iterations=30),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.15:
        return dict(form="batch", members=rng.randint(2, 8), pick=rng.randint(0, 999),
                    nmin=48, nmax=rng.randint(80, 144), zmin=96, zmax=rng.randint(120, 220),
                    iterations=rng.choice([10, 20, 30]))
    magnetic = rng.choice([0, 0, 1, 2, 2, 2, 2])
    precision = rng.choice(["fp64", "fp32"])
    periodic = magnetic == 0 or rng.random() < 0.2
    nx = _log(rng, 32, 224)
    ny = nx if rng.random() < 0.5 else min(224, max(32, int(nx * rng.uniform(0.6, 1.6))))
    nz = _log(rng, 48, 280)
    small = nx * ny * nz < 200000
    return _c("driver" if small and rng.random() < 0.5 else "run", nx, ny, nz,
              rng.choice([10, 20, 30, 40]), magnetic=magnetic, precision=precision,
              periodic=periodic,
              source=rng.choice(["pulse", "psr", "psr", "random"]),
              pulses=_log(rng, 20, 400), filt=rng.choice([11, 11, 7]),
              damping=precision == "fp64" and rng.random() < 0.1)


# ---------------------------------------------------------------- inputs

def _members(case):
    """The member boxes of a batch case: quiet or magnetic, sizes as served."""
    r = random.Random(case["pick"])
    out = []
    for m in range(case["members"]):
        n = r.randint(case["nmin"], case["nmax"])
        out.append(_c("run", n, n, r.randint(case["zmin"], case["zmax"]), case["iterations"],
                      magnetic=0 if m % 3 == 2 else 2, precision="fp32", periodic=m % 3 == 2,
                      source="psr" if m % 2 else "pulse", pulses=r.randint(50, 200)))
    return out


def _problem(c, seed):
    """(params, background, source) of one box: the flux-tube grid spacing,
    the top at +1 Mm, dt = 0.5 s, z filter every 10 steps, xy every 30."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    lx, ly = nx * W.DX_MM * MM, ny * W.DX_MM * MM
    npml = min(NPML, nx // 2, ny // 2, nz // 4)
    p = W.base_params(nx, ny, nz, magnetic=c["magnetic"], periodic=c["periodic"],
                      hpml=not c["periodic"], xlength=lx, ylength=ly, timestep=0.5, t_z=5.0,
                      t_xy=15.0, npml=npml, maxva=4.0e6,
                      precision=abi.SPARC_FP32 if c["precision"] == "fp32" else abi.SPARC_FP64)
    if c["filt"] == 7:
        p.filter_mode_xy = p.filter_mode_z = 2
    p.damping = 1 if c["damping"] else 0
    z_bot = 1.0 - (nz - 1) * W.DZ_MM
    if c["magnetic"] == 0:
        bg = W.quiet_background(nx, ny, nz, z_bot, 1.0)
    else:
        bg = W.fluxtube_background(nx, ny, nz, lx, ly, z_bot, 1.0, B0=2000.0,
                                   periodic=c["periodic"])
        if c["magnetic"] == 1:
            bg = dict(bg, bx0=None, by0=None, bz0=None)
    r = random.Random(seed)
    if c["source"] == "pulse":
        src = W.pulse_source(px=r.uniform(0.3, 0.7) * lx, py=r.uniform(0.3, 0.7) * ly,
                             pz=-0.5 * MM, sr=0.8 * MM, sz=0.4 * MM, t1=20.0, st=10.0)
    elif c["source"] == "psr":
        src = W.psr_source(W.psr_table(p, c["pulses"], seed))
    else:
        series = W.random_series(p, 64, 4.0, seed)
        src = W.random_source(series, cadforcing=4.0, ampl=3.0e3, depth=-0.5 * MM,
                              sigma=0.3 * MM)
    return p, bg, src


def _state(p, bg, seed, device):
    """A seeded field of small waves over the stratification, in code units:
    a few plane waves per field, in proportion to the background's density,
    sound speed and pressure at each depth."""
    nx, ny, nz, V = p.nx, p.ny, p.nz, 8 if p.magnetic == 2 else 5
    r = random.Random(seed * 2 + 1)
    f64 = dict(dtype=torch.float64, device=device)
    x = torch.arange(nx, **f64) / nx
    y = torch.arange(ny, **f64) / ny
    z = torch.arange(nz, **f64) / nz
    rho, cs, pre = (torch.tensor(np.ascontiguousarray(bg[k][:, 0, 0]), **f64)
                    for k in ("rho0", "cs0", "pre0"))
    amp = [rho / rho[0]] + [cs / cs[0]] * 3 + [pre / (rho[0] * cs[0] ** 2)]
    amp += [torch.full((nz,), 0.01, **f64)] * (V - 5)
    a = torch.zeros((V, nz, ny, nx), **f64)
    for l in range(V):
        for _ in range(3):
            fx = torch.sin(2 * math.pi * (r.randint(1, 5) * x + r.random()))
            fy = torch.sin(2 * math.pi * (r.randint(1, 5) * y + r.random()))
            fz = torch.sin(2 * math.pi * (r.uniform(1, 5) * z + r.random()))
            a[l] += (1e-4 * amp[l] * fz)[:, None, None] * fy[None, :, None] * fx[None, None, :]
    return a


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _State:
    pass


def _open(c, seed):
    p, bg, src = _problem(c, seed)
    sim = Simulation(p, bg, src)
    a = _state(p, bg, seed, _device()).cpu().numpy()
    if c["tune"]:
        sim.tune(1)
    psi = np.zeros(sim.n_psi)
    sim.set_state(a, psi)
    return sim


def prepare(case, seed):
    s = _State()
    s.case, s.next = case, 1
    if case["form"] == "batch":
        s.sims = [_open(c, seed * 64 + m) for m, c in enumerate(_members(case))]
        s.batch = Batch(len(s.sims))
    else:
        s.sims = [_open(case, seed)]
    return s


def _read(sim):
    """The whole state, in the precision it was computed in."""
    a, psi = sim.get_state()
    if sim.params.precision == abi.SPARC_FP32:
        return {"a": torch.from_numpy(a).to(torch.float32),
                "psi": torch.from_numpy(psi).to(torch.float32)}
    return {"a": a, "psi": psi}


def run(state):
    case, first, n = state.case, state.next, state.case["iterations"]
    state.next = first + n
    if case["form"] == "batch":
        slots = [state.batch.add(sim, first, n) for sim in state.sims]
        state.batch.run(n)
        for slot in slots:
            state.batch.remove(slot)
        return [_read(sim) for sim in state.sims]
    sim = state.sims[0]
    if case["form"] == "driver":
        norms = []
        for nn in range(first, first + n):
            sim.step(nn)
            d, _ = sim.diagnostics()
            norms.append(d.ke_norm)
            sim.filter_vars(nn)
        return dict(_read(sim), norm=np.array(norms))
    sim.run(first, n)
    d, _ = sim.diagnostics()
    return dict(_read(sim), diag=[d.ke_norm, d.min_rho, d.min_p])


def work(case):
    """Bytes and operations of one pass.  Each of the five RK stages reads
    the stage input and the step's base state and writes the stage output
    (14 words per field and step), reads the 3-D background inputs, and
    updates the CPML fields of its slabs; a filter pass reads and writes the
    state; the state is read once at the end."""
    if case["form"] == "batch":
        parts = [work(c) for c in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    nx, ny, nz, it = case["nx"], case["ny"], case["nz"], case["iterations"]
    mhd = case["magnetic"] == 2
    V, C, P = (8, 6, 6) if mhd else (5, 3 if case["magnetic"] == 1 else 0, 2)
    w = 4 if case["precision"] == "fp32" else 8
    n = nx * ny * nz
    npml = min(NPML, nx // 2, ny // 2, nz // 4)
    slabs = 2 * npml / nz + (0 if case["periodic"] else 2 * npml / nx + 2 * npml / ny)
    words = 14 * V + 5 * C + 14 * P * slabs + 2 * V * (1 / 10 + 1 / 30)
    if w == 4:
        words += 2 * V
    flops = 5 * (18 * 16 + 130 if mhd else 6 * 16 + 45) + V * (2 * 22 / 30 + 22 / 10)
    if case["damping"]:
        words += 5 * 3 * 4
        flops += 5 * 3 * 5 * math.log2(nx * ny)
    return {"bytes": it * n * words * w + V * n * w, "flops": it * n * flops}


# ------------------------------------------------- the same in 64 bits

RSUN, PI = W.RSUN, W.PI_REF
ROWS = [
    [-2.391602219538, 5.832490322294, -7.650218001182 + 0.000000000001, 7.907810563576,
     -5.922599052629, 3.071037015445, -1.014956769726, 0.170022256519, 0.002819958377,
     -0.004791009708, -0.000013063429],
    [-0.180022054228, -1.237550583044, 2.484731692990, -1.810320814061, 1.112990048440,
     -0.481086916514, 0.126598690230, -0.015510730165, 0.000024609059 - 0.000003,
     0.000156447571 - 0.000000000001, -0.000007390277],
    [0.057982271137, -0.536135360383, -0.264089548967 + 0.000000000002,
     0.917445877606 - 0.000000000002, -0.169688364841, -0.029716326170, 0.029681617641,
     -0.005222483773, -0.000118806260, -0.000118806260, -0.000020069730],
    [-0.013277273810, 0.115976072920, -0.617479187931, -0.274113948206 + 0.000000000002,
     1.086208764655 - 0.000000000002, -0.402951626982, 0.131066986242, -0.028154858354,
     0.002596328316, 0.000128743150, 0.0],
    [0.016756572303, -0.117478455239, 0.411034935097, -1.130286765151,
     0.341435872100 - 0.000000000001, 0.556396830543, -0.082525734207, 0.003565834658,
     0.001173034777, -0.000071772671 + 0.000000000064, -0.000000352273],
    [-0.002484594688, 0.020779405824, -0.090320001280, 0.286511173973, -0.872756993962, 0.0,
     0.872756993962, -0.286511173973, 0.090320001280, -0.020779405824, 0.002484594688]]
FILT11 = [0.5 * 0.001953125, -0.5 * 0.01953125, 0.5 * 0.087890625, -0.5 * 0.234375,
          0.5 * 0.41015625, 0.75390625, 0.5 * 0.41015625, -0.5 * 0.234375, 0.5 * 0.087890625,
          -0.5 * 0.01953125, 0.5 * 0.001953125]
FILT7 = [-0.015625, 0.09375, -0.234375, 0.3125, -0.234375, 0.09375, -0.015625]


def _sub(dim, lo, hi):
    """Index of [lo, hi) along dimension dim of a (z, y, x) array."""
    return tuple(slice(lo, hi) if d == dim else slice(None) for d in range(3))


def _deriv(f, dim, scale, per):
    """The 11-point derivative along dim (0 z, 1 y, 2 x): wrapped where
    periodic; else one-sided rows within 5 points of an edge, but along z at
    the top only (the bottom takes zero ghosts)."""
    n = f.shape[dim]
    pad = f.new_zeros([s if d != dim else 5 for d, s in enumerate(f.shape)])
    if per:
        ext = torch.cat([f[_sub(dim, n - 5, n)], f, f[_sub(dim, 0, 5)]], dim)
    else:
        ext = torch.cat([pad, f, pad], dim)
    out = torch.zeros_like(f)
    for m in range(11):
        if m != 5:
            out.add_(ext[_sub(dim, m, m + n)], alpha=ROWS[5][m])
    if not per:
        for q in range(5):
            if dim != 0:
                lo = sum(f[_sub(dim, m, m + 1)] * ROWS[q][m] for m in range(11))
                out[_sub(dim, q, q + 1)] = lo
            hi = sum(f[_sub(dim, n - 1 - m, n - m)] * -ROWS[q][m] for m in range(11))
            out[_sub(dim, n - 1 - q, n - q)] = hi
    return out.mul_(scale)


def _filter(f, dim, g, s, per):
    """One direction of the filter event on one field."""
    n = f.shape[dim]
    if not per:
        src = f.clone()
        for q in list(range(1, g)) + list(range(n - g, n - 1)):
            f[_sub(dim, q, q + 1)] = (src[_sub(dim, q + 1, q + 2)] +
                                      src[_sub(dim, q - 1, q)]) / 2.0
    row = FILT11 if g == 5 else FILT7
    if per:
        ext = torch.cat([f[_sub(dim, n - g, n)], f, f[_sub(dim, 0, g)]], dim)
        r = sum(ext[_sub(dim, m, m + n)] * row[m] for m in range(2 * g + 1))
    else:
        r = f.clone() if g == 5 or dim == 0 else torch.zeros_like(f)
        r[_sub(dim, g, n - g)] = sum(f[_sub(dim, m, m + n - 2 * g)] * row[m]
                                     for m in range(2 * g + 1))
    return f - s * r if g == 3 else r


def _blocks(n, b):
    size = [n // b + (1 if i < n % b else 0) for i in range(b)]
    return [sum(size[:i]) for i in range(b)], size


class _Exact:
    """One box of the linear wave equations, plain torch, 64 bits."""

    def __init__(self, p, bg, src, device):
        self.p, self.src, self.dev = p, src, device
        T = lambda v: torch.tensor(v, dtype=torch.float64, device=device)  # noqa: E731
        nx, ny, nz = self.nx, self.ny, self.nz = p.nx, p.ny, p.nz
        self.mhd, self.per = p.magnetic == 2, bool(p.periodic)
        per = self.per
        self.hpml = bool(p.use_hpml)
        self.V = 8 if self.mhd else 5
        dx, dy = (nx, ny) if per else (nx - 1, ny - 1)
        self.x, self.y = np.arange(nx) / dx, np.arange(ny) / dy
        self.z = 1.0 + np.asarray(bg["zaxis"]) * 1.0e8 / RSUN
        self.sx, self.sy = RSUN / p.xlength * dx, RSUN / p.ylength * dy
        rho, pre, cs = T(bg["rho0"]), T(bg["pre0"]), T(bg["cs0"])
        dimc, dimrho = float(cs[0, 0, 0]), float(rho[0, 0, 0])
        self.dimc, self.dimrho = dimc, dimrho
        dimb = math.sqrt(4.0 * PI * dimc ** 2 * dimrho)
        cq = cs[:, 0, 0] / dimc
        self.invrho0q = 2.5440390e-7 / rho[:, 0, 0]
        if p.magnetic == 0:
            rho, pre, cs = (v[:, :1, :1].expand(nz, ny, nx).clone() for v in (rho, pre, cs))
        self.ssb = torch.ones_like(rho)
        B = None
        if self.mhd:
            B = [T(bg[k]) for k in ("bx0", "by0", "bz0")]
            b2 = B[0] ** 2 + B[1] ** 2 + B[2] ** 2
            k8 = float(np.float32(0.01) * np.float32(8.0))
            self.ssb = torch.clamp(k8 * PI * pre / torch.clamp(b2, min=1e-20), max=1.0)
            B = [b / dimb for b in B]
        g = np.asarray(bg["grav"]) * RSUN / dimc ** 2
        pre, rho, cs = pre / (dimrho * dimc ** 2), rho / dimrho, cs / dimc
        c2 = cs * cs
        self.rho0, self.p0, self.B = rho, pre, B
        rows = np.array(ROWS)
        u = np.empty(nz)
        for k in range(nz):
            if k < 5:
                u[k] = rows[k] @ self.z[:11]
            elif k >= nz - 5:
                u[k] = -(rows[nz - 1 - k] @ self.z[nz - 11:][::-1])
            else:
                u[k] = rows[5] @ self.z[k - 5:k + 6]
        self.sz = T(1.0 / u)[:, None, None]
        self.dt = p.timestep * dimc / RSUN
        self.sponge = torch.zeros_like(rho)
        self.red = None
        if self.mhd:
            b2 = B[0] ** 2 + B[1] ** 2 + B[2] ** 2
            red = b2 / (rho * (cq * cq)[:, None, None])
            va, step = 0.0, 1.0e9
            t = -step
            if float(red.max()) > 0.0:
                w = dimb ** 2 * b2 / (4.0 * PI * dimrho * rho)
                while step > 1.0e-5 and t < 1.0e10 - 1.1:
                    while va < p.maxva and t < 1.0e10:
                        t += step
                        va = torch.sqrt(t / (t + red) * w).max().item()
                        va = 0.0 if math.isnan(va) else va
                    t -= step
                    step /= 10.0
                    va = 0.0
            else:
                t = 1.0e10
            self.red = t / (t + red)
            self.cb = [self.ddy(B[2]) - self.ddz(B[1]), self.ddz(B[0]) - self.ddx(B[2]),
                       self.ddx(B[1]) - self.ddy(B[0])]
        self.ri, self.c2r = 1.0 / rho, c2 * rho
        self.grz, gpz = self.ddz(rho), self.ddz(pre)
        if p.stabilise:
            lo, hi = float(np.float32(0.9998)), float(np.float32(1.0001))
            add = 1.0e-4 * RSUN / (dimrho * dimc ** 2)
            for k in range(nz):
                zk, floor = self.z[k], -rho[k] * g[k]
                if lo < zk < 1.0:
                    gpz[k] = torch.maximum(c2[k] * self.grz[k] + add, floor)
                elif zk <= lo or zk >= hi:
                    gpz[k] = torch.maximum(c2[k] * self.grz[k], floor)
        self.gpz = gpz
        self._cpml(c2, g)
        if self.mhd:
            self.grx, self.gry = self.ddx(rho), self.ddy(rho)
            self.gpx, self.gpy = self.ddx(pre), self.ddy(pre)
        o = [1.0, 0.5, 0.1665579725791151184, 0.03950410250586729987, 0.007810706393337838236]
        b5 = o[1]
        b4 = o[2] / b5
        b3 = o[3] / (b5 * b4)
        b2_ = o[4] / (b5 * b4 * b3)
        self.betas = [0.0, b2_ * self.dt, b3 * self.dt, b4 * self.dt, b5 * self.dt]
        self.rates = None
        if p.damping:
            kx = np.arange(nx // 2 + 1)
            ky = np.minimum(np.arange(ny), ny - np.arange(ny))
            k = np.sqrt((2 * PI * RSUN / p.xlength * kx)[None, :] ** 2 +
                        (2 * PI * RSUN / p.ylength * ky)[:, None] ** 2)
            self.rates = T(RSUN / dimc / nx / ny * 1.0e-6 * (500.0 * (k / 902.0) ** 2.2) * 20.0)
        self._source()

    def ddx(self, f):
        return _deriv(f, 2, self.sx, self.per)

    def ddy(self, f):
        return _deriv(f, 1, self.sy, self.per)

    def ddz(self, f):
        return _deriv(f, 0, self.sz, False)

    def _cpml(self, c2, g):
        """Profiles of the faces (z bottom, z top, x, x, y, y), the damped
        gradients and gravity, the slab sponge and source_damp."""
        p, nx, ny, nz = self.p, self.nx, self.ny, self.nz
        c = torch.sqrt(c2 + self.red * (self.B[0] ** 2 + self.B[1] ** 2 + self.B[2] ** 2) /
                       self.rho0) if self.mhd else torch.sqrt(c2)
        T = lambda v: torch.tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        f0 = PI * 0.005 * RSUN / self.dimc
        bxs, byl = _blocks(nx, p.block_x)[0], _blocks(ny, p.block_y)[0]
        gb = np.tile(np.asarray(g), (p.block_y, p.block_x, 1))
        self.faces = []
        sd = [np.zeros(nx), np.zeros(ny)]
        spec = [(0, False, self.z, p.npml_zb, p.pml_zb), (0, True, self.z, p.npml_zt, p.pml_zt)]
        if self.hpml:
            spec += [(2, False, self.x, p.npml_xb, p.pml_xb),
                     (2, True, self.x, p.npml_xt, p.pml_xt),
                     (1, False, self.y, p.npml_yb, p.pml_yb),
                     (1, True, self.y, p.npml_yt, p.pml_yt)]
        for dim, top, axis, n, q in spec:
            size = len(axis)
            lo, hi = (size - n, size) if top else (0, n)
            edge = lo if top else n - 1
            L = axis[hi - 1] - axis[lo]
            ratio = ((axis[lo:hi] - axis[lo]) if top else (axis[n - 1] - axis[lo:hi])) / L
            rn = ratio ** q[1]
            alpha = f0 * ((axis[hi - 1] - axis[lo:hi]) if top else (axis[lo:hi] - axis[0])) / L
            kap = 1.0 + (q[2] - 1.0) * rn
            shape = [-1 if d == dim else 1 for d in range(3)]
            rn_, al_, ka_ = (T(v).reshape(shape) for v in (rn, alpha, kap))
            cin = c[_sub(dim, edge, edge + 1)]
            damp = q[0] * cin * (q[1] + 1.0) / (2.0 * L) * rn_
            at = _sub(dim, lo, hi)
            self.sponge[at] += q[3] * cin * T(ratio ** (q[1] + 1.0)).reshape(shape)
            if dim == 0:
                f = al_ / ka_ / (damp / ka_ + al_)
                self.grz[at] *= f
                self.gpz[at] *= f
                for by, j0 in enumerate(byl):
                    for bx, i0 in enumerate(bxs):
                        gb[by, bx, lo:hi] *= f[:, j0, i0].cpu().numpy()
            else:
                sd[0 if dim == 2 else 1][lo:hi] = rn
            P = 6 if self.mhd else 2
            size3 = [n if d == dim else s for d, s in enumerate((nz, ny, nx))]
            self.faces.append(dict(dim=dim, at=at, a=-damp / (ka_ * ka_), b=-al_ - damp / ka_,
                                   k=ka_, v=c.new_zeros([P] + size3),
                                   r=c.new_zeros([P] + size3)))
        self.sd = T(np.ones((ny, nx)) if self.per else
                    1.0 - np.maximum(sd[0][None, :], sd[1][:, None]))
        bx = np.searchsorted(np.array(bxs), np.arange(nx), side="right") - 1
        by = np.searchsorted(np.array(byl), np.arange(ny), side="right") - 1
        self.grav = T(np.ascontiguousarray(gb[by][:, bx].transpose(2, 0, 1)))

    def _source(self):
        """The parts of the forcing that do not depend on time."""
        p, s, nz = self.p, self.src, self.nz
        T = lambda v: torch.tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        ex = lambda d, w: T(np.exp(-d ** 2 / (2.0 * w ** 2)))  # noqa: E731
        if s.kind == abi.SPARC_SRC_PULSE:
            sr, sz = s.sr / RSUN, s.sz / RSUN
            self.f3 = (ex(self.z - (s.pz / RSUN + 1.0), sz)[:, None, None] *
                       ex(self.y * p.ylength / RSUN - s.py / RSUN, sr)[None, :, None] *
                       ex(self.x * p.xlength / RSUN - s.px / RSUN, sr)[None, None, :])
        elif s.kind == abi.SPARC_SRC_PSR:
            near = lambda v, c: np.minimum(np.minimum(abs(v - c), abs(v - 1.0 - c)),  # noqa: E731
                                           abs(v + 1.0 - c))
            self.pulses = []
            bx, by, bz = (_blocks(n, b) for n, b in ((self.nx, p.block_x), (self.ny, p.block_y),
                                                    (nz, p.block_z)))
            reach = lambda v, c, w, o, n: (  # noqa: E731
                ((c + 3 * w) % 1.0 >= v[o] or c + 3 * w >= v[-1]) and
                ((c - 3 * w) % 1.0 <= v[o + n - 1] or c - 3 * w <= v[0]))
            for q in s.pulses[:s.npulses]:
                m = [np.zeros(len(v)) for v in (self.z, self.y, self.x)]
                for o, n in zip(*bz):
                    if q.pz + 3 * q.sz >= self.z[o] and q.pz - 3 * q.sz <= self.z[o + n - 1]:
                        m[0][o:o + n] = 1.0
                for d, v, c, blk in ((1, self.y, q.py, by), (2, self.x, q.px, bx)):
                    for o, n in zip(*blk):
                        if reach(v, c, q.sr, o, n):
                            m[d][o:o + n] = 1.0
                fz = T(m[0]) * ex(self.z - q.pz, q.sz) * self.invrho0q
                self.pulses.append((q.amp, q.t0, q.t1, fz,
                                    T(m[1]) * ex(near(self.y, q.py), q.sr),
                                    T(m[2]) * ex(near(self.x, q.px), q.sr)))
        elif s.kind == abi.SPARC_SRC_RANDOM:
            self.series = T(s._keep) * (s.rnd_ampl / self.dimc)
            d = abs(self.z - (1.0 + s.rnd_depth / RSUN))
            e = nz - 1 - int(np.argmin(d[::-1]))
            self.dep = T(np.exp(-0.5 * (self.z - self.z[e]) ** 2 / 2.0 /
                                (s.rnd_sigma / RSUN) ** 2))

    def forcing(self, nn):
        s, t = self.src, nn * self.p.timestep
        if s.kind == abi.SPARC_SRC_PULSE:
            f = s.amp / 0.56458272 / self.dimc * math.sin(2.0 * PI * (t - s.t1 + 2.0 * s.t0) / s.t0)
            return f * math.exp(-(t - s.t1) ** 2 / (2.0 * s.st ** 2)) * self.f3
        if s.kind == abi.SPARC_SRC_PSR:
            fz, fy, fx = (torch.stack([q[i] for q in self.pulses]) for i in (3, 4, 5))
            w = [q[0] * math.sin(2.0 * PI * (t - q[2]) / q[1]) *
                 math.exp(-(t - q[2]) ** 2 / (2.0 * s.psr_st ** 2)) for q in self.pulses]
            w = torch.tensor(w, dtype=torch.float64, device=self.dev)
            f = torch.stack([(w[:, None] * fz[:, k:k + 1] * fy).t() @ fx
                             for k in range(self.nz)])
            return f * self.sd * self.ssb * (2.0 if nn == s.init else 1.0)
        cad, ns = s.cadforcing, s.nseries
        t1 = math.floor(t / cad) + 1
        xs = [(t1 - 4 + j) * cad for j in range(7)]
        out = torch.zeros_like(self.sd)
        for j in range(7):
            m = t1 - 4 + j
            if not (0 <= m < ns) or xs[j] < 0.0 or (j == 5 and t1 >= ns) or \
                    (j == 6 and t1 >= ns - 1):
                continue
            w = math.prod((t - xs[i]) / (xs[j] - xs[i]) for i in range(7) if i != j)
            out += w * self.series[m]
        return (out * self.sd)[None] * self.dep[:, None, None]

    def _pml(self, d, dim, slot, psi):
        for i, F in enumerate(self.faces):
            if F["dim"] == dim:
                v, at = psi[i][slot], F["at"]
                F["r"][slot] = F["a"] * d[at] + F["b"] * v
                d[at] = d[at] / F["k"] + v
        return d

    def rhs(self, t, psi, frc):
        dx = lambda f, s: self._pml(self.ddx(f), 2, s, psi)  # noqa: E731
        dy = lambda f, s: self._pml(self.ddy(f), 1, s, psi)  # noqa: E731
        dz = lambda f, s: self._pml(self.ddz(f), 0, s, psi)  # noqa: E731
        rho, vx, vy, vz, p = t[:5]
        S, ri, out = self.sponge, self.ri, torch.empty_like(t)
        div = dx(vx, 0) + dy(vy, 0) + dz(vz, 0)
        gp = [dx(p, 1), dy(p, 1), dz(p, 1)]
        out[0] = -self.grz * vz - self.rho0 * div - S * rho
        out[4] = -self.c2r * div - vz * self.gpz - S * p
        if self.mhd:
            out[0] -= self.grx * vx + self.gry * vy
            out[4] -= vx * self.gpx + vy * self.gpy
            b, (ox, oy, oz), (qx, qy, qz) = t[5:], self.B, self.cb
            f1, f2, f3 = vy * oz - vz * oy, vz * ox - vx * oz, vx * oy - vy * ox
            out[5] = self.red * (dy(f3, 4) - dz(f2, 4))
            out[6] = self.red * (dz(f1, 5) - dx(f3, 4))
            out[7] = self.red * (dx(f2, 5) - dy(f1, 5))
            j1 = dy(b[2], 3) - dz(b[1], 3)
            j2 = dz(b[0], 2) - dx(b[2], 3)
            j3 = dx(b[1], 2) - dy(b[0], 2)
            lor = [j2 * oz - j3 * oy + qy * b[2] - qz * b[1],
                   ox * j3 - j1 * oz + b[0] * qz - qx * b[2],
                   j1 * oy - j2 * ox + qx * b[1] - qy * b[0]]
            for i in range(3):
                gp[i] = gp[i] - lor[i] * self.red
        gp[2] = gp[2] + rho * self.grav
        for i in range(3):
            out[1 + i] = -ri * gp[i] - S * t[1 + i]
        out[self.src.dir] += frc
        out[:, 0] = 0.0
        out[:, -1] = 0.0
        if not self.per:
            out[:, :, 0] = 0.0
            out[:, :, -1] = 0.0
            out[..., 0] = 0.0
            out[..., -1] = 0.0
        if self.rates is not None:
            n = (self.ny, self.nx)
            out[1:4] -= torch.fft.irfft2(torch.fft.rfft2(t[1:4]) * self.rates, s=n,
                                         norm="forward")
        return out

    def iterate(self, a, nn):
        """One driver iteration; (state before the filter, minima)."""
        frc = self.forcing(nn)
        r, t, psi = None, a, [F["v"] for F in self.faces]
        for st in range(5):
            if st:
                t = a + self.betas[st] * r
                psi = [F["v"] + self.betas[st] * F["r"] for F in self.faces]
            r = self.rhs(t, psi, frc)
        for F in self.faces:
            F["v"] = F["v"] + self.dt * F["r"]
        a = a + self.dt * r
        ke = (self.rho0 + a[0]) * (a[1] ** 2 + a[2] ** 2 + a[3] ** 2) / 2.0
        norm = math.sqrt((ke * ke).mean().item()) * self.dimc ** 2 * self.dimrho
        return a, [norm, (t[0] + self.rho0).min().item(), (t[4] + self.p0).min().item()]

    def filters(self, a, nn):
        p = self.p
        gxy, gz = (5 if m == 1 else 3 for m in (p.filter_mode_xy, p.filter_mode_z))
        for l in range(self.V):
            if nn % int(p.t_xy / p.timestep + 1e-5) == 0:
                a[l] = _filter(a[l].clone(), 1, gxy, p.s_xy, self.per)
                a[l] = _filter(a[l].clone(), 2, gxy, p.s_xy, self.per)
            if nn % int(p.t_z / p.timestep + 1e-5) == 0:
                a[l] = _filter(a[l].clone(), 0, gz, p.s_z, False)
        return a


def _exact_box(c, seed):
    dev = _device()
    p, bg, src = _problem(c, seed)
    box = _Exact(p, bg, src, dev)
    a, diags = _state(p, bg, seed, dev), []
    for nn in range(1, c["iterations"] + 1):
        a, d = box.iterate(a, nn)
        diags.append(d)
        a = box.filters(a, nn)
    psi = torch.cat([F["v"].reshape(-1) for F in box.faces])
    return {"a": a, "psi": psi}, diags


def exact(case, seed):
    if case["form"] == "batch":
        return [_exact_box(c, seed * 64 + m)[0] for m, c in enumerate(_members(case))]
    out, diags = _exact_box(case, seed)
    if case["form"] == "driver":
        return dict(out, norm=np.array([d[0] for d in diags]))
    return dict(out, diag=diags[-1])
