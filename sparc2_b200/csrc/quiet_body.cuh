// quiet_body.cuh -- the fused MP_QUIET_3D stage body (RHS.f90:18-175 with the
// CPML of RHS.f90:50-93 and one RK stage of step.f90:26-61), shared by the
// plain form (R = double, step.cu), the precision form (R = float with
// depth-scaled state and a compensated final update, step32.cu) and the
// batched engine.
//
// A block of 32 x TY threads owns as many columns and marches up a chunk of
// layers, one thread per column.  The traffic it cannot do without is 15
// words per point and stage, against about 110 arithmetic instructions; what
// bounds it is the latency of what a layer waits for, so:
//   * Everything a layer reads (the p, vx and vy planes with the halos their
//     x/y derivatives need, rho, the window heads of layer k + 5, the base
//     state, the 3-D background inputs, the carries of the precision form's
//     last stage) is copied by cp.async into a ring of NS layer buffers,
//     NS - 1 layers ahead; a thread's copies go to offsets fixed before the
//     loop.  cp.async rather than TMA: the usual grids are periodic, and a
//     tensor copy cannot wrap.  Loads carried in registers from one layer to
//     the next were 10 % slower than the ring (they share the few load
//     barriers of a warp with the loads of the layer).
//   * One barrier per layer.  It publishes the layer and frees the buffer of
//     the layer before, into which the copies of layer k + NS - 1 then go.
//   * The profiles of a layer (depth scales, horizontally uniform
//     background, metric, gravity) sit in shared memory.
//   * The z windows are registers; the x/y derivatives of tiles without a
//     one-sided row are the centred antisymmetric sum, the others take
//     per-lane and per-row coefficients from a small table (no divergence).
// Measured per iteration of five stages, against one shared layer tile with
// two barriers per layer and loads at their use (before -> after): FP32
// 256x256x300 8.74 -> 2.34 ms; FP64 64x64x128 0.308 -> 0.121 ms, 32x32x48
// 0.300 -> 0.044 ms, 133x117x171 with a 3-D background and side CPML
// 1.86 -> 1.05 ms.  The FP32 kernel issues 67 % of its cycles (545 thread
// instructions per point, half of them addresses and copies); the FP64 one
// 50 %, at 0.57 of the measured copy rate.
//
// Each translation unit that includes this header defines dcoef<R>(row, m)
// (mhd_body.cuh).
#pragma once

#include "mhd_body.cuh"

namespace sparc {

// cp.async of one value to a shared address
template <class R>
__device__ __forceinline__ void cp_sr(unsigned dst, const R *src) {
  if constexpr (sizeof(R) == 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}

namespace qg {
constexpr int TX = 32;   // tile columns along x
constexpr int PX = 42;   // pitch of a plane with x halos
// own-point slots: rho, window heads of vz and p, base state 0..4, then
// rho0, rhoinv, c2rho0, gradrho0_z, gradp0_z where they are 3-D
constexpr int O_RHO = 0, O_HZ = 1, O_HP = 2, O_A = 3, O_BG = 8;
}  // namespace qg

// ring of a block (R words): NS layer buffers, then the edge coefficients,
// then TW profile words for each of the layers a chunk touches
// (C: the five carries of the precision form's last stage too)
template <class R, int TY, bool BG1D, int NS, bool C>
struct QuietBuf {
  static constexpr int HY = TY + 10, NC = qg::TX * TY;
  static constexpr int P = HY * qg::PX, VX = TY * qg::PX, VY = HY * qg::TX;
  static constexpr int O_VZ = BG1D ? 8 : 13;  // precision form: stored vz
  static constexpr int O_C = O_VZ + (sizeof(R) == 4 ? 1 : 0), NO = O_C + (C ? 5 : 0);
  static constexpr int STAGE = P + VX + VY + NO * NC;
  static constexpr int COEF = (qg::TX + TY) * 12 + 4;
  static constexpr int TW = BG1D ? 16 : 9;  // table words per layer
  static constexpr int RING = (NS * STAGE + 3) & ~3;
  static constexpr size_t bytes(int zext) {
    return ((size_t)RING + COEF + (size_t)(zext + 16) * TW) * sizeof(R);
  }
};

// Two CPML fields of one face at one point (RHS.f90:50-93); loads before
// stores.  slot 1 goes with d1, slot 0 with d0.
template <class R, int MODE>
__device__ __forceinline__ void cpml2_t(const FaceT<R> &F, long long f, int layer, R beta, R dt,
                                        R &d1, R &d0) {
  const long long pf = F.uniform ? (long long)layer : f;
  const R pa = __ldg(F.pa + pf), pb = __ldg(F.pb + pf), pki = __ldg(F.pki + pf);
  const long long o1 = F.cnt + f;
  const R v0 = F.vars[f], v1 = F.vars[o1];
  R p0 = v0, p1 = v1;
  if (MODE != F_FIRST) {
    const R c0 = F.scr[f], c1 = F.scr[o1];
    p0 = v0 + beta * c0;
    p1 = v1 + beta * c1;
  }
  const R r0 = pa * d0 + pb * p0, r1 = pa * d1 + pb * p1;
  d0 = d0 * pki + p0;
  d1 = d1 * pki + p1;
  if (MODE == F_LAST) {
    F.vars[f] = v0 + dt * r0;
    F.vars[o1] = v1 + dt * r1;
  } else {
    F.scr[f] = r0;
    F.scr[o1] = r1;
  }
}

// The body covers the tile (x0, y0) of 32 x TY columns over layers [k0, k1);
// (tx, ty) is the calling thread's column in the tile.  Every thread of the
// block calls it; smem is 16-byte aligned and holds QuietBuf::bytes.  The
// diagnostics of the last stage accumulate into ke, mr, mp.
template <class R, int TY, int MODE, bool BG1D, int NS>
__device__ __forceinline__ void quiet_body(const SimT<R> &S, R *smem, const R *__restrict__ a,
                                           const R *__restrict__ tin, R *__restrict__ so, R beta,
                                           R bnext, int x0, int y0, int k0, int k1, int tx,
                                           int ty, double &ke, double &mr, double &mp) {
  using namespace qg;
  using QB = QuietBuf<R, TY, BG1D, NS, sizeof(R) == 4 && MODE == F_LAST>;
  constexpr int NC = QB::NC, NT = NC;
  constexpr bool SCALED = sizeof(R) == 4;
  const int tid = ty * TX + tx;
  const int nx = S.nx, ny = S.ny, nz = S.nz;
  const long long N = S.N;
  const int NXY = nx * ny;
  const int i = x0 + tx, j = y0 + ty;
  const bool act = i < nx && j < ny;
  const bool per = S.periodic;
  const int col = j * nx + i;
  const int xo = origin_t(x0, TX, nx, per), yo = origin_t(y0, TY, ny, per);
  const int cx0 = x0 - xo, cy0 = y0 - yo;  // interior offset in the tile
  const R dt = (R)S.deltat, sx = (R)S.stretchx, sy = (R)S.stretchy;

  const int fk = S.frc.kind, fdir = S.frc.dir;

  // profiles of the layers the chunk touches; the gravity of the tile's
  // first point serves where the tile lies in one block column
  const int xe = min(x0 + TX, nx) - 1, ye = min(y0 + TY, ny) - 1;
  const int gc0 = S.colx[x0] + S.bxdim * S.coly[y0];
  const bool g_one = S.colx[xe] + S.bxdim * S.coly[ye] == gc0;
  constexpr int TW = QB::TW;
  R *coef = smem + QB::RING;
  R *tab = coef + QB::COEF;
  const int zb = max(0, min(k0 - 5, nz - 11));
  {
    const int ze = min(nz, max(k1 + 5, zb + 11));
    for (int t = tid; t < (ze - zb) * TW; t += NT) {
      const int kk = zb + t / TW, c = t % TW;
      R v = R(0);
      if (c == 3) v = S.stretch[kk];
      if (c == 7 && fk == SPARC_SRC_PULSE) v = S.frc.fz[kk];
      if (c == 7 && fk == SPARC_SRC_RANDOM) v = S.frc.sdep[kk];
      if constexpr (SCALED) {  // the three velocities share a scale
        if (c < 3) v = S.isc[(c == 0 ? 0 : (c == 1 ? 1 : 4)) * nz + kk];
        else if (c >= 4 && c < 7) v = S.sc[(c == 4 ? 0 : (c == 5 ? 1 : 4)) * nz + kk];
      }
      if constexpr (BG1D) {
        if (c >= 8 && c < 15) {
          const R *q = c == 8 ? S.rho0 : c == 9 ? S.rhoinv : c == 10 ? S.c2rho0
                     : c == 11 ? S.grz : c == 12 ? S.gpz : c == 13 ? S.sponge : S.p0;
          v = q[kk];
        }
      }
      if (c == TW - 1) v = S.gblk[(long long)gc0 * nz + kk];
      tab[t] = v;
    }
  }
  if (fk == SPARC_SRC_PULSE && tid == NT - 1) coef[QB::COEF - 1] = pulse_time_t(S, *S.iter);
  // one-sided rows: coefficients and window start of each lane (x) and row
  // (y); the centred row elsewhere (derivatives.f90:72, 98)
  const bool cen_x = per || (x0 >= 5 && x0 + TX <= nx - 5);
  const bool cen_y = per || (y0 >= 5 && y0 + TY <= ny - 5);
  if (!(cen_x && cen_y) && tid < TX + TY) {
    const bool isx = tid < TX;
    const int q0 = isx ? tid : tid - TX;
    const int g = isx ? x0 + q0 : y0 + q0, n = isx ? nx : ny, o = isx ? xo : yo;
    R *c = coef + tid * 12;
    int base;
    if (per || (g >= 5 && g < n - 5) || g >= n) {
      for (int m = 0; m < 11; ++m) c[m] = dcoef<R>(5, m);
      base = g >= n ? 0 : g - 5 - o;
    } else if (g < 5) {
      for (int m = 0; m < 11; ++m) c[m] = dcoef<R>(g, m);
      base = -o;
    } else {
      for (int m = 0; m < 11; ++m) c[m] = -dcoef<R>(n - 1 - g, 10 - m);
      base = n - 11 - o;
    }
    c[11] = (R)base;
  }

  // copy plan: the own point of each plane, and up to two halo points
  // (y halo: ten rows of p and vy, one per warp; x halo: ten columns of p
  // and vx).  Offsets within a layer.  Positions outside a non-periodic grid
  // are clamped into it: their copies land where nothing reads, which is
  // cheaper than a branch per copy.
  auto at = [&](int lx, int ly) -> int {
    int gx = xo + lx, gy = yo + ly;
    if (per) {  // at most a tile and a halo outside, the grid is 22 or more
      if (gx < 0) gx += nx;
      if (gy < 0) gy += ny;
      while (gx >= nx) gx -= nx;
      while (gy >= ny) gy -= ny;
    } else {
      gx = min(max(gx, 0), nx - 1);
      gy = min(max(gy, 0), ny - 1);
    }
    return gy * nx + gx;
  };
  const unsigned g_own = at(cx0 + tx, cy0 + ty);
  const int s_px = (cy0 + ty) * PX + cx0 + tx;                   // own point in p
  const int s_vx = QB::P + ty * PX + cx0 + tx;                   // in vx
  const int s_vy = QB::P + QB::VX + (cy0 + ty) * TX + tx;        // in vy
  // halo slot 0: warps 0..9 a y-halo row (32 columns); TY = 16: warps 11..15
  // the x halo.  Slot 1 (TY = 8): warps 0, 1 the y-halo rows 8, 9; warps 2..4
  // the x halo.  g: offset of the point, f: of its velocity (vy on y halos,
  // vx on x halos); s, t: their places in the layer buffer.
  int g_h0 = 0, s_h0 = 0, t_h0 = 0, g_h1 = 0, s_h1 = 0, t_h1 = 0;
  bool x_h0 = false, x_h1 = false, on_h0 = false, on_h1 = false;
  {
    auto yrow = [&](int h, int &g, int &s, int &t, bool &on) {
      on = true;
      const int ly = h < cy0 ? h : h + TY;
      g = at(cx0 + tx, ly);
      s = ly * PX + cx0 + tx;
      t = QB::P + QB::VX + ly * TX + tx;
    };
    auto xcol = [&](int q, int &g, int &s, int &t, bool &on) {
      if (q >= 10 * TY) return;
      on = true;
      const int r = q / 10, h = q - r * 10, lx = h < cx0 ? h : h + TX;
      g = at(lx, cy0 + r);
      s = (cy0 + r) * PX + lx;
      t = QB::P + r * PX + lx;
    };
    if (TY == 8 || ty < 10) yrow(ty, g_h0, s_h0, t_h0, on_h0);
    if (TY == 8) {
      if (ty < 2) yrow(8 + ty, g_h1, s_h1, t_h1, on_h1);
      else if (ty < 5) { x_h1 = true; xcol(tid - 64, g_h1, s_h1, t_h1, on_h1); }
    } else if (ty >= 11) {
      x_h0 = true;
      xcol(tid - 11 * 32, g_h0, s_h0, t_h0, on_h0);
    }
  }
  // shared addresses of buffer 0
  constexpr unsigned W = sizeof(R), BB = QB::STAGE * W;
  const unsigned sb = sm_addr_t(smem);
  const unsigned a_own = sb + (QB::P + QB::VX + QB::VY + tid) * W;
  const unsigned a_px = sb + s_px * W, a_vx = sb + s_vx * W, a_vy = sb + s_vy * W;
  const unsigned a_s0 = sb + s_h0 * W, a_t0 = sb + t_h0 * W;
  const unsigned a_s1 = sb + s_h1 * W, a_t1 = sb + t_h1 * W;
  const bool slab_xy = (S.xb.on && (x0 < S.xb.np || x0 + TX > nx - S.xt.np)) ||
                       (S.yb.on && (y0 < S.yb.np || y0 + TY > ny - S.yt.np));
  auto sponge_at = [&](int k) -> bool {
    return !S.sponge_slabs || slab_xy || (S.zb.on && (k < S.zb.np || k >= nz - S.zt.np));
  };
  const unsigned gcl = at(min(cx0 + tx, nx - 1 - xo), min(cy0 + ty, ny - 1 - yo));  // own column
  auto issue = [&](int k, int b) {
    const unsigned o = b * BB;
    const long long kb = (long long)k * NXY;
    const R *t0 = tin + kb, *t1 = t0 + N, *t2 = t1 + N, *t3 = t2 + N, *t4 = t3 + N;
    cp_sr(a_px + o, t4 + g_own);
    cp_sr(a_vx + o, t1 + g_own);
    cp_sr(a_vy + o, t2 + g_own);
    if (TY == 8 || on_h0) {
      cp_sr(a_s0 + o, t4 + g_h0);
      cp_sr(a_t0 + o, (TY != 8 && x_h0 ? t1 : t2) + g_h0);
    }
    if (TY == 8 && on_h1) {
      cp_sr(a_s1 + o, t4 + g_h1);
      cp_sr(a_t1 + o, (x_h1 ? t1 : t2) + g_h1);
    }
    const unsigned ao = a_own + o;
    cp_sr(ao + O_RHO * NC * W, t0 + gcl);
    if constexpr (SCALED) cp_sr(ao + QB::O_VZ * NC * W, t3 + gcl);
    if (k > k0 && k <= nz - 6) {  // window heads
      const long long up = 5LL * NXY;
      const R *u3 = t3 + up, *u4 = t4 + up;
      cp_sr(ao + O_HZ * NC * W, u3 + gcl);
      cp_sr(ao + O_HP * NC * W, u4 + gcl);
    }
    if (MODE != F_FIRST) {
      const R *ab = a + kb;
#pragma unroll
      for (int l = 0; l < 5; ++l) cp_sr(ao + (O_A + l) * NC * W, ab + l * N + gcl);
    }
    if constexpr (!BG1D) {
      cp_sr(ao + (O_BG + 0) * NC * W, S.rho0 + kb + gcl);
      cp_sr(ao + (O_BG + 1) * NC * W, S.rhoinv + kb + gcl);
      cp_sr(ao + (O_BG + 2) * NC * W, S.c2rho0 + kb + gcl);
      cp_sr(ao + (O_BG + 3) * NC * W, S.grz + kb + gcl);
      cp_sr(ao + (O_BG + 4) * NC * W, S.gpz + kb + gcl);
    }
    if (SCALED && MODE == F_LAST) {
      const R *cb = S.carry + kb;
#pragma unroll
      for (int l = 0; l < 5; ++l) cp_sr(ao + (QB::O_C + l) * NC * W, cb + l * N + gcl);
    }
  };
#pragma unroll
  for (int s = 0; s < NS - 1; ++s) {
    if (k0 + s < k1) issue(k0 + s, s);
    cp_commit_t();
  }
  // z windows (physical values), first loads all in flight at once
  R wvz[11], wp[11];
  {
    const int b0 = min(k0 - 5, nz - 11);
#pragma unroll
    for (int m = 0; m < 11; ++m) {
      const int kk = b0 + m;
      const bool ok = act && kk >= 0;
      const long long id = (long long)kk * NXY + col;
      wvz[m] = ok ? __ldg(tin + 3 * N + id) : R(0);
      wp[m] = ok ? __ldg(tin + 4 * N + id) : R(0);
    }
    __syncthreads();  // the tables
    if constexpr (SCALED) {
#pragma unroll
      for (int m = 0; m < 11; ++m) {
        const R *q = tab + max(0, b0 + m - zb) * TW;
        wvz[m] *= q[1];
        wp[m] *= q[2];
      }
    }
  }
  // forcing of this column: the PULSE = 1 factors (the time factor is fixed
  // during a stage), the PULSE = 0 plane
  const R Tp = fk == SPARC_SRC_PULSE ? coef[QB::COEF - 1] : R(1);
  R fxy = R(0);
  if (act) {
    if (fk == SPARC_SRC_PULSE) fxy = __ldg(S.frc.fy + j) * __ldg(S.frc.fx + i);
    else if (fk == SPARC_SRC_RANDOM) fxy = S.frc.f2d[col];
  }
  // gravity: from the table where the tile lies in one block column
  const R *gcol = S.gblk + (act ? S.colx[i] + S.bxdim * S.coly[j] : 0) * nz;
  const bool psr = fk == SPARC_SRC_PSR;

  int b = 0;
  for (int k = k0; k < k1; ++k, b = b == NS - 1 ? 0 : b + 1) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(NS - 2) : "memory");
    __syncthreads();
    if (k + NS - 1 < k1) issue(k + NS - 1, b == 0 ? NS - 1 : b - 1);
    cp_commit_t();
    if (!act) continue;
    const R *P = smem + b * QB::STAGE, *O = P + QB::P + QB::VX + QB::VY + tid;
    const R *tk = tab + (k - zb) * TW;
    const long long kb = (long long)k * NXY, id = kb + col;
    if (k > k0 && k <= nz - 6) {
      const R *tu = tk + 5 * TW;
      shift_t(wvz, SCALED ? O[O_HZ * NC] * tu[1] : O[O_HZ * NC]);
      shift_t(wp, SCALED ? O[O_HP * NC] * tu[2] : O[O_HP * NC]);
    }
    R gk = tk[TW - 1], frc;
    if (!g_one) gk = __ldg(gcol + k);
    if (psr) {
      frc = R(0);
      if (k >= S.frc.klo && k < S.frc.khi)
        frc = S.frc.psr[(long long)(k - S.frc.klo) * NXY + col];
    } else {
      frc = Tp * tk[7] * fxy;
    }
    R sg = R(0), p0v = R(0);
    if constexpr (BG1D) {
      sg = tk[13];
      p0v = tk[14];
    } else {
      if (sponge_at(k)) sg = __ldg(S.sponge + id);
      if (MODE == F_LAST) p0v = __ldg(S.p0 + id);
    }
    // own values: stored, then physical
    R s_vz;
    if constexpr (SCALED) s_vz = O[QB::O_VZ * NC];
    else s_vz = k <= nz - 6 ? wvz[5] : __ldg(tin + 3 * N + id);
    const R s_rho = O[O_RHO * NC], s_vx1 = P[s_vx], s_vy1 = P[s_vy],
            s_p = P[s_px];
    R is0 = R(1), is1 = R(1), is4 = R(1), sc0 = R(1), sc1 = R(1), sc4 = R(1);
    const R szk = tk[3];
    if constexpr (SCALED) {
      is0 = tk[0]; is1 = tk[1]; is4 = tk[2];
      sc0 = tk[4]; sc1 = tk[5]; sc4 = tk[6];
    }
    const R rho = s_rho * is0, vx = s_vx1 * is1, vy = s_vy1 * is1, vz = s_vz * is1,
            p = s_p * is4;
    // derivatives (RHS.f90:42-48)
    R dvxdx, gpx, dvydy, gpy;
    if (cen_x) {
      dvxdx = csum_t(P + s_vx - 5, 1);
      gpx = csum_t(P + s_px - 5, 1);
    } else {
      const R *q = coef + tx * 12;
      const int o = (int)q[11] - (cx0 + tx);
      const R *f = P + s_vx + o, *g = P + s_px + o;
      dvxdx = gpx = R(0);
#pragma unroll
      for (int m = 0; m < 11; ++m) {
        dvxdx += f[m] * q[m];
        gpx += g[m] * q[m];
      }
    }
    if (cen_y) {
      dvydy = csum_t(P + s_vy - 5 * TX, TX);
      gpy = csum_t(P + s_px - 5 * PX, PX);
    } else {
      const R *q = coef + (TX + ty) * 12;
      const int o = (int)q[11] - (cy0 + ty);
      const R *f = P + s_vy + o * TX, *g = P + s_px + o * PX;
      dvydy = gpy = R(0);
#pragma unroll
      for (int m = 0; m < 11; ++m) {
        dvydy += f[m * TX] * q[m];
        gpy += g[m * PX] * q[m];
      }
    }
    dvxdx = is1 * (sx * dvxdx);
    gpx = is4 * (sx * gpx);
    dvydy = is1 * (sy * dvydy);
    gpy = is4 * (sy * gpy);
    R dvzdz, gpz;
    if (k < nz - 5) {
      dvzdz = szk * csum_t(wvz, 1);
      gpz = szk * csum_t(wp, 1);
    } else {
      dvzdz = dz_t(wvz, k, nz, szk);
      gpz = dz_t(wp, k, nz, szk);
    }
    // CPML (RHS.f90:50-93); psi slots: 0 vz/vx/vy, 1 p
    if (S.zb.on) {
      if (k < S.zb.np) {
        cpml2_t<R, MODE>(S.zb, id, k, beta, dt, gpz, dvzdz);
      } else if (k >= nz - S.zt.np) {
        const int kl = k - (nz - S.zt.np);
        cpml2_t<R, MODE>(S.zt, (long long)kl * NXY + col, kl, beta, dt, gpz, dvzdz);
      }
    }
    if (S.xb.on) {
      if (i < S.xb.np) {
        cpml2_t<R, MODE>(S.xb, i + (long long)S.xb.np * (j + (long long)ny * k), i, beta, dt,
                         gpx, dvxdx);
      } else if (i >= nx - S.xt.np) {
        const int il = i - (nx - S.xt.np);
        cpml2_t<R, MODE>(S.xt, il + (long long)S.xt.np * (j + (long long)ny * k), il, beta, dt,
                         gpx, dvxdx);
      }
      if (j < S.yb.np) {
        cpml2_t<R, MODE>(S.yb, i + (long long)nx * (j + (long long)S.yb.np * k), j, beta, dt,
                         gpy, dvydy);
      } else if (j >= ny - S.yt.np) {
        const int jl = j - (ny - S.yt.np);
        cpml2_t<R, MODE>(S.yt, i + (long long)nx * (jl + (long long)S.yt.np * k), jl, beta, dt,
                         gpy, dvydy);
      }
    }
    // RHS algebra (RHS.f90:95-152)
    R r0, ri, c2r, grz, gp0;
    if constexpr (BG1D) {
      r0 = tk[8]; ri = tk[9]; c2r = tk[10]; grz = tk[11]; gp0 = tk[12];
    } else {
      r0 = O[(O_BG + 0) * NC]; ri = O[(O_BG + 1) * NC]; c2r = O[(O_BG + 2) * NC];
      grz = O[(O_BG + 3) * NC]; gp0 = O[(O_BG + 4) * NC];
    }
    const R div = dvxdx + dvydy + dvzdz;
    R F[5];
    F[0] = -grz * vz - r0 * div - sg * rho;
    F[1] = -ri * gpx - sg * vx;
    F[2] = -ri * gpy - sg * vy;
    F[3] = -ri * (gpz + rho * gk) - vz * sg;
    if (fk != SPARC_SRC_NONE) {
      F[1] = fdir == 1 ? F[1] + frc : F[1];
      F[2] = fdir == 2 ? F[2] + frc : F[2];
      F[3] = fdir == 1 || fdir == 2 ? F[3] : F[3] + frc;
    }
    F[4] = -c2r * div - vz * gp0 - sg * p;
    // boundary planes (RHS.f90:154-164)
    const bool zero = k == 0 || k == nz - 1 ||
                      (!per && (i == 0 || i == nx - 1 || j == 0 || j == ny - 1));
    // DAMPING (plain form): the velocity RHS minus the damping term after the
    // boundary zeroing (RHS.f90:166-172), so the boundary planes move by -term
    bool zv = zero;
    if constexpr (!SCALED) {
      if (S.term) {
#pragma unroll
        for (int l = 1; l < 4; ++l)
          F[l] = (zero ? R(0) : F[l]) - __ldg(S.term + (long long)(l - 1) * N + id);
        zv = false;
      }
    }
    const R sv[5] = {s_rho, s_vx1, s_vy1, s_vz, s_p};
    const R scl[5] = {sc0, sc1, sc1, sc1, sc4};
    R *sp = so + id;
    if (MODE == F_LAST) {
      double an[5];
#pragma unroll
      for (int l = 0; l < 5; ++l) {
        const R av = O[(O_A + l) * NC];
        if constexpr (SCALED) {
          R c = O[(QB::O_C + l) * NC];
          const R t = zero ? av : kahan(av, dt * (scl[l] * F[l]), c);
          sp[l * N] = t;
          S.carry[l * N + id] = c;
          an[l] = ((double)t - (double)c) * (double)(l == 0 ? is0 : (l == 4 ? is4 : is1));
        } else {
          const bool z = l >= 1 && l < 4 ? zv : zero;
          const R t = z ? av : av + dt * F[l];
          sp[l * N] = t;
          an[l] = t;
        }
      }
      const double m =
          ((double)r0 + an[0]) * (an[1] * an[1] + an[2] * an[2] + an[3] * an[3]) / 2.0;
      ke += m * m;
      mr = fmin(mr, (double)rho + (double)r0);
      mp = fmin(mp, (double)p + (double)p0v);
    } else {
#pragma unroll
      for (int l = 0; l < 5; ++l) {
        const R av = MODE == F_FIRST ? sv[l] : O[(O_A + l) * NC];
        const bool z = l >= 1 && l < 4 ? zv : zero;
        sp[l * N] = z ? av : av + bnext * (scl[l] * F[l]);
      }
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

}  // namespace sparc
