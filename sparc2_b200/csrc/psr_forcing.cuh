// psr_forcing.cuh -- the PULSE = 2 forcing of one 32 x 8 tile of a layer
// (all_modules.f90:592-611 / 644-660, driver.f90:153), shared by the single
// path's kernels of both precisions: the sum over the layer's pulses of
// T_n(t) * Z_n(k) * X_n(i) * Y_n(j), culled per reference rank block, twice at
// the run's first iteration, times source_damp * src_scale_beta.
//
// A pulse is a few grid points wide, so most of a layer's pulses do not reach
// a given tile: the block first keeps, in order, those whose X factor is not
// below 1e-40 at every column of the tile and whose Y factor not at every row
// (the cut the layer lists make in z, far below the resolution of any sum it
// could join), a pulse per warp and step.  What bounds it then is the write
// of the plane; summing every pulse at every point was 6 % of an iteration
// at 300 pulses (149x149x211 FP32).
#pragma once

#include "internal.h"

namespace sparc {

// D: PsrDev (FP64 sums) or Psr32 (FP32 sums); sh: the dynamic buffer, a value
// of R and an int per pulse, and no static shared memory beside it: the 48 KB that
// a launch may take without asking hold 4096 pulses in FP64, 6144 in FP32.
// Block (32, 8); blockIdx: tile x, tile y, layer.
template <class R, class D>
__device__ __forceinline__ void psr_tile(const D &P, R *sh, int maxp) {
  const int k = P.klo + blockIdx.z;
  const int e0 = P.off[k], ne = P.off[k + 1] - e0;
  R *sT = sh;
  int *sN = (int *)(sh + maxp);
  const int lane = threadIdx.x, warp = threadIdx.y;
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 8;
  const int i = x0 + lane, j = y0 + warp;
  // which pulses reach the tile
  for (int e = warp; e < ne; e += 8) {
    const int n = P.idx[e0 + e];
    const bool hx = i < P.nx && !((double)P.px[(long long)n * P.nx + i] < 1e-40);
    const bool hy = lane < 8 && y0 + lane < P.ny &&
                    !((double)P.py[(long long)n * P.ny + y0 + lane] < 1e-40);
    const bool in = __any_sync(0xffffffffu, hx) && __any_sync(0xffffffffu, hy);
    if (lane == 0) sN[e] = in ? n : -1;
  }
  __syncthreads();
  // their list, in order
  if (warp == 0) {
    int at = 0;
    for (int b = 0; b < ne; b += 32) {
      const int e = b + lane;
      const int n = e < ne ? sN[e] : -1;
      const unsigned m = __ballot_sync(0xffffffffu, n >= 0);
      if (n >= 0) sN[at + __popc(m & ((1u << lane) - 1u))] = e;
      __syncwarp();
      at += __popc(m);
    }
    if (lane == 0) *(int *)sh = at;  // their count, where their factors go next
  }
  __syncthreads();
  const int kept = *(const volatile int *)sh;
  __syncthreads();
  const long long it = *P.iter;
  const double t = (double)it * P.timestep;
  const double passes = (it == P.init) ? 2.0 : 1.0;
  for (int q = warp * 32 + lane; q < kept; q += 256) {
    const int e = sN[q], n = P.idx[e0 + e];
    const double amp = P.ptime[3 * n], t0 = P.ptime[3 * n + 1], t1 = P.ptime[3 * n + 2];
    double v = amp * sin(2.0 * PI * (t - t1) / t0);
    v = v * exp(-((t - t1) * (t - t1)) / (2.0 * (P.st * P.st)));
    sT[q] = (R)(v * P.zv[e0 + e] * passes);
    sN[q] = n;
  }
  __syncthreads();
  if (i >= P.nx || j >= P.ny) return;
  const int blk = P.colx[i] + P.bx * P.coly[j] + P.bxy * P.colz[k];
  R f = R(0);
  for (int q = 0; q < kept; ++q) {
    const int n = sN[q];
    if (!P.mask[(long long)n * P.nblocks + blk]) continue;
    f = f + sT[q] * (P.px[(long long)n * P.nx + i] * P.py[(long long)n * P.ny + j]);
  }
  const long long g = ((long long)k * P.ny + j) * P.nx + i;
  P.out[((long long)blockIdx.z * P.ny + j) * P.nx + i] = f * P.sd[g] * P.ssb[g];
}

}  // namespace sparc
