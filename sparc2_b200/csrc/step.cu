// step.cu -- the time step on the device: one fused kernel per RK stage
// (stage values, 11-point derivatives, CPML, RHS, boundary zeroing, stage or
// final update, diagnostics), the PULSE = 2 forcing of an iteration, and
// the FILTER_VARS passes.
//
// Stage kernel layout: a CTA owns a TX x TY tile of (x, y) columns and
// marches up a chunk of z layers.  z derivatives come from an 11-deep window
// per z-differentiated field (the thread's own column): in registers for the
// quiet equations, in tensor memory for MHD; x and y derivatives from a
// shared-memory layer tile with a 5-point halo.
// Stage values are forwarded: stage k writes temp_{k+1} = a + beta_{k+1}*F_k
// (step.f90:33) instead of F_k, so every halo and window load of the next
// stage reads one array; stage 5 writes a + deltat*F_5 (step.f90:58).  The
// HBM traffic is that of the reference's scheme (14 V words per point and
// step) and the values are bitwise those of forming a + beta*F on load.

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>

#include "filter_body.cuh"
#include "mhd_body.cuh"
#include "psr_forcing.cuh"
#include "quiet_body.cuh"
#include "random_forcing.cuh"

namespace sparc {

__constant__ double c_dp[6][11];   // derivative rows, initialize.f90:1959-2031
__constant__ double c_df[2][11];   // filter stencils: [0] 11-point, [1] 7-point

enum { FIRST = 0, MID = 1, LAST = 2 };

template <>
__device__ __forceinline__ double dcoef<double>(int r, int m) {
  return c_dp[r][m];
}
template <>
__device__ __forceinline__ double fcoef<double>(int t, int m) {
  return c_df[t][m];
}

int step_constants() {
  if (cudaMemcpyToSymbol(c_dp, kDerivRows, sizeof(double) * 66) != cudaSuccess)
    return SPARC_ERR_CUDA;
  return SPARC_OK;
}


// ------------------------------------------------ MP_QUIET_3D stage kernel
// One RK stage of the quiet equations (quiet_body.cuh): a block of 32 x 8
// threads per (tile, z chunk), two per SM.  Layer ring: 30 KB a layer with
// the uniform background (three layers), 40 KB with the 3-D one (two).
template <bool BG1D>
struct Quiet64 {
  static constexpr int TY = 8, NS = BG1D ? 3 : 2;
  using Buf = QuietBuf<double, TY, BG1D, NS, false>;
};
template <int MODE, bool BG1D>
__global__ void __launch_bounds__(qg::TX *Quiet64<BG1D>::TY, 2)
    k_quiet64(const SimDev S, const double *__restrict__ a, const double *__restrict__ tin,
              double *__restrict__ so, double beta, double bnext, int zchunk) {
  extern __shared__ __align__(16) double smem_q64[];
  double ke = 0.0, mr = 1e300, mp = 1e300;
  const int k0 = blockIdx.z * zchunk;
  quiet_body<double, Quiet64<BG1D>::TY, MODE, BG1D, Quiet64<BG1D>::NS>(
      S, smem_q64, a, tin, so, beta, bnext, blockIdx.x * qg::TX, blockIdx.y * Quiet64<BG1D>::TY,
      k0, min(S.nz, k0 + zchunk), threadIdx.x, threadIdx.y, ke, mr, mp);
  if (MODE == F_LAST)
    diag_reduce_t(S, ke, mr, mp,
                  blockIdx.x + (long long)gridDim.x *
                                   (blockIdx.y + (long long)gridDim.y * blockIdx.z),
                  (long long)gridDim.x * gridDim.y * gridDim.z);
}

// Layers per z chunk of the quiet kernels: the extent with the least time,
// where a block of zc layers costs zc + 2 layer times (its start and window
// loads), an SM's resident blocks (two in FP64, three in FP32) share its
// issue slots, and a lone block is bound by its own latency (1.3 of a
// shared one's time).  At most 32 layers (256x256x300 FP32: 2.36 ms per
// iteration at 24 and 32, 2.54 at 8; 64x64x128 FP64: 0.122 at the chosen 8,
// 0.148 at 11 and 16, 0.133 at 4), and 8 with x/y CPML slabs, whose tiles
// take longer than the others.  With slabs, ms per iteration at 4 / 8 / 16 /
// 32 layers, 3-D background, FP64 and FP32:
//   64x64x128    0.235 / 0.238 / 0.347 / 0.604   0.180 / 0.167 / 0.247 / 0.445
//   96x96x150    0.466 / 0.484 / 0.571 / 0.690   0.360 / 0.410 / 0.460 / 0.724
//   133x117x171  1.048 / 1.058 / 1.128 / 1.373   0.844 / 0.964 / 1.082 / 1.069
//   192x160x200  1.537 / 1.471 / 1.444 / 1.620   1.143 / 1.189 / 1.204 / 1.414
//   512x64x200   1.649 / 1.578 / 1.552 / 1.699   1.253 / 1.278 / 1.286 / 1.453
//   256x256x300  4.455 / 4.194 / 4.138 / 4.122   3.262 / 3.170 / 3.148 / 3.233
// so that the share of slab tiles hardly matters: wide grids give away 2 % at 8
// and narrow ones would lose up to half at 16.
static int quiet_zchunk(const Handle *h) {
  const int occ = h->fp32 ? 3 : 2, zmax = h->use_hpml ? 8 : QUIET_ZMAX;
  const long long tiles = (long long)((h->nx + 31) / 32) * ((h->ny + 7) / 8);
  int best = std::min(h->nz, zmax);
  double cost = 1e300;
  for (int n = 1; n <= h->nz / 2; ++n) {
    const int zc = (h->nz + n - 1) / n;
    if (zc > zmax) continue;
    const long long blocks = tiles * ((h->nz + zc - 1) / zc);
    const long long full = blocks / (148 * occ), m = (blocks - full * 148 * occ + 147) / 148;
    const double c = (zc + 2) * (full * occ + (m ? std::max<double>(m, 1.3) : 0.0));
    if (c < cost) {
      cost = c;
      best = zc;
    }
  }
  return best;
}

// Layers per z chunk of the MHD kernels: the extent whose items, taken by
// one block per SM in the kernels' order (edge/CPML tiles first), finish
// first, where an item costs its layers and two more (window loads, start)
// and a layer of an edge tile one and a half of an interior one's time
// (measured: 9,600 against 6,100 cycles in FP64, 6,100 against 4,150 in
// FP32).  ms per iteration at the chosen extent and at others (layers): FP64
// 40x40x48 0.184 (4), 0.287 (8), 0.390 (12); 149x151x203 3.21 (52), 3.17 (24), 3.34
// (40), 3.28 (68); 256x256x300 10.31 (76), 10.47 (40), 10.25 (80), 10.80 (100);
// FP32 149x149x211 2.41 (36), 2.47 (24), 2.53 (40), 2.63 (72); 128x160x180
// periodic 1.767 (32), 1.779 (20), 1.787 (40), 1.914 (48).
static int mhd_zchunk(const Handle *h) {
  constexpr int SMS = 148, ROUNDS = 24;
  const sparc_params &P = h->P;
  const bool hp = h->use_hpml;
  const int np[4] = {hp ? P.npml_xb : 0, hp ? P.npml_xt : 0, hp ? P.npml_yb : 0,
                     hp ? P.npml_yt : 0};
  int ix0, ix1, iy0, iy1;
  mhd_interior_rect(h->nx, h->ny, np, ix0, ix1, iy0, iy1);
  const int tiles = ((h->nx + mg::TX - 1) / mg::TX) * ((h->ny + mg::TY - 1) / mg::TY);
  const int nint = ix1 > ix0 && iy1 > iy0 ? (ix1 - ix0) * (iy1 - iy0) : 0, ngen = tiles - nint;
  // without tensor copies an interior FP64 layer costs nearly as much as an edge
  // one (odd rows, which are left unpadded only where padding would pass the
  // 32-bit indexing)
  const double ratio = !h->fp32 && (h->px & 1) ? 1.15 : 1.5;
  int best = std::min(h->nz, 40), last = 0;
  double least = 1e300;
  for (int n = 1; n <= h->nz / mg::KSEG; ++n) {
    const int zc = ((h->nz + n - 1) / n + mg::KSEG - 1) / mg::KSEG * mg::KSEG;
    const int nch = (h->nz + zc - 1) / zc;
    if (zc == last || zc > 160) continue;
    last = zc;
    if ((long long)tiles * nch > SMS * ROUNDS && n > 1) break;
    std::vector<double> free_at(SMS, 0.0);  // a heap, the earliest in front
    double end = 0.0;
    for (int part = 0; part < 2; ++part)
      for (int c = 0; c < nch; ++c) {
        const double cost = (std::min(zc, h->nz - c * zc) + 2) * (part == 0 ? ratio : 1.0);
        for (int t = 0; t < (part == 0 ? ngen : nint); ++t) {
          std::pop_heap(free_at.begin(), free_at.end(), std::greater<double>());
          free_at.back() += cost;
          end = std::max(end, free_at.back());
          std::push_heap(free_at.begin(), free_at.end(), std::greater<double>());
        }
      }
    // extents come longest first; a shorter one has to gain 1 %
    if (end < 0.99 * least) {
      least = end;
      best = zc;
    }
  }
  return best;
}

int stage_geometry(Handle *h) {
  const long long tiles = (long long)((h->nx + 31) / 32) * ((h->ny + 7) / 8);
  int zc;
  zc = h->magnetic ? mhd_zchunk(h) : quiet_zchunk(h);
  zc = std::min(zc, h->nz);
  if (const char *kv = std::getenv("SPARC_ZCHUNK")) {  // A/B timing only
    const int v = std::atoi(kv);
    if (v >= 4) zc = std::min(v, h->nz);
  }
  h->zchunk = h->zchunk0 = zc;
  h->max_stage_blocks = (int)(tiles * ((h->nz + zc - 1) / zc));
  const int zmin = std::min(zc, 11);
  h->partials_blocks = (int)(tiles * ((h->nz + zmin - 1) / zmin));
  return SPARC_OK;
}

static int launch_quiet(Handle *h, const SimDev &S, int stage, const double *a,
                        const double *tin, double *so, cudaStream_t s) {
  const int zc = std::min(h->zchunk, QUIET_ZMAX);
  const dim3 blk(qg::TX, 8);
  const dim3 grd((h->nx + qg::TX - 1) / qg::TX, (h->ny + 7) / 8, (h->nz + zc - 1) / zc);
  const double beta = h->betas[stage - 1];
  const double bnext = stage < 5 ? h->betas[stage] : h->deltat;
  const int mode = stage == 1 ? FIRST : (stage == 5 ? LAST : MID);
#define QL(M, B)                                                                          \
  k_quiet64<M, B><<<grd, blk, Quiet64<B>::Buf::bytes(zc), s>>>(S, a, tin, so, beta, bnext, zc)
  if (S.bg1d) {
    if (mode == FIRST) QL(F_FIRST, true);
    else if (mode == MID) QL(F_MID, true);
    else QL(F_LAST, true);
  } else {
    if (mode == FIRST) QL(F_FIRST, false);
    else if (mode == MID) QL(F_MID, false);
    else QL(F_LAST, false);
  }
#undef QL
  return SPARC_OK;
}

int encode_tensor_maps(Handle *h) {
  h->ftma = false;
  // rows of a multiple of 16 bytes; the filter's tiles read zero outside
  // the grid, so its maps serve non-periodic grids only
  const bool want_f = !h->periodic && !(h->px & 1);
  h->ztma = false;
  const bool want_z = !(h->px & 1);
  h->tma = h->magnetic && !(h->px & 1) && h->allow_tma64 &&
           encode_stage_maps(h, MhdBuf<double, true>::HXL);
  if (!want_f && !want_z) return SPARC_OK;
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) !=
          cudaSuccess || !fn || q != cudaDriverEntryPointSuccess) {
    cudaGetLastError();
    return SPARC_OK;  // the cp.async kernel serves instead
  }
  auto enc = (CUresult(*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                          const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                          const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                          CUtensorMapL2promotion, CUtensorMapFloatOOBfill))fn;
  auto boxed = [&](CUtensorMap *m, const double *base, unsigned long long depth, int bx,
                   int by) {
    cuuint64_t dims[3] = {(cuuint64_t)h->nx, (cuuint64_t)h->ny, (cuuint64_t)depth};
    cuuint64_t strides[2] = {(cuuint64_t)h->px * 8, (cuuint64_t)h->px * h->ny * 8};
    cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, 1};
    cuuint32_t es[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, (void *)base, dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (want_f) {
    // FILTER_VARS xy pass: the 44 x 44 neighbourhood of a 32 x 32 tile
    bool fok = true;
    for (int b = 0; b < 3; ++b)
      fok = fok && boxed(&h->fmaps[b], h->buf[b], (unsigned long long)h->nz * h->V, fb::RX,
                         fb::RY);
    h->ftma = fok;
  }
  if (want_z) {
    // FILTER_VARS z pass: a slab of 32 x 4 columns over 44 layers of one
    // field, in a 4-D view (nx, ny, nz, V), so layers outside [0, nz) read
    // zero instead of the neighbouring field
    bool zok = true;
    for (int b = 0; b < 3 && zok; ++b) {
      cuuint64_t dims[4] = {(cuuint64_t)h->nx, (cuuint64_t)h->ny, (cuuint64_t)h->nz,
                            (cuuint64_t)h->V};
      cuuint64_t strides[3] = {(cuuint64_t)h->px * 8, (cuuint64_t)h->px * h->ny * 8,
                               (cuuint64_t)h->px * h->ny * h->nz * 8};
      cuuint32_t box[4] = {(cuuint32_t)fb::ZX, (cuuint32_t)fb::ZY, (cuuint32_t)fb::ZH, 1};
      cuuint32_t es[4] = {1, 1, 1, 1};
      zok = enc(&h->zmaps[b], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, (void *)h->buf[b], dims,
                strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    h->ztma = zok;
  }
  return SPARC_OK;
}

// The tensor maps of the MHD stage kernels, as TmaSet lists them (both
// precisions: rows of a multiple of 16 bytes; hxl: the columns of a halo
// box).  False where the driver does not give them; the cp.async kernels
// serve then.
bool encode_stage_maps(Handle *h, int hxl) {
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) !=
          cudaSuccess || !fn || q != cudaDriverEntryPointSuccess) {
    cudaGetLastError();
    return false;
  }
  auto enc = (CUresult(*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                          const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                          const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                          CUtensorMapL2promotion, CUtensorMapFloatOOBfill))fn;
  const cuuint64_t w = h->fp32 ? 4 : 8, nx = h->nx, px = h->px, ny = h->ny, nz = h->nz;
  auto one = [&](CUtensorMap *m, void *base, int fields, int bx, int by, int bf) {
    if (!base) return false;
    const cuuint64_t dims[4] = {nx, ny, nz, (cuuint64_t)fields};
    const cuuint64_t strides[3] = {px * w, px * ny * w, px * ny * nz * w};
    const cuuint32_t box[4] = {(cuuint32_t)bx, (cuuint32_t)by, 1, (cuuint32_t)bf};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return enc(m, h->fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4,
               base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  bool ok = true;
  for (int b = 0; b < 3; ++b) {
    void *st = h->fp32 ? (void *)h->fbuf[b] : (void *)h->buf[b];
    ok = ok && one(&h->tmaps.m[b], st, h->V, mg::TX, mg::TY, 1) &&
         one(&h->tmaps.m[3 + b], st, h->V, mg::TX, mg::TY, 8) &&
         one(&h->tmaps.m[6 + b], st, h->V, hxl, mg::HY, 7);
  }
  return ok && one(&h->tmaps.m[9], h->bg_pack, PK_COUNT, mg::TX, mg::TY, 13) &&
         one(&h->tmaps.m[10], h->bg_pack, PK_COUNT, mg::TX, mg::TY, 1) &&
         one(&h->tmaps.m[11], h->bg_pack, PK_COUNT, hxl, mg::HY, 3) &&
         one(&h->tmaps.m[12], h->bg_pack, PK_COUNT, mg::TX, mg::TY, 3);
}

// ------------------------- MP_MHD_3D, shared-body stage kernel

// One FP64 MHD RK stage as a single persistent launch: each CTA (one per
// SM) allocates its tensor memory once and pulls work items (32x8 tile, z
// chunk) from a device counter until the list is done.  The edge/CPML
// tiles' items come first (they are the slower ones, so the last items to
// start are short), each list chunk-major so that neighbouring tiles of a
// chunk run together; interior tiles take the branch-free body, the others
// the general one, both with TMA halo planes (TH; not where halos wrap).  The diagnostics partials are
// per work item (the last stage reduces each item in the CTA and the item
// that finishes last sums them in item order), so the norm does not depend
// on which CTA took which item.
template <int MODE, bool TMA, bool TH>
__global__ void __launch_bounds__(mg::NT, 1)
    k_mhd64p(const SimDev S, const __grid_constant__ TmaSet T, const double *__restrict__ a,
             const double *__restrict__ tin, double *__restrict__ so, double beta,
             double bnext, int zchunk, int mt, int ma, int ix0, int iy0, int nix, int nint,
             int ngen, const int2 *__restrict__ gen, unsigned *ctr) {
  const int nch = (S.nz + zchunk - 1) / zchunk;
  extern __shared__ __align__(1024) double smem_raw64[];
  double *smem = (double *)(((size_t)smem_raw64 + 127) & ~(size_t)127);
  __shared__ uint32_t s_tmem;
  __shared__ int s_w;
  __shared__ unsigned long long bar[2];
  unsigned phase = 0;
  const int tid = (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
  const int warp = tid / 32;
  if (warp == 0) {
    if (TMA && tid == 0) mhd_bars_init(bar);
    __syncwarp();
    tm_alloc_all(&s_tmem);
  }
  tm_fence_before();
  __syncthreads();
  tm_fence_after();
  const uint32_t tbase = s_tmem, tw = tm_warp_addr(tbase, warp);
  const int ngi = ngen * nch, total = (ngen + nint) * nch;
  bool ok = true;
  for (;;) {
    if (tid == 0) s_w = (int)atomicAdd(ctr, 1u);
    __syncthreads();
    const int w = s_w;
    if (w >= total) break;
    int x0, y0, c;
    const bool in = w >= ngi;
    if (!in) {
      c = w / ngen;
      const int2 g = gen[w - c * ngen];
      x0 = g.x * mg::TX;
      y0 = g.y * mg::TY;
    } else {
      const int w2 = w - ngi;
      c = w2 / nint;
      const int t = w2 - c * nint;
      const int ty = t / nix;
      x0 = (ix0 + t - ty * nix) * mg::TX;
      y0 = (iy0 + ty) * mg::TY;
    }
    const int k0 = c * zchunk, k1 = min(S.nz, k0 + zchunk);
    // the body's first barrier orders every thread's read of s_w before
    // thread 0 takes the next item
    double ke = 0.0, mr = 1e300, mp = 1e300;
    const int tiles = ngen + nint;
    double *kseg = S.kseg + (y0 / mg::TY) * ((S.nx + mg::TX - 1) / mg::TX) + x0 / mg::TX;
    if (in)
      ok = mhd_body<double, MODE, TMA, true, TMA, true>(S, &T, smem, a, tin, so, beta, bnext, x0,
                                                        y0, k0, k1, mt, ma, ke, mr, mp, bar, phase,
                                                        tw, kseg, tiles);
    else
      ok = mhd_body<double, MODE, TMA, false, TH, true>(S, &T, smem, a, tin, so, beta, bnext, x0,
                                                        y0, k0, k1, mt, ma, ke, mr, mp, bar, phase,
                                                        tw, kseg, tiles);
    if (!ok) break;
    if (MODE == F_LAST) diag_reduce_mhd(S, mr, mp, w, total, tiles, zchunk);
  }
  __syncwarp();
  tm_wait_st();
  tm_fence_before();
  __syncthreads();
  tm_fence_after();
  if (warp == 0) tm_free_all(tbase);
}

// The persistent launch's plan: the edge/CPML tiles (all tiles outside the
// interior rectangle), a work counter per stage (cleared at the start of
// each step), one CTA per SM.
int mhd64_plan(Handle *h) {
  if (!h->magnetic || h->fp32) return SPARC_OK;
  const int np[4] = {h->faces[2].on ? h->faces[2].np : 0, h->faces[3].on ? h->faces[3].np : 0,
                     h->faces[4].on ? h->faces[4].np : 0, h->faces[5].on ? h->faces[5].np : 0};
  int ix0, ix1, iy0, iy1;
  mhd_interior_rect(h->nx, h->ny, np, ix0, ix1, iy0, iy1);
  const int gx = (h->nx + mg::TX - 1) / mg::TX, gy = (h->ny + mg::TY - 1) / mg::TY;
  const bool has_int = ix1 > ix0 && iy1 > iy0;
  std::vector<int2> gen;
  for (int ty = 0; ty < gy; ++ty)
    for (int tx = 0; tx < gx; ++tx)
      if (!(has_int && tx >= ix0 && tx < ix1 && ty >= iy0 && ty < iy1))
        gen.push_back(make_int2(tx, ty));
  h->gix0 = has_int ? ix0 : 0;
  h->giy0 = has_int ? iy0 : 0;
  h->gnix = has_int ? ix1 - ix0 : 0;
  h->gniy = has_int ? iy1 - iy0 : 0;
  h->ngen = (int)gen.size();
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
  h->pgrid = sms;
  h->d_wctr64 = (unsigned *)dev_alloc(h, 8 * sizeof(unsigned));
  if (!h->d_wctr64) return SPARC_ERR_NOMEM;
  if (!gen.empty()) {
    h->d_gen = (int2 *)dev_alloc(h, gen.size() * sizeof(int2));
    if (!h->d_gen) return SPARC_ERR_NOMEM;
    if (cudaMemcpy(h->d_gen, gen.data(), gen.size() * sizeof(int2), cudaMemcpyHostToDevice) !=
        cudaSuccess)
      return SPARC_ERR_CUDA;
  }
  return cudaMemset(h->d_wctr64, 0, 8 * sizeof(unsigned)) == cudaSuccess ? SPARC_OK
                                                                        : SPARC_ERR_CUDA;
}

static int launch_mhd64p(Handle *h, const SimDev &S, int stage, const double *a,
                         const double *tin, double *so, cudaStream_t s) {
  const double beta = h->betas[stage - 1];
  const double bnext = stage < 5 ? h->betas[stage] : h->deltat;
  const int mode = stage == 1 ? FIRST : (stage == 5 ? LAST : MID);
  const bool tma = h->tma;
  // halo boxes for the edge tiles too, except where their halos wrap
  const bool th = tma && !h->periodic;
  const size_t sm = tma ? MhdBuf<double, true>::SMEM_GEN : MhdBuf<double>::SMEM_GEN;
  static_assert(MhdBuf<double, true>::SMEM_GEN + 1024 <= 227 * 1024, "shared memory of an SM");
  int mt = -1, ma = -1;
  for (int b = 0; b < 3; ++b) {
    if (h->buf[b] == tin) mt = b;
    if (h->buf[b] == a) ma = b;
  }
  if (mt < 0 || ma < 0 || !h->d_wctr64) return SPARC_ERR_INVALID;
  TmaSet T;
  if (tma)
    T = h->tmaps;
  else
    std::memset(&T, 0, sizeof(T));
  const int nch = (h->nz + h->zchunk - 1) / h->zchunk;
  const int nint = h->gnix * h->gniy;
  const long long total = (long long)(h->ngen + nint) * nch;
  const int grid = (int)std::min<long long>(h->pgrid, total);
  unsigned *ctr = h->d_wctr64 + (stage - 1);
  const dim3 blk(mg::TX, mg::TY, 2);
#define MP64(M, U, H)                                                                        \
  k_mhd64p<M, U, H><<<grid, blk, sm, s>>>(S, T, a, tin, so, beta, bnext, h->zchunk, mt, ma,   \
                                      h->gix0, h->giy0, h->gnix, nint, h->ngen, h->d_gen, ctr)
  if (th) {
    if (mode == FIRST) MP64(F_FIRST, true, true);
    else if (mode == MID) MP64(F_MID, true, true);
    else MP64(F_LAST, true, true);
  } else if (tma) {
    if (mode == FIRST) MP64(F_FIRST, true, false);
    else if (mode == MID) MP64(F_MID, true, false);
    else MP64(F_LAST, true, false);
  } else {
    if (mode == FIRST) MP64(F_FIRST, false, false);
    else if (mode == MID) MP64(F_MID, false, false);
    else MP64(F_LAST, false, false);
  }
#undef MP64
  return SPARC_OK;
}

// The stage kernels that the handle launches, allowed their shared memory
// (after encode_tensor_maps).
int stage_limits(Handle *h) {
  int r = SPARC_OK;
#define LIM(K, ...) \
  r |= allow_smem(K<F_FIRST, __VA_ARGS__>) | allow_smem(K<F_MID, __VA_ARGS__>) | \
       allow_smem(K<F_LAST, __VA_ARGS__>)
  if (!h->magnetic) {
    if (h->bg1d) LIM(k_quiet64, true);
    else LIM(k_quiet64, false);
  } else if (h->tma && !h->periodic) {
    LIM(k_mhd64p, true, true);
  } else if (h->tma) {
    LIM(k_mhd64p, true, false);
  } else {
    LIM(k_mhd64p, false, false);
  }
#undef LIM
  return r ? SPARC_ERR_CUDA : SPARC_OK;
}

int launch_stage(Handle *h, const SimDev &S, int stage, const double *a,
                 const double *tin, double *so, cudaStream_t s) {
  int r = SPARC_ERR_INVALID;
  r = h->magnetic ? launch_mhd64p(h, S, stage, a, tin, so, s)
                  : launch_quiet(h, S, stage, a, tin, so, s);
  ++h->launches;
  if (r == SPARC_OK && cudaGetLastError() != cudaSuccess) r = SPARC_ERR_CUDA;
  return r;
}

// ------------------------------------------------------- PULSE = 2 forcing
// The layers that carry any pulse (psr_forcing.cuh).
struct PsrDev {
  int nx, ny, nz, klo, npulses, nblocks;
  long long init;
  double timestep, st;
  const int *off, *idx;
  const double *zv, *px, *py, *ptime, *sd, *ssb;
  const unsigned char *mask;
  const int *colx, *coly, *colz;
  int bx, bxy;
  double *out;
  const long long *iter;
};

__global__ void __launch_bounds__(256) k_psr(PsrDev D) {
  extern __shared__ double sh[];
  psr_tile<double>(D, sh, D.npulses);
}

int launch_psr_forcing(Handle *h, const SimDev &S, cudaStream_t s);

// ------------------------------------------------------ FILTER_VARS
// FILTER_VARS of a filter event (filter_body.cuh): the fused y-then-x pass
// (blockIdx.z: field and a group of LPB layers, pipelined)
template <int G, bool TMA>
__global__ void __launch_bounds__(fb::NT, 4)
    k_filt_xy64(FiltArgs<double> F, const __grid_constant__ CUtensorMap map) {
  const int nzc = (F.nz + fb::LPB - 1) / fb::LPB;
  const int l = blockIdx.z / nzc, k0 = (blockIdx.z - l * nzc) * fb::LPB;
  filt_xy_layers<double, G, TMA>(F, l, k0, min(fb::LPB, F.nz - k0), blockIdx.x * fb::TX,
                                 blockIdx.y * fb::TR, &map);
}
// the z pass: blockIdx.x is the z chunk (the chunks of a slab run
// together), blockIdx.y the slab of the layer, blockIdx.z the field
// (the launch gives 128 bytes of slack for a 128-byte aligned slab and 16
// for the mbarrier after it)
template <int G, bool TMA>
__global__ void __launch_bounds__(2 * fb::ZX * fb::ZY)
    k_filt_z64(FiltArgs<double> F, const __grid_constant__ CUtensorMap map) {
  extern __shared__ __align__(128) unsigned char zraw64[];
  double *zsl = (double *)(zraw64 + ((128u - (sm_addr_t(zraw64) & 127u)) & 127u));
  const int nxb = (F.nx + fb::ZX - 1) / fb::ZX;
  const int yb = blockIdx.y / nxb, xb = blockIdx.y - yb * nxb;
  filt_z_slab<double, G, false, false, TMA>(F, blockIdx.z, xb * fb::ZX, yb * fb::ZY,
                                            blockIdx.x * fb::ZC, zsl, &map);
}

// xy: the y and x passes fused; z: the z pass (in -> out, never in place)
int launch_filter_event(Handle *h, bool xy, const double *in, double *out, cudaStream_t s) {
  FiltArgs<double> F{};
  F.nx = h->nx; F.ny = h->ny; F.nz = h->nz; F.px = h->px; F.V = h->V; F.N = h->NP;
  F.periodic = h->periodic ? 1 : 0;
  F.s = xy ? h->P.s_xy : h->P.s_z;
  F.in = in;
  F.out = out;
  F.err = h->d_err;
  const int g = xy ? h->gxy : h->gz;
  if (xy) {
    const dim3 grid((h->nx + fb::TX - 1) / fb::TX, (h->ny + fb::TR - 1) / fb::TR,
                    h->V * ((h->nz + fb::LPB - 1) / fb::LPB));
    // the tensor map of the input buffer (neighbourhoods by TMA), if any
    int mb = -1;
    if (h->ftma)
      for (int b = 0; b < 3; ++b)
        if (h->buf[b] == in) mb = b;
    CUtensorMap map;
    if (mb >= 0) map = h->fmaps[mb];
    else std::memset(&map, 0, sizeof(map));
    const dim3 blk(fb::TX, fb::TY);
    if (mb >= 0) {
      if (g == 5) k_filt_xy64<5, true><<<grid, blk, 0, s>>>(F, map);
      else k_filt_xy64<3, true><<<grid, blk, 0, s>>>(F, map);
    } else {
      if (g == 5) k_filt_xy64<5, false><<<grid, blk, 0, s>>>(F, map);
      else k_filt_xy64<3, false><<<grid, blk, 0, s>>>(F, map);
    }
  } else {
    const size_t zs = filt_z_smem<double>() + 128 + 16;
    const long long slabs = (long long)((h->nx + fb::ZX - 1) / fb::ZX) *
                            ((h->ny + fb::ZY - 1) / fb::ZY);
    if (slabs > 65535) return SPARC_ERR_INVALID;
    const dim3 grid((h->nz + fb::ZC - 1) / fb::ZC, (unsigned)slabs, h->V);
    // the tensor map of the input buffer (slabs by TMA), if any
    int mb = -1;
    if (h->ztma)
      for (int b = 0; b < 3; ++b)
        if (h->buf[b] == in) mb = b;
    CUtensorMap map;
    if (mb >= 0) map = h->zmaps[mb];
    else std::memset(&map, 0, sizeof(map));
    const dim3 blk(fb::ZX, fb::ZY, 2);
#define ZP(GG, TT)                                                                          \
  do {                                                                                      \
    cudaFuncSetAttribute(k_filt_z64<GG, TT>, cudaFuncAttributeMaxDynamicSharedMemorySize,   \
                         (int)zs);                                                          \
    k_filt_z64<GG, TT><<<grid, blk, zs, s>>>(F, map);                                       \
  } while (0)
    if (mb >= 0) {
      if (g == 5) ZP(5, true);
      else ZP(3, true);
    } else {
      if (g == 5) ZP(5, false);
      else ZP(3, false);
    }
#undef ZP
  }
  ++h->launches;
  return cudaGetLastError() == cudaSuccess ? SPARC_OK : SPARC_ERR_CUDA;
}

// Both stencils stay resident, so handles with different filter modes can
// coexist; a pass picks its table by half-width.
int filter_constants() {
  double t[2][11] = {};
  for (int m = 0; m < 11; ++m) t[0][m] = kFilter11[m];
  for (int m = 0; m < 7; ++m) t[1][m] = kFilter7[m];
  return cudaMemcpyToSymbol(c_df, t, sizeof(t)) == cudaSuccess ? SPARC_OK
                                                               : SPARC_ERR_CUDA;
}

// PULSE = 0: the forcing plane of the device's iteration
// (random_forcing.cuh), one value per column.
template <class D, class T>
__global__ void k_random(const double *__restrict__ vr, const D *__restrict__ damp, int nxy,
                         int ns, double timestep, double cad, const long long *iter,
                         T *__restrict__ out) {
  const RndStencil R = rnd_stencil(*iter, timestep, cad, ns);
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nxy; q += gridDim.x * blockDim.x)
    out[q] = (T)rnd_column(R, vr, nxy, q, damp[q]);
}

int launch_random_forcing(Handle *h, cudaStream_t s) {
  if (h->src.kind != SPARC_SRC_RANDOM) return SPARC_OK;
  const int nxy = h->nx * h->ny;
  const int grid = std::min((nxy + 255) / 256, 4 * 148);
  if (h->fp32)
    k_random<float, float><<<grid, 256, 0, s>>>(h->d_series, h->f_sd, nxy, h->src.nseries,
                                               h->P.timestep, h->src.cadforcing, h->d_iter,
                                               h->f_f2d);
  else
    k_random<double, double><<<grid, 256, 0, s>>>(h->d_series, h->source_damp, nxy,
                                                 h->src.nseries, h->P.timestep,
                                                 h->src.cadforcing, h->d_iter, h->d_f2d);
  ++h->launches;
  return cudaGetLastError() == cudaSuccess ? SPARC_OK : SPARC_ERR_CUDA;
}

int launch_psr_forcing(Handle *h, const SimDev &S, cudaStream_t s) {
  (void)S;
  if (h->src.kind != SPARC_SRC_PSR || h->psr_khi <= h->psr_klo) return SPARC_OK;
  PsrDev D;
  D.nx = h->nx; D.ny = h->ny; D.nz = h->nz;
  D.klo = h->psr_klo;
  D.npulses = (int)h->pulses.size();
  D.nblocks = h->nblocks;
  D.init = h->src.init;
  D.timestep = h->P.timestep;
  D.st = h->src.psr_st;
  D.off = h->d_plane_off;
  D.idx = h->d_plane_idx;
  D.zv = h->d_plane_z;
  D.px = h->d_px;
  D.py = h->d_py;
  D.ptime = h->d_ptime;
  D.sd = h->source_damp;
  D.ssb = h->ssb;
  D.mask = h->d_pmask;
  D.colx = h->d_colx;
  D.coly = h->d_coly;
  D.colz = h->d_colx + h->nx + h->ny;  // packed after colx, coly
  D.bx = h->P.block_x;
  D.bxy = h->P.block_x * h->P.block_y;
  D.out = h->d_psr;
  D.iter = h->d_iter;
  dim3 blk(32, 8);
  dim3 grd((h->nx + 31) / 32, (h->ny + 7) / 8, h->psr_khi - h->psr_klo);
  size_t smem = (size_t)D.npulses * (sizeof(double) + sizeof(int));
  k_psr<<<grd, blk, smem, s>>>(D);
  ++h->launches;
  return cudaGetLastError() == cudaSuccess ? SPARC_OK : SPARC_ERR_CUDA;
}

SimDev make_simdev(Handle *h) {
  SimDev S{};
  S.nx = h->nx; S.ny = h->ny; S.nz = h->nz; S.px = h->px; S.N = h->NP;
  S.periodic = h->periodic ? 1 : 0;
  S.magnetic = h->magnetic ? 1 : 0;
  S.bg1d = h->bg1d ? 1 : 0;
  S.sponge_slabs = h->sponge_slabs ? 1 : 0;
  S.V = h->V;
  S.stretchx = h->stretchx;
  S.stretchy = h->stretchy;
  S.stretch = h->d_stretch;
  S.deltat = h->deltat;
  S.dimc2rho = (h->dimc * h->dimc) * h->dimrho;
  S.term = h->damping ? h->d_term : nullptr;
  if (h->bg1d) {
    S.rho0 = h->rho0_1; S.p0 = h->p0_1; S.rhoinv = h->rhoinv_1;
    S.c2rho0 = h->c2rho0_1; S.grz = h->grz_1; S.gpz = h->gpz_1;
    S.sponge = h->sponge_1;
  } else {
    S.rho0 = h->rho0; S.p0 = h->p0; S.rhoinv = h->rhoinv;
    S.c2rho0 = h->c2rho0; S.grz = h->grz; S.gpz = h->gpz;
    S.sponge = h->sponge;
  }
  S.box = h->box; S.boy = h->boy; S.boz = h->boz;
  S.cbx = h->cbx; S.cby = h->cby; S.cbz = h->cbz;
  S.grx = h->grx; S.gry = h->gry; S.gpx = h->gpx; S.gpy = h->gpy;
  S.red = h->red;
  S.gblk = h->d_gblk;
  S.colx = h->d_colx;
  S.coly = h->d_coly;
  S.bxdim = h->P.block_x;
  S.zb = h->faces[0]; S.zt = h->faces[1];
  S.xb = h->faces[2]; S.xt = h->faces[3];
  S.yb = h->faces[4]; S.yt = h->faces[5];
  ForcingDev &F = S.frc;
  F.kind = h->src.kind;
  F.dir = h->src.dir;
  F.init = h->src.init;
  F.fx = h->d_fx; F.fy = h->d_fy; F.fz = h->d_fz;
  F.amp_c = h->src.amp / 0.56458272 / h->dimc;
  F.t0 = h->src.t0; F.t1 = h->src.t1; F.st = h->src.st;
  F.timestep = h->P.timestep;
  F.psr = h->d_psr;
  F.klo = h->psr_klo;
  F.khi = h->psr_khi;
  F.f2d = h->d_f2d;
  F.sdep = h->d_sdep;
  S.iter = h->d_iter;
  S.err = h->d_err;
  S.partials = h->d_partials;
  S.kseg = h->d_kseg;
  S.counter = h->d_counter;
  S.diag = h->d_diag;
  S.fail_iter = h->d_fail;
  return S;
}

}  // namespace sparc
