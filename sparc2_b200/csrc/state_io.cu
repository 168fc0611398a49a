// state_io.cu -- the state between host and device (sparc_set_state,
// sparc_get_state): staged copies of large pageable arrays, and the
// precision form's conversions.
//
// A copy between device memory and a caller's pageable array runs at about
// 4 GB/s when the driver stages it on one thread (the 1.26 GB state of
// 256x256x300 FP64 took 0.31 s to read).  Large copies are therefore cut
// into pieces that several host threads move through a pinned slab: each
// thread keeps one piece on the wire while it copies the other to or from
// the caller's memory, so the page faults of a fresh array are taken in
// parallel too.  The slab is shared by the process's handles, allocated at
// the first large copy, used by one copy at a time (another one meanwhile
// takes the plain path) and freed with the last handle.  Pinned arrays and
// small ones go by a plain copy.
//
// The precision form's state is converted on the device: stored FP32 values
// and carries to FP64 physical values in the two free state buffers (which
// hold nothing between iterations), 8 bytes per value on the wire either
// way, in place of two host passes over two FP32 copies (0.61 s before).

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "internal.h"

namespace sparc {

namespace {

constexpr size_t PIECE = 1u << 20;      // bytes of a piece (a 32 MB slab: pinning
                                        // the 64 MB of 2 MB pieces took 40 ms, and
                                        // 512 KB pieces move 20 % slower)
constexpr int THREADS = 16;             // host threads of a copy at most
constexpr size_t SMALL = 32u << 20;     // below: one plain copy (21 MB: 1.1 ms
                                        // plain, 2.0 ms staged)

std::mutex g_mu;       // handle count and slab pointer
std::mutex g_use;      // held by the copy that uses the slab
int g_handles = 0;
char *g_slab = nullptr;

// the slab, or null where it cannot be had (the caller holds g_use)
char *slab() {
  std::lock_guard<std::mutex> l(g_mu);
  if (!g_slab &&
      cudaHostAlloc((void **)&g_slab, 2 * THREADS * PIECE, cudaHostAllocPortable) !=
          cudaSuccess) {
    cudaGetLastError();
    g_slab = nullptr;
  }
  return g_slab;
}

// pageable memory as the driver sees it (registered and pinned memory copies
// asynchronously by itself)
bool pageable(const void *p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

// One thread's share of a staged copy: pieces taken from a shared counter,
// two in flight through its own two slots.
struct Staged {
  char *host, *dev;
  size_t bytes;
  bool up;          // host to device
  int device;
  char *slab;
  std::atomic<size_t> next{0};
  std::atomic<int> bad{0};

  void run(int t) {
    if (cudaSetDevice(device) != cudaSuccess) {
      bad = 1;
      return;
    }
    cudaStream_t s = nullptr;
    cudaEvent_t e[2] = {nullptr, nullptr};
    bool ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
    for (int i = 0; ok && i < 2; ++i)
      ok = cudaEventCreateWithFlags(&e[i], cudaEventDisableTiming) == cudaSuccess;
    char *slot[2] = {slab + (size_t)(2 * t) * PIECE, slab + (size_t)(2 * t + 1) * PIECE};
    size_t at[2] = {0, 0}, len[2] = {0, 0};
    const size_t pieces = (bytes + PIECE - 1) / PIECE;
    auto drain = [&](int i) {  // finishes the piece in slot i
      if (!len[i]) return;
      ok = cudaEventSynchronize(e[i]) == cudaSuccess && ok;
      if (ok && !up) std::memcpy(host + at[i], slot[i], len[i]);
      len[i] = 0;
    };
    for (int i = 0; ok && !bad; i ^= 1) {
      const size_t p = next.fetch_add(1);
      if (p >= pieces) break;
      drain(i);
      if (!ok) break;
      at[i] = p * PIECE;
      len[i] = std::min(PIECE, bytes - at[i]);
      if (up) std::memcpy(slot[i], host + at[i], len[i]);
      ok = cudaMemcpyAsync(up ? dev + at[i] : slot[i], up ? slot[i] : dev + at[i], len[i],
                           up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost,
                           s) == cudaSuccess &&
           cudaEventRecord(e[i], s) == cudaSuccess;
      if (!up) drain(i ^ 1);
    }
    drain(0);
    drain(1);
    if (s && cudaStreamSynchronize(s) != cudaSuccess) ok = false;
    for (int i = 0; i < 2; ++i)
      if (e[i]) cudaEventDestroy(e[i]);
    if (s) cudaStreamDestroy(s);
    if (!ok) bad = 1;
  }
};

int state_copy(Handle *h, void *host, void *dev, size_t bytes, bool up) {
  if (bytes >= SMALL && pageable(host)) {
    std::unique_lock<std::mutex> use(g_use, std::try_to_lock);
    char *sl = use.owns_lock() ? slab() : nullptr;
    if (sl) {
      // the worker streams are not ordered with the handle's
      if (!cuda_ok(h, cudaStreamSynchronize(h->stream), "state copy")) return SPARC_ERR_CUDA;
      Staged S;
      S.host = (char *)host;
      S.dev = (char *)dev;
      S.bytes = bytes;
      S.up = up;
      S.device = h->device;
      S.slab = sl;
      const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
      const int n = (int)std::min<size_t>(std::min<unsigned>(THREADS, hw), bytes / PIECE);
      std::vector<std::thread> th;
      try {
        th.reserve(n);
        for (int t = 1; t < n; ++t) th.emplace_back([&S, t] { S.run(t); });
      } catch (...) {  // fewer threads: the pieces are shared out by a counter
      }
      S.run(0);
      for (auto &t : th) t.join();
      return cuda_ok(h, S.bad ? cudaErrorUnknown : cudaSuccess, "staged state copy")
                 ? SPARC_OK
                 : SPARC_ERR_CUDA;
    }
  }
  return cuda_ok(h,
                 cudaMemcpyAsync(up ? dev : host, up ? host : dev, bytes,
                                 up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost,
                                 h->stream),
                 "state copy") &&
                 cuda_ok(h, cudaStreamSynchronize(h->stream), "state copy")
             ? SPARC_OK
             : SPARC_ERR_CUDA;
}

}  // namespace

void state_io_open() {
  std::lock_guard<std::mutex> l(g_mu);
  ++g_handles;
}

void state_io_close() {
  // no copy is in flight where no handle is left; otherwise the slab stays, and
  // another handle's copy is not waited for
  std::lock_guard<std::mutex> l(g_mu);
  if (--g_handles == 0 && g_slab) {
    cudaFreeHost(g_slab);
    g_slab = nullptr;
  }
}

int state_to_host(Handle *h, double *host, const void *dev, size_t count) {
  return state_copy(h, host, const_cast<void *>(dev), count * 8, false);
}
int state_to_device(Handle *h, void *dev, const double *host, size_t count) {
  return state_copy(h, const_cast<double *>(host), dev, count * 8, true);
}

// rows of nx values, sp apart at the source, dp apart at the destination
__global__ void k_repitch(const double *__restrict__ src, int sp, double *__restrict__ dst, int dp,
                          int nx, long long rows) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (long long r = (long long)blockIdx.x * nw + warp; r < rows; r += (long long)gridDim.x * nw)
    for (int i = lane; i < nx; i += 32) dst[r * dp + i] = src[r * sp + i];
}

int repitch(const double *src, int sp, double *dst, int dp, int nx, long long rows,
            cudaStream_t s) {
  k_repitch<<<(unsigned)std::min<long long>((rows + 7) / 8, 148 * 16), 256, 0, s>>>(src, sp, dst,
                                                                                  dp, nx, rows);
  return cudaGetLastError() == cudaSuccess ? SPARC_OK : SPARC_ERR_CUDA;
}

// plain form: rows px apart on the device, packed in a free buffer on the way
int set_state64(Handle *h, const double *a) {
  double *st = h->buf[h->ra], *tmp = h->buf[h->rf1];
  const size_t n = (size_t)h->V * h->N;
  if (h->px == h->nx) return state_to_device(h, st, a, n);
  const int r = state_to_device(h, tmp, a, n);
  return r ? r
           : repitch(tmp, h->nx, st, h->px, h->nx, (long long)h->V * h->ny * h->nz, h->stream);
}
int get_state64(Handle *h, double *a) {
  const double *st = h->buf[h->ra];
  double *tmp = h->buf[h->rf1];
  if (h->px != h->nx) {
    if (repitch(st, h->px, tmp, h->nx, h->nx, (long long)h->V * h->ny * h->nz, h->stream))
      return SPARC_ERR_CUDA;
    st = tmp;
  }
  return state_to_host(h, a, st, (size_t)h->V * h->N);
}

// ------------------------------------------------ precision form
// Values [0, half) of the FP64 image lie in lo, the others in hi (the two
// free state buffers).  One (field, layer) plane per block and step, a row
// per warp; device rows are px apart.
__global__ void k_state_out(const float *__restrict__ st, const float *__restrict__ carry,
                            const float *__restrict__ isc, int planes, int nx, int ny, int px,
                            long long half, double *__restrict__ lo, double *__restrict__ hi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int p = blockIdx.x; p < planes; p += gridDim.x) {
    const double q = (double)isc[p];
    for (int j = warp; j < ny; j += nw) {
      const long long row = (long long)p * ny + j;
      for (int i = lane; i < nx; i += 32) {
        const long long t = row * nx + i, d = row * px + i;
        const double v = ((double)st[d] - (double)carry[d]) * q;
        if (t < half) lo[t] = v;
        else hi[t - half] = v;
      }
    }
  }
}
__global__ void k_state_in(const double *__restrict__ lo, const double *__restrict__ hi,
                           const float *__restrict__ sc, int planes, int nx, int ny, int px,
                           long long half, float *__restrict__ st) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int p = blockIdx.x; p < planes; p += gridDim.x) {
    const double q = (double)sc[p];
    for (int j = warp; j < ny; j += nw) {
      const long long row = (long long)p * ny + j;
      for (int i = lane; i < nx; i += 32) {
        const long long t = row * nx + i;
        st[row * px + i] = (float)(q * (t < half ? lo[t] : hi[t - half]));
      }
    }
  }
}
__global__ void k_widen(const float *__restrict__ in, long long n, double *__restrict__ out) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    out[t] = (double)in[t];
}
__global__ void k_narrow(const double *__restrict__ in, long long n, float *__restrict__ out) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    out[t] = (float)in[t];
}

#define CKS(x)                                                 \
  do {                                                         \
    if (!cuda_ok(h, (x), "state conversion")) return SPARC_ERR_CUDA; \
  } while (0)

// (A face's CPML fields fit in a free buffer, half the state in FP64: a slab is
// no thicker than the boundary block, 12 of 23 points at most, so its 6 (quiet: 2)
// fields are below 3.2 (1.1) state fields, and a buffer holds 4 (2.5).)
// stored = float(sc * a), carry 0
int set_state32(Handle *h, const double *a, const double *psi) {
  const long long VN = (long long)h->V * h->N, half = VN / 2;
  double *lo = (double *)h->fbuf[h->rf1], *hi = (double *)h->fbuf[h->rf2];
  const int planes = h->V * h->nz;
  int r;
  if (a) {
    if ((r = state_to_device(h, lo, a, half))) return r;
    if ((r = state_to_device(h, hi, a + half, VN - half))) return r;
    k_state_in<<<std::min(planes, 148 * 16), 256, 0, h->stream>>>(
        lo, hi, h->f_sc, planes, h->nx, h->ny, h->px, half, h->fbuf[h->ra]);
    CKS(cudaGetLastError());
    CKS(cudaMemsetAsync(h->f_carry, 0, (size_t)h->V * h->NP * 4, h->stream));
    CKS(cudaStreamSynchronize(h->stream));
  }
  if (psi)
    for (auto &F : h->f_faces)
      if (F.on) {
        const long long n = F.cnt * F.P;
        if ((r = state_to_device(h, lo, psi, n))) return r;
        k_narrow<<<148 * 4, 256, 0, h->stream>>>(lo, n, F.vars);
        CKS(cudaGetLastError());
        CKS(cudaStreamSynchronize(h->stream));
        psi += n;
      }
  return SPARC_OK;
}

// a = (stored - carry) / sc
int get_state32(Handle *h, double *a, double *psi) {
  const long long VN = (long long)h->V * h->N, half = VN / 2;
  double *lo = (double *)h->fbuf[h->rf1], *hi = (double *)h->fbuf[h->rf2];
  const int planes = h->V * h->nz;
  int r;
  if (a) {
    k_state_out<<<std::min(planes, 148 * 16), 256, 0, h->stream>>>(
        h->fbuf[h->ra], h->f_carry, h->f_isc, planes, h->nx, h->ny, h->px, half, lo, hi);
    CKS(cudaGetLastError());
    if ((r = state_to_host(h, a, lo, half))) return r;
    if ((r = state_to_host(h, a + half, hi, VN - half))) return r;
  }
  if (psi)
    for (auto &F : h->f_faces)
      if (F.on) {
        const long long n = F.cnt * F.P;
        k_widen<<<148 * 4, 256, 0, h->stream>>>(F.vars, n, lo);
        CKS(cudaGetLastError());
        if ((r = state_to_host(h, psi, lo, n))) return r;
        psi += n;
      }
  return SPARC_OK;
}

}  // namespace sparc
