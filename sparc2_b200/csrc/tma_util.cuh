// tma_util.cuh -- shared-memory addresses, mbarriers and 3-D / 4-D TMA
// tile loads (cp.async.bulk.tensor, each into the issuing CTA's own shared
// memory), used by the stage and filter kernels.  Every wait on an
// mbarrier is bounded.
#pragma once

#include "internal.h"

namespace sparc {

// A wait on an mbarrier gives up and raises the error flag after kMbarWaitNs
// of the global timer (copies land within microseconds; another context's time
// slices may come in between), or after kMbarWaitLimit polls where that timer
// stands still.  Polls alone are no bound on time: each may itself suspend.
constexpr unsigned kMbarWaitLimit = 1u << 26;
constexpr unsigned kMbarWaitNs = 1000000000u;

__device__ __forceinline__ unsigned sm_addr_t(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init_t(unsigned long long *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_addr_t(bar)) : "memory");
}
__device__ __forceinline__ void mbar_tx_t(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sm_addr_t(bar)),
               "r"(bytes)
               : "memory");
}
// one 3-D tile of the tensor map at (x, y, z) into shared memory at dst,
// completing on bar.  x times the element size must be a multiple of 16
// bytes; coordinates outside the tensor read zero.
__device__ __forceinline__ void tma3d_t(void *dst, const CUtensorMap *map, int x, int y, int z,
                                        unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(sm_addr_t(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(sm_addr_t(bar))
      : "memory");
}
// the same for a 4-D tile at (x, y, z, w)
__device__ __forceinline__ void tma4d_t(void *dst, const CUtensorMap *map, int x, int y, int z,
                                        int w, unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(sm_addr_t(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(sm_addr_t(bar))
      : "memory");
}
// brings the 4-D tile into L2 (no shared memory, no completion)
__device__ __forceinline__ void tma4d_l2(const CUtensorMap *map, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global [%0, {%1, %2, %3, %4}];" ::"l"(map),
               "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
// Polls `done` until it is true, at most `polls` times and about `ns` of the
// clock `now` (32 bits of nanoseconds, read every 64 polls: waits that end soon
// do not read it).
template <class Done, class Now>
__host__ __device__ __forceinline__ bool bounded_polls(Done done, Now now, unsigned polls,
                                                       unsigned ns) {
  unsigned t0 = 0;
  for (unsigned n = 0; n < polls; ++n) {
    if (done()) return true;
    if ((n & 63u) == 63u) {
      const unsigned t = now();
      if (n == 63u) t0 = t;
      else if (t - t0 > ns) return false;
    }
  }
  return false;
}
// bounded wait: the error flag where it gave up
__device__ __forceinline__ bool mbar_wait_t(unsigned long long *bar, unsigned parity, int *err,
                                            unsigned polls = kMbarWaitLimit,
                                            unsigned ns = kMbarWaitNs) {
  const bool ok = bounded_polls(
      [&] {
        unsigned r;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(r)
            : "r"(sm_addr_t(bar)), "r"(parity)
            : "memory");
        return r != 0;
      },
      [] {
        unsigned t;
        asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
        return t;
      },
      polls, ns);
  if (!ok) atomicExch(err, 1);
  return ok;
}

}  // namespace sparc
