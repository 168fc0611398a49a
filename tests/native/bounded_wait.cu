// Host-only check of the bound of the kernels' waits (compiled by nvcc, run on
// the CPU): a wait whose copies never land ends by the clock however long a
// poll takes, by the number of polls where the clock stands still, and one
// whose copies land within the limit succeeds; also across a wrap of the
// 32-bit clock.  Prints "ok"; exit status 0 / 1.
#include <cstdio>

#include "../../sparc2_b200/csrc/tma_util.cuh"

using namespace sparc;

// elapsed nanoseconds of a wait whose poll takes `poll_ns`, done after `after`
static bool wait(unsigned long long start, unsigned poll_ns, unsigned long long after,
                 unsigned polls, unsigned ns, unsigned long long &elapsed) {
  unsigned long long t = start;
  const bool ok = bounded_polls(
      [&] {
        t += poll_ns;
        return t - start > after;
      },
      [&] { return (unsigned)t; }, polls, ns);
  elapsed = t - start;
  return ok;
}

int main() {
  const unsigned long long never = ~0ull;
  unsigned long long e;
  if (kMbarWaitNs > 2000000000u) return std::printf("limit of %u ns\n", kMbarWaitNs), 1;
  for (unsigned long long start : {0ull, 4294000000ull, 4294967295ull}) {
    for (unsigned poll : {20u, 1000u, 20000u, 1000000u}) {
      // two intervals of 64 polls pass beside the limit at most
      if (wait(start, poll, never, kMbarWaitLimit, kMbarWaitNs, e) ||
          e < kMbarWaitNs || e > kMbarWaitNs + 128ull * poll)
        return std::printf("poll %u ns: gave up after %llu ns\n", poll, e), 1;
      if (!wait(start, poll, kMbarWaitNs / 2, kMbarWaitLimit, kMbarWaitNs, e))
        return std::printf("poll %u ns: gave up early\n", poll), 1;
    }
    if (wait(start, 0, never, 1u << 20, kMbarWaitNs, e))
      return std::printf("a clock that stands still\n"), 1;
  }
  std::printf("ok\n");
  return 0;
}
