// Host-only check that closing a handle does not wait for another handle's
// staged copy in progress (compiled by nvcc, run on the CPU, no CUDA call is
// reached): the slab's user holds its lock while a handle that is not the last
// is closed.  Prints "ok"; exit status 0 / 1.
#include <chrono>
#include <cstdio>
#include <future>

#include "../../sparc2_b200/csrc/state_io.cu"

namespace sparc {
bool cuda_ok(Handle *, cudaError_t e, const char *) { return e == cudaSuccess; }
}  // namespace sparc

using namespace sparc;

int main() {
  state_io_open();
  state_io_open();
  std::unique_lock<std::mutex> copying(g_use);
  auto closed = std::async(std::launch::async, [] { state_io_close(); });
  const bool waits = closed.wait_for(std::chrono::seconds(5)) != std::future_status::ready;
  copying.unlock();
  closed.get();
  state_io_close();
  if (waits || g_handles != 0) {
    std::printf("a close waited for another handle's copy\n");
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
