// Host-only check of what DAMPING's set-up does where memory is short (compiled
// by nvcc, run on the CPU): damping.cu itself, with the allocations, the
// library's plans and its transforms replaced by ones that count against a
// budget.  Whatever fails with three velocities at a time, one at a time must
// serve, as long as that fits, with nothing left behind.  Prints "ok"; exit
// status 0 / 1.
#include <cufft.h>

#include <cstdio>
#include <map>
#include <vector>

#include "../../sparc2_b200/csrc/internal.h"

static size_t g_free;                      // bytes left
static std::map<const void *, size_t> g_mem;
static std::map<int, size_t> g_plans;      // live plans and their work areas
static int g_plan_id, g_plan_calls, g_fail_call;
static std::vector<const void *> g_in, g_out;

namespace sparc {
void *dev_alloc(Handle *h, size_t bytes) {
  if (bytes > g_free) {
    h->err = "no memory";
    return nullptr;
  }
  void *p = std::malloc(bytes);
  g_free -= bytes;
  g_mem[p] = bytes;
  return p;
}
void dev_free(Handle *, const void *p) {
  if (!g_mem.count(p)) return;
  g_free += g_mem[p];
  g_mem.erase(p);
  std::free(const_cast<void *>(p));
}
}  // namespace sparc

// (a work area of the batch's size, as large as the spectrum)
static cufftResult fake_plan(int *plan, int, int *, int *, int, int, int *, int, int, cufftType type,
                             int batch) {
  const size_t work = (size_t)batch * 1000;
  (void)type;
  if (++g_plan_calls == g_fail_call || work > g_free) return CUFFT_ALLOC_FAILED;
  g_free -= work;
  *plan = ++g_plan_id;
  g_plans[*plan] = work;
  return CUFFT_SUCCESS;
}
static cufftResult fake_destroy(int plan) {
  if (!g_plans.count(plan)) return CUFFT_INVALID_PLAN;
  g_free += g_plans[plan];
  g_plans.erase(plan);
  return CUFFT_SUCCESS;
}
static cufftResult fake_exec(const void *in, const void *out) {
  g_in.push_back(in);
  g_out.push_back(out);
  return CUFFT_SUCCESS;
}
#define cufftPlanMany fake_plan
#define cufftDestroy fake_destroy
#define cufftSetStream(p, s) CUFFT_SUCCESS
#define cufftExecD2Z(p, in, out) fake_exec(in, out)
#define cufftExecZ2D(p, in, out) fake_exec(in, out)
#define cudaMemcpyAsync(...) cudaSuccess
#define cudaStreamSynchronize(s) cudaSuccess
#define cudaGetLastError() cudaSuccess
#include "../../sparc2_b200/csrc/damping.cu"

using namespace sparc;

#define NEED(x)                                          \
  do {                                                   \
    if (!(x)) {                                          \
      std::printf("%s: %s\n", what, #x);                 \
      return 1;                                          \
    }                                                    \
  } while (0)

// set-up with `bytes` of memory and the plan call `fail` failing: `fields` at a
// time (0: refused)
static int check(const char *what, size_t bytes, int fail, int fields) {
  Handle h;
  h.nx = 23;
  h.px = 24;
  h.ny = 22;
  h.nz = 30;
  h.N = 23LL * 22 * 30;
  h.NP = 24LL * 22 * 30;
  h.P.xlength = h.P.ylength = 1e9;
  h.diml = h.dimc = 1.0;
  h.damping = true;
  h.err = "before";
  g_free = bytes;
  g_plan_calls = 0;
  g_fail_call = fail;
  const int r = damping_setup(&h);
  if (fields == 0) {
    NEED(r != SPARC_OK && g_plans.empty() && !h.fft_plans);
  } else {
    NEED(r == SPARC_OK && h.damp_fields == fields && g_plans.size() == 2 && h.fft_plans);
    NEED(h.err == "before");
    NEED(g_mem.size() == 3 && g_mem.count(h.d_spec) && g_mem.count(h.d_term));
    NEED(g_mem[h.d_spec] == (size_t)fields * 12 * 22 * 30 * 16);
    // the transforms of a stage
    g_in.clear();
    g_out.clear();
    const double *tin = (const double *)4096;
    NEED(damping_enqueue(&h, tin, nullptr) == SPARC_OK);
    const int calls = 3 / fields;
    NEED((int)g_in.size() == 2 * calls);
    for (int l = 0; l < calls; ++l) {
      NEED(g_in[2 * l] == tin + (1 + l) * h.NP && g_out[2 * l] == h.d_spec);
      NEED(g_in[2 * l + 1] == h.d_spec && g_out[2 * l + 1] == h.d_term + l * h.NP);
    }
  }
  damping_destroy(&h);
  NEED(g_plans.empty());
  while (!g_mem.empty()) dev_free(&h, g_mem.begin()->first);
  return 0;
}

int main() {
  const size_t rates = 12 * 22 * 8, term = 3 * 24 * 22 * 30 * 8, spec = 12 * 22 * 30 * 16,
               work = 30 * 1000, base = rates + term;
  const size_t all = base + 3 * spec + 6 * work;
  int bad = check("ample", all, 0, 3);
  bad |= check("no spectrum of three", base + 3 * spec - 1, 0, 1);
  bad |= check("no room for a plan of three", base + 3 * spec + 3 * work - 1, 0, 1);
  bad |= check("no room for the second plan", all - 1, 0, 1);
  bad |= check("the first plan refused", all, 1, 1);
  bad |= check("the second plan refused", all, 2, 1);
  bad |= check("just room for one", base + spec + 2 * work, 0, 1);
  bad |= check("not even one", base + spec + 2 * work - 1, 0, 0);
  bad |= check("no terms", base - 1, 0, 0);
  if (!bad) std::printf("ok\n");
  return bad;
}
