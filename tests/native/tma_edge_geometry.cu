// Host-only check of the edge tiles' TMA halo boxes (compiled by nvcc, run
// on the CPU): for every grid width and every tile of it, the box must start
// at a multiple of 16 bytes and hold the stencil window of every active column,
// and the columns turned into fluxes (32 own ones from the tile's first, ten
// around them) must cover those windows and stay inside a box row.
// Prints "ok <tiles checked>" or the first violation; exit status 0 / 1.
#include <cstdio>
#include <vector>

#include "../../sparc2_b200/csrc/mhd_body.cuh"

using namespace sparc;

template <class R>
static bool check(int n, long long &tiles) {
  using MB = MhdBuf<R, true>;
  for (int x0 = 0; x0 < n; x0 += mg::TX) {
    const int o = origin_th<R>(x0, mg::TX, n), start = o - MB::XOFF, cx0 = x0 - o;
    if ((start * (int)sizeof(R)) % 16 != 0 || cx0 < 5) return false;
    std::vector<char> have(MB::HXL, 0);
    for (int t = 0; t < mg::TX; ++t) {
      const int p = cx0 + t + MB::XOFF;
      if (p >= MB::HXL) return false;
      have[p] = 1;
    }
    for (int c = 0; c < 10; ++c) {
      const int cl = cx0 < 10 ? cx0 : 10;
      const int p = (c < cl ? c + cx0 - cl : c + mg::TX) + MB::XOFF;
      if (p >= MB::HXL) return false;
      have[p] = 1;
    }
    for (int i = x0; i < n && i < x0 + mg::TX; ++i) {
      const int b = i < 5 ? 0 : (i >= n - 5 ? n - 11 : i - 5);
      for (int m = 0; m < 11; ++m) {
        const int p = b + m - start;
        if (p < 0 || p >= MB::HXL || !have[p]) return false;
      }
    }
    ++tiles;
  }
  return true;
}

int main() {
  long long tiles = 0;
  for (int n = 22; n <= 1026; ++n) {
    if (!check<double>(n, tiles) || !check<float>(n, tiles)) {
      std::printf("violation n=%d\n", n);
      return 1;
    }
  }
  std::printf("ok %lld\n", tiles);
  return 0;
}
