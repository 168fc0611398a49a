// Host-only model of the layer barriers of a batch's persistent stage blocks
// (compiled by nvcc, run on the CPU, against the kernels' own parity rule):
// blocks take the items of a work-list in turn, items of members with tensor
// copies and of members (or tiles) without them mixed, of any layer counts.
// Before each wait the parity that the body waits for must be that of the
// barrier's next phase.  The same model with a rule that flips the parity in
// every body must find violations.  Prints "ok <waits checked>" or the first
// violation; exit status 0 / 1.
#include <cstdio>
#include <random>
#include <vector>

#include "../../sparc2_b200/csrc/mhd_body.cuh"

using namespace sparc;

struct Item {
  bool tma;
  int layers;
};

struct Block {
  unsigned phase = 0;
  long long done[2] = {0, 0};  // phases each barrier has completed
  double busy = 0;
};

// waits that would look at the wrong phase
static long long run(const std::vector<Item> &items, int nblocks, bool always_flip,
                     long long &waits) {
  std::vector<Block> blocks(nblocks);
  long long bad = 0;
  for (const Item &it : items) {
    Block *B = &blocks[0];
    for (Block &q : blocks)
      if (q.busy < B->busy) B = &q;
    B->busy += it.layers + 2;
    for (int k = 0; k < it.layers; ++k) {
      const int b = k & 1;
      if (it.tma) {
        ++waits;
        if (((B->phase >> b) & 1u) != (unsigned)(B->done[b] & 1)) ++bad;
        ++B->done[b];
      }
      B->phase = it.tma || always_flip ? mhd_next_phase<true>(B->phase, b)
                                       : mhd_next_phase<false>(B->phase, b);
    }
  }
  return bad;
}

// a member's edge items at a z extent
static void add(std::vector<Item> &v, int tiles, int nz, int zc, bool tma) {
  for (int k0 = 0; k0 < nz; k0 += zc)
    for (int t = 0; t < tiles; ++t) v.push_back({tma, k0 + zc < nz ? zc : nz - k0});
}

int main() {
  long long waits = 0, planted = 0, none = 0;
  for (int zc : {11, 33, 48, 50})
    for (int nz : {105, 150, 171})
      for (int order = 0; order < 2; ++order)
        for (int blocks : {1, 7, 148}) {
          std::vector<Item> v;
          add(v, 36, nz, zc, order != 0);
          add(v, 40, nz, zc, order == 0);
          add(v, 36, nz + 1, zc, order != 0);
          add(v, 40, nz, zc, true);
          if (run(v, blocks, false, waits)) {
            std::printf("violation zc=%d nz=%d order=%d blocks=%d\n", zc, nz, order, blocks);
            return 1;
          }
          planted += run(v, blocks, true, none);
        }
  std::mt19937 rng(1);
  for (int n = 0; n < 200; ++n) {
    std::vector<Item> v;
    for (int i = 0; i < 400; ++i) v.push_back({rng() % 3 != 0, 1 + (int)(rng() % 40)});
    if (run(v, 1 + (int)(rng() % 20), false, waits)) {
      std::printf("violation in list %d\n", n);
      return 1;
    }
  }
  if (planted == 0) {
    std::printf("the planted rule was not found out\n");
    return 1;
  }
  std::printf("ok %lld\n", waits);
  return 0;
}
