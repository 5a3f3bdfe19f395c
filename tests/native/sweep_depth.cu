// Host check of the sweeps' copy depth (sweep_cp_depth): the rule for two
// blocks per SM counts the device's SMs, and every depth that the rule gives
// fits the shared memory it leaves.  Prints the number of failures.
#include "cadmas_dev.cuh"
#include "kernels.h"
#include "sweep_cp.cuh"
#include <cstdio>
using namespace cadmas;

static SkewGeo tiles(int TI, int TJ, int ntx, int nty, int nsm, int occ = 0) {
  SkewGeo q{};
  q.TI = TI; q.TJ = TJ; q.TIp = (TI + 3) & ~3; q.T = q.TIp * TJ; q.W = 126 + (TI - 1) + (TJ - 1);
  q.ntx = ntx; q.nb = ntx * nty; q.split = 1; q.nsm = nsm; q.occ = occ;
  return q;
}
static size_t bytes(const SkewGeo &q, int mode, int es) {
  return sweep_cp_bytes(mode, sweep_cp_depth(q, mode, es), sweep_cp_unrolled(q, mode, es), q.T, q.TIp, q.TI, q.TJ, es);
}

int main() {
  long long fails = 0, checks = 0;
  auto check = [&](bool c, const char *what, int a, int b) {
    ++checks;
    if (!c && fails++ < 10) printf("%s: %d %d\n", what, a, b);
  };
  // 100 tiles of 16x16, FP32: one block per SM on 148 SMs, two on 74
  for (int mode : {SWEEP_FWD_AX, SWEEP_BWD, SWEEP_BWD5}) {
    const SkewGeo many = tiles(16, 16, 10, 10, 74), few = tiles(16, 16, 10, 10, 148);
    check(2 * bytes(many, mode, 4) <= 226 * 1024, "two blocks per SM", mode, (int)bytes(many, mode, 4));
    check(sweep_cp_depth(few, mode, 4) >= sweep_cp_depth(many, mode, 4), "one block is as deep", mode, 0);
  }
  check(sweep_cp_depth(tiles(16, 16, 10, 10, 148), SWEEP_FWD_AX, 4) == 8, "full depth", 0, 0);
  check(sweep_cp_depth(tiles(16, 16, 10, 10, 74), SWEEP_FWD_AX, 4) == 6, "shared depth", 0, 0);
  check(sweep_cp_depth(tiles(16, 16, 12, 13, 148), SWEEP_FWD_AX, 4) == 6, "156 tiles on 148 SMs", 0, 0);
  check(sweep_cp_depth(tiles(16, 16, 12, 13, 160), SWEEP_FWD_AX, 4) == 8, "156 tiles on 160 SMs", 0, 0);
  const int shapes[][2] = {{2, 2}, {8, 16}, {16, 8}, {16, 16}, {32, 8}, {7, 5}, {24, 16}, {32, 20}, {40, 21}, {427, 2}};
  for (auto &t : shapes)
    for (int n : {1, 10, 20})
      for (int occ : {0, 1, 2, 4})
        for (int es : {4, 8})
          for (int mode = SWEEP_FWD; mode <= (es == 4 ? SWEEP_BWD5 : SWEEP_BWD); ++mode) {
            const SkewGeo q = tiles(t[0], t[1], n, n, 148, occ);
            if (sweep_cp_depth(q, mode, es) > 0) check(bytes(q, mode, es) <= 227 * 1024, "shared memory", q.T, mode);
          }
  printf("%lld checks, %lld failures\n", checks, fails);
  return fails != 0;
}
