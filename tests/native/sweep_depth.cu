// Host check of the sweeps' copy depth (sweep_cp_depth): the rule for two
// blocks per SM counts the device's SMs, and every depth that the rule gives
// fits the shared memory it leaves; and which tiles run the thread copies.  Prints the number of failures.
#include "cadmas_dev.cuh"
#include "kernels.h"
#include "sweep_cp.cuh"
#include <cstdio>
#include <vector>
using namespace cadmas;

static SkewGeo tiles(int TI, int TJ, int ntx, int nty, int nsm, int occ = 0) {
  SkewGeo q{};
  q.TI = TI; q.TJ = TJ; q.TIp = (TI + 3) & ~3; q.T = q.TIp * TJ; q.W = 126 + (TI - 1) + (TJ - 1);
  q.ntx = ntx; q.nb = ntx * nty; q.split = 1; q.nsm = nsm; q.occ = occ;
  q.one = sweep_one_wide(q);
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
  // tiles one column wide beside others are told from slices and from the rest
  check(!sweep_one_wide(tiles(400, 1, 1, 1, 148)) && !sweep_one_wide(tiles(16, 1, 30, 1, 148)), "slice", 0, 0);
  check(sweep_one_wide(tiles(16, 1, 1, 2, 148)) && sweep_one_wide(tiles(1, 16, 2, 1, 148)), "one wide", 0, 0);
  check(!sweep_one_wide(tiles(2, 2, 9, 9, 148)), "two wide", 0, 0);
  // tiles one column wide along either direction, slices and others: a depth
  // for every mode, among those that are built; every value has its own entry
  // in a slot of P
  for (int n : {1, 2, 3, 4, 16, 29, 31, 32, 33, 64, 200, 255, 256, 257, 400, 800})
    for (int along = 0; along < 2; ++along)
      for (int nb : {1, 3}) {
        const int TI = along ? 1 : n, TJ = along ? n : 1;
        const SkewGeo q = tiles(TI, TJ, along ? nb : 1, along ? 1 : nb, 148);
        if (q.T > 800) continue;
        for (int es : {4, 8})
          for (int mode : {SWEEP_FWD, SWEEP_FWD_AX, SWEEP_BWD}) {
            const int d = sweep_cp_depth(q, mode, es);
            check((d > 0) == (mode != SWEEP_FWD_AX || q.T <= 576), "depth of a one-wide tile", q.T, mode);
            if (mode == SWEEP_FWD_AX && q.one && d > 0) check(d == 8 || d == 4 || d == 2, "built", q.T, d);
          }
        const SweepP p = sweep_cp_pslot(q.T, q.TIp, TI, TJ);
        std::vector<char> s(p.size, 0);
        auto put = [&](int e) {
          check(e >= 0 && e < p.size && !s[e], "P slot of a one-wide tile", q.T, e);
          if (e >= 0 && e < p.size) s[e] = 1;
        };
        for (int t = 0; t < q.T; ++t) put(p.main + t);
        for (int i = 0; i < TI; ++i) { put(p.down + i); put(p.up + i); }
        for (int j = 0; j < TJ; ++j) { put(p.left + p.xs * j); put(p.right + p.xs * j); }
        put(p.zero);
      }
  // more than 576 columns: no fused FP64 sweep, an FP32 one for square tiles
  check(sweep_cp_depth(tiles(24, 24, 4, 4, 148), SWEEP_FWD_AX, 8) == 2, "576 columns", 0, 0);
  check(sweep_cp_depth(tiles(32, 20, 4, 4, 148), SWEEP_FWD_AX, 8) == 0, "640 columns, FP64", 0, 0);
  check(sweep_cp_depth(tiles(32, 20, 4, 4, 148), SWEEP_FWD_AX, 4) == 8, "640 columns, FP32", 0, 0);
  check(sweep_cp_depth(tiles(128, 5, 4, 4, 148), SWEEP_FWD_AX, 4) == 0, "640 flat columns, FP32", 0, 0);
  printf("%lld checks, %lld failures\n", checks, fails);
  return fails != 0;
}
