// Host check of the U-Net's convolution tilings (conv_plan): every
// convolution of the network, forward and input gradient, has one at every
// width up to X = 8192 (and some far wider), and it covers the layer, fits
// shared memory and TMEM, and stages all that its row blocks read.  Prints
// the number of failures.
#include "conv_plan.h"
#include <cstdio>
using namespace cadmas;

static long long fails = 0, checks = 0;
static void check(bool c, const char *what, int X, int Y, int ci, int co) {
  ++checks;
  if (!c && fails++ < 10) printf("%s: %d x %d, %d -> %d\n", what, X, Y, ci, co);
}

static void run(int X, int Y, int ci, int co) {
  const ConvPlan p = conv_plan(X, Y, ci, co);
  check(p.MT > 0, "no plan", X, Y, ci, co);
  if (p.MT == 0) return;
  check(p.bx >= 1 && p.by >= 1 && (long long)p.bx * p.nxt >= X && (long long)p.by * p.nyt >= Y && p.P == p.bx + 2,
        "coverage", X, Y, ci, co);
  check(p.MT * CONV_M >= p.by * p.P && p.MT * co <= 512, "row blocks", X, Y, ci, co);
  // the last row block's last tap reads 2 P + 2 voxels on; the staged rows
  check(p.PL >= p.MT * CONV_M + 2 * p.P + 2 && p.PL >= (p.by + 2) * p.P, "staged rows", X, Y, ci, co);
  check(p.a_bytes == (uint32_t)ci / 8 * p.PL * 16 && p.b_bytes == (uint32_t)(9 * ci * co * 2) && p.a_bytes % 16 == 0,
        "stage bytes", X, Y, ci, co);
  check((p.NST == 2 || p.NST == 3) && p.NST * ((size_t)p.a_bytes + p.b_bytes) + 24 <= p.smem && p.smem <= 227 * 1024,
        "shared memory", X, Y, ci, co);
}

int main() {
  const int layers[][3] = {{16, 16, 0}, {16, 32, 1}, {32, 32, 1}, {32, 64, 2}, {64, 64, 2}, {96, 32, 1}, {48, 16, 0}};
  for (auto &l : layers)
    for (int Y : {4, 36, 512}) {
      for (int X = 4; X <= 8192; X += Y == 4 ? 4 : 76) {
        run(X >> l[2], Y >> l[2], l[0], l[1]);
        run(X >> l[2], Y >> l[2], l[1], l[0]);
      }
      for (int X : {16384, 65536, 1000000}) {
        run(X >> l[2], Y >> l[2], l[0], l[1]);
        run(X >> l[2], Y >> l[2], l[1], l[0]);
      }
    }
  printf("%lld checks, %lld failures\n", checks, fails);
  return fails != 0;
}
