// Host check of the tile-overlapped layout and of the P slots of the sweeps:
// every cell of the inner grid has one entry of its own inside the skewed
// arrays, the coefficients of the system's entries are distinct and their
// chunks start on 16 bytes, and the entries of a P slot (tile, halo rows and
// columns, zero) do not overlap.  Prints the number of failures.
#include "cadmas_dev.cuh"
#include "kernels.h"
#include "sweep_cp.cuh"
#include <cstdio>
#include <vector>
using namespace cadmas;

static long long fails = 0, checks = 0;
static void check(bool c, const char *what, int a, int b, int d, int e) {
  ++checks;
  if (!c && fails++ < 10) printf("%s: %d %d %d %d\n", what, a, b, d, e);
}

template <typename V> static void system_entries(const SkewGeo &q) {
  const int T = q.T;
  std::vector<char> used((size_t)SYS_N * T, 0);
  for (int t = 0; t < T; ++t) {
    for (int c = 0; c < SYS_N; ++c) {
      const long long e = c == SYS_T ? sys_t(3, T, t) : sys_at<V>(3, c, T, t), o = e - 3LL * SYS_N * T;
      const bool ok = o >= 0 && o < (long long)used.size() && !used[(size_t)o];
      check(ok, "system entry", T, t, c, (int)o);
      if (ok) used[(size_t)o] = 1;
    }
    for (int c = 0; c < 8 * (int)sizeof(V) / 16; ++c)
      check(sys_chunk<V>(3, c, T, t) * sizeof(V) % 16 == 0, "chunk alignment", T, t, c, 0);
  }
}

static void run(int NI, int NJ, int NK, int TI, int TJ) {
  SkewGeo q{};
  q.TI = TI; q.TJ = TJ; q.TIp = (TI + 3) & ~3; q.T = q.TIp * TJ; q.W = (NK - 2) + (TI - 1) + (TJ - 1);
  q.WS = (TI - 1) + (TJ - 1) <= NK - 2 ? NK - 2 : q.W;
  q.ntx = (NI - 2 + TI - 1) / TI;
  q.nb = q.ntx * ((NJ - 2 + TJ - 1) / TJ); q.split = 1;
  std::vector<char> used((size_t)skew_entries(q), 0);
  for (int b = 0; b < q.nb; ++b)
    for (int tj = 0; tj < TJ; ++tj)
      for (int ti = 0; ti < TI; ++ti) {
        if (2 + (b % q.ntx) * TI + ti > NI - 1 || 2 + (b / q.ntx) * TJ + tj > NJ - 1) continue;
        for (int k = 0; k < NK - 2; ++k) {
          const long long slab = (long long)b * skew_stride(q) + k + ti + tj, e = slab * q.T + ti + q.TIp * tj;
          const bool ok = slab < skew_slabs(q) && e >= 0 && e < (long long)used.size() && !used[(size_t)e];
          check(ok, "cell's entry", b, ti, tj, k);
          if (ok) used[(size_t)e] = 1;
        }
      }
  system_entries<double>(q);
  system_entries<float>(q);
  const SweepP p = sweep_cp_pslot(q.T, q.TIp, TI, TJ);
  std::vector<char> s(p.size, 0);
  const auto put = [&](int e, const char *what, int i) {
    const bool ok = e >= 0 && e < p.size && !s[e];
    check(ok, what, TI, TJ, i, e);
    if (ok) s[e] = 1;
  };
  for (int t = 0; t < q.T; ++t) put(p.main + t, "P entry", t);
  for (int i = 0; i < TI; ++i) { put(p.down + i, "P below", i); put(p.up + i, "P above", i); }
  for (int j = 0; j < TJ; ++j) { put(p.left + p.xs * j, "P left", j); put(p.right + p.xs * j, "P right", j); }
  put(p.zero, "P zero", 0);
}

int main() {
  const int tiles[][2] = {{2, 2}, {4, 3}, {7, 5}, {8, 16}, {16, 8}, {16, 16}, {15, 17}, {31, 8}, {32, 8}, {64, 4},
                          {24, 16}, {32, 20}, {40, 25}, {3, 60}, {100, 2}};
  const int grids[][3] = {{3, 3, 3}, {18, 18, 5}, {39, 11, 23}, {35, 19, 22}, {102, 9, 40}, {67, 66, 128}};
  for (auto &t : tiles)
    for (auto &g : grids) run(g[0], g[1], g[2], t[0], t[1]);
  printf("%lld checks, %lld failures\n", checks, fails);
  return fails != 0;
}
