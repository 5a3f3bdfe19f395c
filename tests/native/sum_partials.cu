// Host check of the buffers that sums over the grid leave their partials in:
// sum_partials holds what a slab sum writes (a partial per block of slabs) and
// what a backward sweep with sums writes (a partial per tile), for tiles with
// few slabs and with many.  Prints the number of failures.
#include "cadmas_dev.cuh"
#include "kernels.h"
#include <cstdio>
using namespace cadmas;

int main() {
  long long fails = 0, checks = 0;
  for (int TI : {1, 2, 3, 4, 16})
    for (int TJ : {1, 2, 3, 16})
      for (int nk : {3, 4, 5, 8, 126})
        for (int n : {1, 5, 60, 200}) {
          SkewGeo q{};
          q.TI = TI; q.TJ = TJ; q.TIp = (TI + 3) & ~3; q.T = q.TIp * TJ; q.W = nk + (TI - 1) + (TJ - 1);
          q.ntx = n; q.nb = n * n; q.split = 1;
          // the last slab's block; the last tile
          const long long slab = ((long long)q.nb * q.W - 1) / ROWS_PER_BLOCK, tile = q.nb - 1;
          checks += 3;
          fails += !(slab < sum_partials(q)) + !(tile < sum_partials(q)) + !(slab_partials(q) == slab + 1);
        }
  printf("%lld checks, %lld failures\n", checks, fails);
  return fails != 0;
}
