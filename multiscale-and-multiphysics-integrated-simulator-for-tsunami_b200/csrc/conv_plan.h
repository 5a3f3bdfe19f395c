// conv_plan.h -- tiling of the U-Net's convolutions (k_conv, k_unet.cu),
// chosen on the host.
#pragma once
#include <cstddef>
#include <cstdint>
#include "umma.cuh"

namespace cadmas {

constexpr int CONV_M = 128;  // voxels of an MMA row block
// Tiling of one convolution: tiles of bx x by voxels, nxt x nyt of them per
// layer; P = bx + 2 voxels per padded row; MT row blocks of CONV_M; PL rows
// of a staged layer (the last row block reads 2 P + 2 rows past its own);
// NST stages (3: all layers resident, 2: the third reuses the first's).
// MT = 0: no tiling fits.
struct ConvPlan {
  int bx, by, nxt, nyt, P, PL, MT, NST;
  uint32_t a_bytes, b_bytes;  // of one stage
  size_t smem;
};

// The CTAs that share an SM must find their TMEM columns free (512 per
// SM): a CTA with more columns asks for more shared memory.
inline size_t smem_floor(size_t b, uint32_t cols) {
  const size_t f = cols <= 128 ? 56 * 1024 : (cols <= 256 ? 80 * 1024 : 120 * 1024);
  return b < f ? f : b;
}

// Tile of a convolution of X x Y voxels a layer: rows of at most 126 voxels;
// as many rows as make the least work per voxel, counting the MMAs' rows (128
// per row block) and half as much for each staged voxel, within the shared
// memory of two CTAs per SM where that can be (else of one) and 256 TMEM
// columns (one row block may use more).  Three stages where they fit.  The
// fewest tiles along x and up to three more are compared; where even one row
// of those is too wide for a stage (96 channels leave 85 voxels a row, which
// X / 2 > 851 does not give in three more tiles), the fewest that fit.
inline ConvPlan conv_plan(int X, int Y, int Cin, int Cout) {
  ConvPlan best{};
  double cost = 0.0;
  auto try_tiles = [&](int nxt, size_t cap) {
    for (int nst = 3; nst >= 2; --nst) {
      const int bx = (X + nxt - 1) / nxt, P = bx + 2;
      for (int by = 1; by <= Y && by <= 128; ++by) {
        ConvPlan p{};
        p.bx = bx; p.by = by; p.nxt = nxt; p.nyt = (Y + by - 1) / by; p.P = P; p.NST = nst;
        p.MT = (by * P + CONV_M - 1) / CONV_M;
        if (p.MT > 1 && p.MT * Cout > 256) break;
        p.PL = (p.MT * CONV_M + 2 * P + 2 + 7) & ~7;
        p.PL += 4;  // the two 8-channel rows of a voxel in different banks
        p.a_bytes = (uint32_t)(Cin / 8 * p.PL * 16);
        p.b_bytes = (uint32_t)(9 * Cin * Cout * 2);
        const size_t need = (size_t)nst * (p.a_bytes + p.b_bytes) + 64;
        if (need > cap) break;
        p.smem = smem_floor(need, umma::tmem_cols((uint32_t)(p.MT * Cout)));
        const double c = (double)nxt * p.nyt * (p.MT * 128.0 + 0.5 * (by + 2) * P + 128.0) * (nst == 2 ? 1.15 : 1.0);
        if (best.MT == 0 || c < cost) { best = p; cost = c; }
      }
    }
  };
  constexpr size_t two = 112 * 1024, one = 225 * 1024;  // shared memory for two CTAs per SM, and for one
  const int nxt0 = (X + 125) / 126;
  for (size_t cap : {two, one})
    if (cap == two || best.MT == 0)
      for (int nxt = nxt0; nxt <= nxt0 + 3; ++nxt) try_tiles(nxt, cap);
  for (int nxt = nxt0 + 4; best.MT == 0 && nxt <= X; ++nxt) try_tiles(nxt, one);
  return best;
}

}  // namespace cadmas
