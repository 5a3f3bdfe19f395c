// sweep_cp.cuh -- the MILU sweeps with per-thread copies (VF_MZFRWD,
// vf_mzfrwd.f:37-48, optionally fused with VF_MZAX, vf_mzax.f:42-56, and
// VF_MZBKWD, vf_mzbkwd.f:37-47); included by k_poisson.cu.
#pragma once
#include "cadmas_dev.cuh"
#include "kernels.h"

namespace cadmas {

// A tile's NDOT sums from its threads' sums: warps by a butterfly, then the
// warps' partials by warp 0, in a fixed order; sum c into rb[c*nb + b].
template <int NDOT>
__device__ __forceinline__ void sweep_sums(const double *a, double *rb, int nb, int b) {
  __shared__ double s_red[5][32];
  const int tid = threadIdx.x, lane = tid & 31;
#pragma unroll
  for (int c = 0; c < NDOT; ++c) {
    double v = a[c];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) s_red[c][tid >> 5] = v;
  }
  __syncthreads();
  if (tid < 32) {
    const int nw = (int)(blockDim.x >> 5);
#pragma unroll
    for (int c = 0; c < NDOT; ++c) {
      double v = (tid < nw) ? s_red[c][tid] : 0.0;
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (tid == 0) rb[(long long)c * nb + b] = v;
    }
  }
}

// ---------------------------------------------- sweeps with thread copies
// The sweeps without a producer warp: every thread streams its own column's
// values with cp.async into a shared-memory ring, D wavefront steps ahead.
//   * Copies are predicated on the column having a cell at that step, so the
//     wavefront's ramp (the slabs only partly inside the tile) is not read.
//   * The coefficients come as 16-byte chunks (sys_chunk): one copy and one
//     shared-memory load move two FP64 or four FP32 values.  A thread reads
//     only chunks that it copied itself, after its own wait.
//   * P (SWEEP_FWD_AX) lies in a ring of its own that runs two steps ahead
//     of the coefficients', because the neighbours to the right and above
//     visit a cell one step later.  A column on the tile's edge also copies
//     its neighbour's P from the neighbouring tile, into the slot in which
//     that neighbour's P would lie if it were a column of this tile.  At most
//     one along x and one along y: tiles have at least two columns each way,
//     or one tile covers that direction, and only the last tile of a row,
//     which has no right neighbour, may be one wide.  ONE is the form for
//     tiles one column wide with neighbours on both sides (SkewGeo::one).
//   * The result of step s and DD of step s+1 are published as one pair.
//   * One barrier per step; the recurrence of step s and the preparation of
//     step s+1 are independent and scheduled into one another.
//   * For the tile shapes that are compiled in (CT, CTIP) the loop is
//     unrolled over the ring, so that slots, buffers and the copies' sources
//     are constant offsets: a warp's instructions per step, each waiting
//     for the one before, are what a small grid's step takes.
// Zero entries of the shared P and X arrays stand for neighbours outside.  The expressions and their order are those of the reference loops.
__device__ __forceinline__ void cpa16(unsigned dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
template <int B> __device__ __forceinline__ void cpa(unsigned dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(src), "n"(B) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <typename V> struct SweepPair;
template <> struct SweepPair<double> { using type = double2; };
template <> struct SweepPair<float> { using type = float2; };

// Values per column and step in the ring, besides P: the chunks, then the
// vector of the mode (Y, or T and R0 and RR).
// (the plain forward sweep needs no AUI, AUJ: in FP64 their chunk stays out)
__host__ __device__ constexpr int sweep_cp_first(int mode, int es) { return mode == SWEEP_FWD && es == 8 ? 1 : 0; }
__host__ __device__ constexpr int sweep_cp_chunked(int mode, int es) {
  return mode >= SWEEP_BWD ? 4 : 8 - 2 * sweep_cp_first(mode, es);
}
__host__ __device__ constexpr int sweep_cp_plain(int mode) {
  return mode == SWEEP_FWD_AX ? 0 : (mode == SWEEP_FWD ? 1 : 1 + (mode - SWEEP_BWD));
}
// One slot of P: the tile's T entries from `main` on, the halo rows and
// columns, a zero.  Up to 256 columns each halo value lies in the bank that
// its reader's own neighbour entry would have (the lower row before the
// tile's entries, the upper one after them, left and right ones spread by
// TIp), so that a warp's load has no conflicts; larger tiles, whose rings are
// short of memory, pack them.
struct SweepP {
  int main, zero, left, right, xs, down, up, size;  // left + xs*tj, right + xs*tj, down + ti, up + ti
};
__host__ __device__ inline SweepP sweep_cp_pslot(int T, int TIp, int TI, int TJ) {
  SweepP p;
  if (T <= 256) {
    p.main = (TIp + 31) & ~31;
    p.down = p.main - TIp;
    p.up = p.main + T;
    p.zero = (p.up + TIp + 31) & ~31;
    p.xs = TIp;
    p.left = p.zero + 31;
    p.right = p.zero + TIp;
    p.size = p.zero + TIp * (TJ - 1) + (TIp > 31 ? TIp : 31) + 1;
  } else {
    p.main = 0;
    p.zero = T;
    p.xs = 1;
    p.left = T + 1;
    p.right = T + 1 + TJ;
    p.down = T + 1 + 2 * TJ;
    p.up = T + 1 + 2 * TJ + TI;
    p.size = T + 1 + 2 * (TI + TJ);
  }
  p.size = (p.size + 3) & ~3;  // 16 bytes
  return p;
}
// The compiled-in shapes (ct = T; 0: any shape) run the unrolled loop, but
// for the fused FP64 sweep of 256 columns, whose slots are so large that
// the longer ring costs it two steps of depth (512 tiles: 250 against 242 us).
__host__ __device__ constexpr bool sweep_cp_unroll(int mode, int ct, int es) {
  return ct > 0 && !(mode == SWEEP_FWD_AX && es == 8 && ct >= 256);
}
// slots of the ring for depth D: the unrolled fused sweep takes as many as
// P's
__host__ __device__ constexpr int sweep_cp_slots(int mode, int D, bool unrolled) {
  return D + (mode == SWEEP_FWD_AX && unrolled ? 4 : 1);
}
// shared memory of a block
__host__ __device__ inline size_t sweep_cp_bytes(int mode, int D, bool unrolled, int T, int TIp, int TI, int TJ, int es) {
  size_t n = (size_t)sweep_cp_slots(mode, D, unrolled) * (sweep_cp_chunked(mode, es) + sweep_cp_plain(mode)) * T;
  n += 2 * (size_t)(T + 16) * (mode >= SWEEP_BWD ? 1 : 2);
  if (mode == SWEEP_FWD_AX) n += (size_t)(D + 4) * sweep_cp_pslot(T, TIp, TI, TJ).size;
  return n * es;
}

// Depth of the thread copies: a step (0.1 to 0.35 us) is far shorter than the
// latency of a copy, so as deep as the shared memory allows, shared by two
// blocks per SM where there are more tiles than SMs (by q.occ blocks if that
// is set) as long as that leaves depth 6.  Measured, us per sweep: 128 tiles
// of 8x16 x 96 layers, FP64, depths 4, 8, 12: fused forward 34.8, 28.8, 26.8;
// backward depths 4, 7, 15: 21.2, 14.5, 14.5 (in a solve, where the
// system comes from memory, 19.6 at 7).  512 tiles of 16x16 x 126 layers: FP64
// fused, one block at depth 8 242, at 6 250, two at 4 255; FP32 fused, two at
// depth 6 132, one 143; backward FP64 at depth 7, one block 139, two 141.
// Tiles of more than 576 columns have 64 registers a thread and room for two
// steps (FP64) in the fused sweep: A P on its own before the plain sweep takes
// less, except in FP32 with few edge columns (0: no fused sweep).  Forward
// stage, ms a step, fused and apart: FP64 32x20 18.5, 15.4; 32x25 26.9, 18.3;
// 128x6 38.0, 20.6; 400x2 47.5, 21.6; 24x24 12.6, 14.9 (576 columns); FP32
// 32x20 16.5, 18.7; 32x25 20.2, 21.5; 100x6 18.2, 16.3; 400x2 41.0, 24.3.
inline int sweep_cp_threads(int T) { return (T + 31) & ~31; }
inline bool sweep_cp_unrolled(const SkewGeo &q, int mode, int es) {
  const bool ct = (q.T == 128 && (q.TIp == 8 || q.TIp == 16)) || (q.T == 256 && q.TIp == 16);
  return sweep_cp_unroll(mode, ct ? q.T : 0, es);
}
inline int sweep_cp_depth(const SkewGeo &q, int mode, int es) {
  if (q.split != 1) return 0;
  const bool one = mode == SWEEP_FWD_AX && q.one;  // built for depths 8, 4 and 2
  const int nt = sweep_cp_threads(q.T), blocks = q.occ > 0 ? q.occ : (q.nb > q.nsm ? 2 : 1);
  if (mode == SWEEP_FWD_AX && nt > 576 && (es == 8 || q.TI < 16 || q.TJ < 16)) return 0;
  const bool unr = sweep_cp_unrolled(q, mode, es);
  const int ax[] = {12, 8, 6, 4, 2, 1}, plain[] = {15, 9, 3, 1};
  for (size_t share : {226 * 1024 / (size_t)blocks, (size_t)(227 * 1024)})
    for (int i = 0; i < (mode == SWEEP_FWD_AX ? 6 : 4); ++i) {
      const int d = mode == SWEEP_FWD_AX ? ax[i] : plain[i];
      if ((d >= 12 && nt > 128) || (d == 1 && nt <= 576) || (one && (d == 12 || d == 6))) continue;
      if (q.occ == 0 && blocks > 1 && share < 227 * 1024 && d < 6) continue;
      if (sweep_cp_bytes(mode, d, unr, q.T, q.TIp, q.TI, q.TJ, es) <= share) return d;
    }
  return 0;
}

template <int D, int MODE, typename V, int CT, int CTIP, bool ONE = false>
__device__ __forceinline__ void sweep_cp_body(const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *vin,
                                              V *vout, SolveState *st, const V *vin2, double *rb, int bx, int by) {
  constexpr bool BWD = MODE >= SWEEP_BWD, AX = MODE == SWEEP_FWD_AX;
  constexpr int NDOT = sweep_ndot(MODE);
  constexpr int ES = (int)sizeof(V), G = 16 / ES;                 // elements per chunk
  constexpr int C0 = sweep_cp_first(MODE, ES), NC = sweep_cp_chunked(MODE, ES) / G, NP = sweep_cp_plain(MODE);
  constexpr int E0 = SYS_AUI + C0 * G;                            // first coefficient
  constexpr bool UNR = sweep_cp_unroll(MODE, CT, ES);
  constexpr int R = sweep_cp_slots(MODE, D, UNR), RP = D + 4;     // slots of the rings
  constexpr int U = UNR ? R : 1;                                  // steps per turn of the loop
  static_assert(!UNR || (R % 2 == 0 && (!AX || R == RP)), "unrolled rings: even, and equal");
  using V2 = typename SweepPair<V>::type;
  if (st->done) return;
  const int WS = skew_stride(q);
  const int T = CT > 0 ? CT : q.T, TIp = CT > 0 ? CTIP : q.TIp, TI = q.TI, TJ = CT > 0 ? CT / (CTIP > 0 ? CTIP : 1) : q.TJ;
  const int tid = threadIdx.x, b = bx + q.ntx * by, nty = q.nb / q.ntx;
  const int XB = T + 16;                                          // entries of an exchange buffer
  const int SS = (NC * G + NP) * T, PS = AX ? sweep_cp_pslot(T, TIp, TI, TJ).size : 0;
  const SweepP po = sweep_cp_pslot(T, TIp, TI, TJ);
  extern __shared__ __align__(16) double sm[];
  V *ring = reinterpret_cast<V *>(sm);                            // R slots: chunks, then plain vectors
  V *pb = ring + (size_t)R * SS;                                  // RP slots of P
  V *xb = pb + (size_t)(AX ? RP : 0) * PS;                        // 2 x XB: X, or (X, DD)
  V2 *xd = reinterpret_cast<V2 *>(xb);
  const int wi = min(TI, g.NI - (2 + bx * TI)), wj = min(TJ, g.NJ - (2 + by * TJ));
  const int ti = tid % TIp, tj = tid / TIp;
  const bool col = ti < wi && tj < wj;  // false too on the padding column and past T
  const int nsteps = (g.NK - 2) + (wi - 1) + (wj - 1);
  const int ri = wi - 1 - ti, rj = wj - 1 - tj;
  const int slo = col ? (BWD ? ri + rj : ti + tj) : (1 << 29);
  const unsigned nact = (unsigned)(g.NK - 3);
  const int tq = min(tid, T - 1);
  const int o1 = (col && (BWD ? ri > 0 : ti > 0)) ? tq + (BWD ? 1 : -1) : (BWD ? T : T + 15);
  const int o2 = (col && (BWD ? rj > 0 : tj > 0)) ? tq + (BWD ? TIp : -TIp) : T;
  if (tid < 2) {  // the zeros
    if (BWD) {
      xb[tid * XB + T] = V(0);
    } else {
      V2 z; z.x = V(0); z.y = V(0);
      xd[tid * XB + T] = z;
      xd[tid * XB + T + 15] = z;  // the left column's: in the bank that its neighbours leave free
    }
    if (AX)
      for (int r = tid; r < RP; r += 2) pb[r * PS + po.zero] = V(0);
  }
  const long long slab0 = (long long)b * WS + (BWD ? nsteps - 1 : 0);
  constexpr long long DIR = BWD ? -1 : 1;
  const long long vstep = DIR * T, sstep = DIR * SYS_N * T;
  // next values to copy: chunks, the plain vectors, P and its halo columns
  const V *lc = S.sys + sys_chunk<V>(slab0, C0, T, tq);
  const V *l0 = BWD ? S.sys + sys_t(slab0, T, tq) : (vin ? vin + slab0 * T + tq : nullptr);  // T, Y or P
  const V *l1 = NDOT > 0 ? vin + slab0 * T + tq : nullptr, *l2 = NDOT == 5 ? vin2 + slab0 * T + tq : nullptr;  // R0, RR
  // P's lateral neighbours: entries of the P slots of the steps before (left,
  // lower) and after (right, upper)
  const bool hl = AX && col && ti == 0 && bx > 0, hr = AX && col && ti == wi - 1 && bx < q.ntx - 1;
  const bool hd = AX && col && tj == 0 && by > 0, hu = AX && col && tj == wj - 1 && by < nty - 1;
  const int el = po.left + po.xs * min(tj, TJ - 1), er = po.right + po.xs * min(tj, TJ - 1);
  const int ed = po.down + min(ti, TI - 1), eu = po.up + min(ti, TI - 1);
  const int ehx = hr ? er : el, ehy = hu ? eu : ed;
  const int tp = po.main + tq;
  const int oxm = hl ? el : ((col && ti > 0) ? tp - 1 : po.zero), oxp = hr ? er : ((col && ti < wi - 1) ? tp + 1 : po.zero);
  const int oym = hd ? ed : ((col && tj > 0) ? tp - TIp : po.zero), oyp = hu ? eu : ((col && tj < wj - 1) ? tp + TIp : po.zero);
  const int shx = hr ? -1 : 1, shy = hu ? -1 : 1;  // own step minus the neighbour's
  const bool hx = hl || hr, hy = hd || hu;
  const V *lx = vin, *ly = vin;                    // halo values for P slot 0
  const V *lr = vin, *lu = vin;                    // ONE: the right and upper ones (lx, ly the left and lower)
  const long long hrofs = AX ? ((long long)(b + 1) * WS - TI) * T + TIp * tj : 0,
                  huofs = AX ? ((long long)(b + q.ntx) * WS - TJ) * T + ti : 0;
  if (AX) {  // own step u: the neighbour's cell of the same layer; slot v = u - shx
    if (hl) lx = vin + ((long long)(b - 1) * WS + TI) * T + (TI - 1) + TIp * tj;
    if (hr) (ONE ? lr : lx) = vin + hrofs;
    if (hd) ly = vin + ((long long)(b - q.ntx) * WS + TJ) * T + ti + TIp * (TJ - 1);
    if (hu) (ONE ? lu : ly) = vin + huofs;
  }
  V *vp = BWD ? vout + slab0 * T + tq : S.sys + sys_t(slab0, T, tq);
  auto active = [&](int u) { return (unsigned)(u - slo) <= nact; };
  const unsigned ring0 = (unsigned)__cvta_generic_to_shared(ring) + (unsigned)(tq * 16),
                 plain0 = (unsigned)__cvta_generic_to_shared(ring + NC * G * T + tq);
  const unsigned pb0 = AX ? (unsigned)__cvta_generic_to_shared(pb) : 0u;
  // chunks and plain vectors of step u into the slot at byte offset so;
  // sources r steps past the pointers
  auto load = [&](int u, unsigned so, int r) {
    if (!active(u)) return;
    const V *c0 = lc + r * sstep;
#pragma unroll
    for (int c = 0; c < NC; ++c) cpa16(ring0 + so + (unsigned)(c * T * 16), c0 + c * T * G);
    if (!AX) cpa<ES>(plain0 + so, l0 + r * (BWD ? sstep : vstep));
    if (NDOT > 0) cpa<ES>(plain0 + so + (unsigned)(T * ES), l1 + r * vstep);
    if (NDOT == 5) cpa<ES>(plain0 + so + (unsigned)(2 * T * ES), l2 + r * vstep);
  };
  // P of step v and the halo columns of slot v into the slot at byte offset so
  auto loadp = [&](int v, unsigned so, int r) {
    if (active(v)) cpa<ES>(pb0 + so + (unsigned)(tp * ES), l0 + r * vstep);
    if constexpr (ONE) {
      if (hl && active(v + 1)) cpa<ES>(pb0 + so + (unsigned)(el * ES), lx + r * vstep);
      if (hr && active(v - 1)) cpa<ES>(pb0 + so + (unsigned)(er * ES), lr + r * vstep);
      if (hd && active(v + 1)) cpa<ES>(pb0 + so + (unsigned)(ed * ES), ly + r * vstep);
      if (hu && active(v - 1)) cpa<ES>(pb0 + so + (unsigned)(eu * ES), lu + r * vstep);
      return;
    }
    if (hx && active(v + shx)) cpa<ES>(pb0 + so + (unsigned)(ehx * ES), lx + r * vstep);
    if (hy && active(v + shy)) cpa<ES>(pb0 + so + (unsigned)(ehy * ES), ly + r * vstep);
  };
  auto advance = [&](int n) {  // the sources of the chunks and plain vectors
    lc += n * sstep;
    if (!AX) l0 += n * (BWD ? sstep : vstep);
    if (NDOT > 0) l1 += n * vstep;
    if (NDOT == 5) l2 += n * vstep;
  };
  auto advancep = [&](int n) {
    l0 += n * vstep;
    lx += n * vstep;
    ly += n * vstep;
    if (ONE) {
      lr += n * vstep;
      lu += n * vstep;
    }
  };

  V dd = V(0), y0 = V(0), c1 = V(0), c2 = V(0), c3 = V(0);  // prepared values of the step
  V dk1 = V(0), xk1 = V(0);           // DD and the result of this column at the previous step
  V p0 = V(0), p1 = V(0);             // P of this column one step before, and at, the step to prepare
  V q0 = V(0), q1 = V(0);             // R0 and RR of the step, and of the step before (0 outside the column's cells)
  V zk0 = V(0), zk1 = V(0);
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, a4 = 0.0;
  struct alignas(16) Chunk { V v[G]; };
  // this column's values of a step, read from the slot at sl
  struct Vals { V r[NC * G], y, z0, z1; };
  auto fetch = [&](const V *sl) {
    Vals f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const Chunk k = *reinterpret_cast<const Chunk *>(sl + (c * T + tq) * G);
#pragma unroll
      for (int i = 0; i < G; ++i) f.r[c * G + i] = k.v[i];
    }
    const V *pl = sl + NC * G * T + tq;
    f.y = AX ? V(0) : pl[0];
    f.z0 = NDOT > 0 ? pl[T] : V(0);
    f.z1 = NDOT == 5 ? pl[2 * T] : V(0);
    return f;
  };
  // prepare step u from its values; d1, d2: DD of the neighbouring columns
  auto prepare = [&](int u, const Vals &f, V d1, V d2, V pxm, V pym, V pxp, V pyp, V p2) {
    const V *r = f.r;
    dd = r[SYS_DD - E0];
    if (!BWD) {
      const V ali = r[SYS_ALI - E0], alj = r[SYS_ALJ - E0], alk = r[SYS_ALK - E0];
      const unsigned k = (unsigned)(u - slo);  // layer of the cell (0: the lowest)
      if (AX) {
        const V pzm = k == 0 ? V(0) : p0, pzp = k < nact ? p2 : V(0);
        y0 = r[SYS_AD - E0] * p1 + ali * pxm + alj * pym + alk * pzm + r[0] * pxp + r[1] * pyp + r[2] * pzp;
      } else {
        y0 = f.y;
      }
      c1 = ali * d1;
      c2 = alj * d2;
      c3 = alk * (k == 0 ? V(0) : dk1);
      dk1 = dd;
    } else {
      y0 = f.y;
      c1 = r[0]; c2 = r[1]; c3 = r[2];
      q0 = f.z0;
      q1 = f.z1;
    }
  };
  // the sums of a step from its factors (0 outside the column's cells);
  // products of two single-precision values are exact in double
  auto sums = [&](V x, V z0, V z1) {
    if (NDOT == 1) a0 += (double)z0 * (double)x;
    if (NDOT == 5) {
      const double rv = (double)z1, e = (double)x, z = (double)z0;
      a0 += rv * e;
      a1 += e * e;
      a2 += rv * rv;
      a3 += z * rv;
      a4 += z * e;
    }
  };

  // P slot v lies at position (v+1) % RP, chunks of step u at u % R.  Copy
  // group i (one per iteration, D+1 of them before the first) holds the
  // values of step i+1+D and P slot i+3+D; the first holds P slots -1..1
  // too.  Iteration s waits for its own group s-D (the values of step s+1,
  // P of slot s+3) and the barrier at its end shows that P to the others.
  const unsigned SB = (unsigned)(SS * ES), PSB = (unsigned)(PS * ES);
  if (AX) {
    advancep(-1);
    loadp(-1, 0u, 0);
    loadp(0, PSB, 1);
    loadp(1, 2 * PSB, 2);
    advancep(3);
  }
#pragma unroll 1
  for (int j = 0; j <= D; ++j) {
    load(j, (unsigned)j * SB, 0);
    advance(1);
    if (AX) {
      loadp(j + 2, (unsigned)(j + 3) * PSB, 0);
      advancep(1);
    }
    cpa_commit();
  }
  cpa_wait<D>();
  __syncthreads();
  V pz = V(0);
  if (AX) { p1 = pb[PS + tp]; pz = pb[2 * PS + tp]; }
  prepare(0, fetch(ring), V(0), V(0), AX ? pb[oxm] : V(0), AX ? pb[oym] : V(0), AX ? pb[2 * PS + oxp] : V(0),
          AX ? pb[2 * PS + oyp] : V(0), pz);
  p0 = p1; p1 = pz;
  if (!BWD && tid < T) {
    V2 z; z.x = V(0); z.y = dd;
    xd[XB + tid] = z;
  }
  // iteration s, the r-th of a turn; cs: slot of step s+1; pm, pp: P slots
  // s and s+2; wso, wpo: byte offsets of the next group's slots; wr, rd: the
  // exchange buffers of steps s and s-1
  auto iterate = [&](int s, int r, const V *cs, const V *pm, const V *pp, unsigned wso, unsigned wpo, int wr, int rd) {
    cpa_wait<D - 1>();
    V x1, x2, d1 = V(0), d2 = V(0), pxm = V(0), pym = V(0), pxp = V(0), pyp = V(0), p2 = V(0);
    if (BWD) {
      x1 = xb[rd + o1];
      x2 = xb[rd + o2];
    } else {
      const V2 n1 = xd[rd + o1], n2 = xd[rd + o2];
      x1 = n1.x; d1 = n1.y; x2 = n2.x; d2 = n2.y;
    }
    if (AX) { pxm = pm[oxm]; pym = pm[oym]; pxp = pp[oxp]; pyp = pp[oyp]; p2 = pp[tp]; }
    const Vals f = fetch(cs);
    load(s + 1 + D, wso, r);
    if (AX) loadp(s + 3 + D, wpo, r);
    cpa_commit();
    if (NDOT > 0) sums(xk1, zk0, zk1);  // of step s-1
    const bool a = active(s), live = a && dd != V(0);
    V x = y0 - c1 * x1 - c2 * x2 - c3 * xk1;
    if (BWD) x = x * dd;
    x = live ? x : V(0);
    if (NDOT > 0) { zk0 = a ? q0 : V(0); zk1 = a ? q1 : V(0); }
    prepare(s + 1, f, d1, d2, pxm, pym, pxp, pyp, p2);
    if (AX) { p0 = p1; p1 = p2; }
    if (BWD) {
      if (UNR || tid < T) xb[wr + tid] = x;
    } else if (UNR || tid < T) {
      V2 z; z.x = x; z.y = dd;
      xd[wr + tid] = z;
    }
    if (a) vp[r * (BWD ? vstep : sstep)] = x;
    xk1 = x;
  };
  __syncthreads();
  if (!__any_sync(0xffffffffu, col)) {  // a warp past the grid's edge (a ragged tile)
#pragma unroll 1
    for (int s = 0; s < nsteps; ++s) __syncthreads();
  } else if constexpr (UNR) {
#pragma unroll 1
    for (int s0 = 0; s0 < nsteps; s0 += U) {
#pragma unroll
      for (int r = 0; r < U; ++r) {
        if (s0 + r >= nsteps) break;
        // group s goes where step s (chunks, D = R-1) or, with R = D+4,
        // step s-3 lay; P slot s+3+D where slot s-1 lay
        iterate(s0 + r, r, ring + ((r + 1) % R) * SS, pb + ((r + 1) % RP) * PS, pb + ((r + 3) % RP) * PS,
                (unsigned)((r + 1 + D) % R) * SB, (unsigned)((r + 4 + D) % RP) * PSB, (r & 1) * XB, ((r + 1) & 1) * XB);
        __syncthreads();
      }
      advance(U);
      if (AX) advancep(U);
      vp += U * (BWD ? vstep : sstep);
    }
  } else {
    const V *cs = ring + SS, *const cend = ring + (size_t)R * SS;
    const V *pm = pb + PS, *pp = pb + 3 * PS, *const pend = pb + RP * PS;
    unsigned wso = 0u, wpo = 0u;
    int wr = 0, rd = XB;
    // the warp's steps, one before its first cell to one after its last
    const int wfirst = __reduce_min_sync(0xffffffffu, slo) - 1;
    const int wlast = __reduce_max_sync(0xffffffffu, col ? slo + (int)nact : -1) + 1;
#pragma unroll 1
    for (int s = 0; s < nsteps; ++s) {
      if (CT > 0 || (s >= wfirst && s <= wlast)) {
        iterate(s, 0, cs, pm, pp, wso, wpo, wr, rd);
      } else {  // no column of the warp has a cell at step s or s+1: only the copies
        cpa_wait<D - 1>();
        load(s + 1 + D, wso, 0);
        if (AX) {
          loadp(s + 3 + D, wpo, 0);
          p0 = p1; p1 = pp[tp];
        }
        cpa_commit();
      }
      advance(1);
      vp += BWD ? vstep : sstep;
      cs += SS;
      if (cs == cend) cs = ring;
      wso += SB;
      if (wso == R * SB) wso = 0u;
      if (AX) {
        advancep(1);
        pm += PS;
        if (pm == pend) pm = pb;
        pp += PS;
        if (pp == pend) pp = pb;
        wpo += PSB;
        if (wpo == RP * PSB) wpo = 0u;
      }
      const int xs = wr; wr = rd; rd = xs;
      __syncthreads();
    }
  }
  cpa_wait<0>();
  if (NDOT > 0) {
    sums(xk1, zk0, zk1);  // of the last step
    const double a[5] = {a0, a1, a2, a3, a4};
    sweep_sums<NDOT>(a, rb, q.nb, b);
  }
}
template <int D, int MODE, int MAXT, typename V, int MINB, int CT, int CTIP, bool ONE = false>
__global__ void __launch_bounds__(MAXT, MINB)
    k_sweep_cp(Geo g, SkewGeo q, SkewSysT<V> S, const V *vin, V *vout, SolveState *st, const V *vin2, double *rb) {
  pdl_enter();
  sweep_cp_body<D, MODE, V, CT, CTIP, ONE>(g, q, S, vin, vout, st, vin2, rb, (int)blockIdx.x, (int)blockIdx.y);
}

}  // namespace cadmas
