// k_vof.cu -- donor-acceptor VOF advection and surface-cell flagging of
// VF_F1CAL (vf_f1cal.f:121-230).
//
//   k_fconv        VF_FCONV  (vf_fconv.f:56-206)  three face fluxes per cell
//   k_feuler       VF_FEULER (vf_feuler.f:43-56)
//   k_fmod1_*      VF_FMOD1  (vf_fmod1.f:37-200) as gathers:
//                    count  - NLIM of each fluid/gas cell = surface cells
//                             whose donor (F) or acceptor (E) it is
//                    redist - loop 300 per surface cell; the E/F cells it
//                             writes have NLIM = 1, i.e. belong to it alone
//                    target - loop 400 for E/F cells: the over/under-fill of
//                             the surface neighbours added in ascending
//                             linear index, the order of the INDS list
//                    clamp  - loop 400 for the surface cells themselves
//   k_fcut         VF_FCUT01 (vf_fcut01.f:34-56) cut-off + FSUM/FCUT partials
//   k_fnf_*        VF_FNFINI (vf_fnfini.f:36-197), one pass per sweep of
//                  the reference; the fixed-point loop is driven by the host
//                  with a device change counter
//   k_fbubup       VF_FBUBUP (vf_fbubup.f:35-51) one thread per column
//   k_fnfprv       VF_FNFPRV (vf_fnfprv.f:34-225)
//   k_cindc        VF_CINDC  (vf_cindc.f:35-53), also counts NUMS
//   k_bsppfl       VF_BSPPFL (vf_bsppfl.f:40-67) into a second buffer
//
// Bound by the latency of their loads, so a cell's are issued together and
// the passes that act on few cells scan several flags at once (cell and scan
// kernels of cadmas_dev.cuh): on 519x63x85 cells k_fconv 122 -> 63 us,
// k_fnf_init 54 -> 22, k_bsuwn3 46 -> 11, k_fmod1_target 68 -> 26; the VOF
// stage 282 -> 180 us and the flags 471 -> 368 us.
//
// The surface list INDS of the reference is not kept: every loop over it
// is a pass over the grid that acts on cells with NF in 1..6 (or 7).  The
// loops are free of ordering effects because FNFPRV gives each surface
// cell a fluid neighbour (NF=0) on its fluid side and a gas neighbour
// (NF=8) on the other, so the cells one surface cell writes are never
// read by another in the same loop; the one scatter-add (loop 400 of
// FMOD1) is done as an ordered gather.
#include "cadmas_dev.cuh"
#include "kernels.h"
#include "vof_face.cuh"

namespace cadmas {

#define A(a, i, j, k) a[cid(g, i, j, k)]
#define XX_(m, i) gx(g, m, i)
#define YY_(m, j) gy(g, m, j)
#define ZZ_(m, k) gz(g, m, k)

// ------------------------------------------------------------ VF_FCONV
__global__ void __launch_bounds__(CELL_THREADS) k_fconv(Geo g, Fld f, Prm p, double *FLFU, double *FLFV, double *FLFW) {
  const double DT = p.dtnow, FL = p.flower;
  const int *NF = f.nf;
  const double *FF = f.ff, *GGV = f.ggv;
  CELL_LOOP_BEGIN(g)
  const long long c = cid(g, I, J, K);
  const int NI = g.NI, NJ = g.NJ, NK = g.NK;
  double fu = 0.0, fv = 0.0, fw = 0.0;
  if (K >= 2 && J >= 2 && I >= 2) {
    const bool dox = K <= NK - 1 && J <= NJ - 1, doy = K <= NK - 1 && I <= NI - 1, doz = J <= NJ - 1 && I <= NI - 1;
    // All that the three faces may use, in flight together (cells that a
    // face does not use may lie outside of the grid: any address serves).
    const long long sj = NI, sk = (long long)NI * NJ, last = g.N - 1;
    const int ix = ld_now(f.indx + c), iy = ld_now(f.indy + c), iz = ld_now(f.indz + c);
    const double cx = DT * ld_now(f.ggx + c) * ld_now(f.uu + c), cy = DT * ld_now(f.ggy + c) * ld_now(f.vv + c),
                 cz = DT * ld_now(f.ggz + c) * ld_now(f.ww + c);
    const int n0 = ld_now(NF + c);
    const double f0 = ld_now(FF + c), g0 = ld_now(GGV + c);
    // the cell across the face (a), the one behind it (b), the next on this side (d)
    const auto face = [&](bool doit, double C, int ind, long long st, double wa, double w0, int d1, int d2, int d3, int d4) {
      const long long ca = c - st, cb = max(c - 2 * st, 0LL), cd = min(c + st, last);
      const int na = ld_now(NF + ca), nb = ld_now(NF + cb), nd = ld_now(NF + cd);
      const double fa = ld_now(FF + ca), fb = ld_now(FF + cb), fd = ld_now(FF + cd), ga = ld_now(GGV + ca);
      if (!doit || ind == -1) return 0.0;
      const bool fwd = C >= 0.0;  // the donor is a, else this cell
      const int N = fwd ? na : n0, ndm = (N != -1) ? (fwd ? nb : nd) : -1, nac = fwd ? n0 : na;
      const double fdm = (N != -1 && ndm != -1) ? (fwd ? fb : fd) : 0.0, wd = fwd ? wa : w0;
      const double vd = (N != -1) ? wd * (fwd ? ga : g0) : 0.0, bcf = (N == -1) ? f.bcf[ind - 1] : 0.0;
      const double fl = fconv_face(C, N, (N != -1) ? (fwd ? fa : f0) : 0.0, ndm, fdm, vd, wd, bcf, nac,
                                   (nac != -1) ? (fwd ? f0 : fa) : 0.0, d1, d2, d3, d4, FL);
      return 0.0 - (double)(fwd ? 1 : -1) * fl;
    };
    fu = face(dox, cx, ix, 1, XX_(2, I - 1), XX_(2, I), 3, 4, 5, 6);
    fv = face(doy, cy, iy, sj, YY_(2, J - 1), YY_(2, J), 1, 2, 5, 6);
    fw = face(doz, cz, iz, sk, ZZ_(2, K - 1), ZZ_(2, K), 1, 2, 3, 4);
  }
  FLFU[c] = fu; FLFV[c] = fv; FLFW[c] = fw;
  CELL_LOOP_END
}

// ----------------------------------------------------------- VF_FEULER
__global__ void __launch_bounds__(CELL_THREADS) k_feuler(Geo g, Fld f, Prm p, const double *FLFU, const double *FLFV, const double *FLFW) {
  CELL_LOOP_BEGIN(g)
  if (I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1) {
    const long long c = cid(g, I, J, K);
    if (f.nf[c] != -1) {
      double G = f.ggv[c];
      double G0 = G - (G - G) * 1.0;
      // QF of VF_FGENE (vf_fgene.f:42-70): on the wave source's line, the
      // fluid cells up to and the first surface cell of the column (gas
      // cells below it skipped) gain F * 2 XX(4,I) SRCUV (or YY(4,J))
      double QF = 0.0;
      if ((p.iws == I || p.jws == J) && f.nf[c] != 8) {
        bool below = true;  // no surface cell under this one
        for (int K2 = 2; K2 < K; ++K2) {
          const int n2 = A(f.nf, I, J, K2);
          if (n2 != -1 && n2 != 0 && n2 != 8) { below = false; break; }
        }
        if (below) {
          if (p.iws == I) QF = QF + f.ff[c] * (2.0 * XX_(4, I) * f.srcuv[(J - 1) + (long long)g.NJ * (K - 1)]);
          if (p.jws == J) QF = QF + f.ff[c] * (2.0 * YY_(4, J) * f.srcuv[(I - 1) + (long long)g.NI * (K - 1)]);
        }
      }
      double DF = (XX_(4, I) * (A(FLFU, I + 1, J, K) - FLFU[c]) + YY_(4, J) * (A(FLFV, I, J + 1, K) - FLFV[c]) +
                   ZZ_(4, K) * (A(FLFW, I, J, K + 1) - FLFW[c]) + p.dtnow * QF);
      f.ff[c] = (G0 * f.ff[c] + DF) / G;
    }
  }
  CELL_LOOP_END
}

// ------------------------------------------------------------ VF_FMOD1
// E (acceptor, gas side) and F (donor, fluid side) cells of a surface cell.
__device__ __forceinline__ void fmod_ends(int N, int I, int J, int K, int &IE, int &JE, int &KE, int &IF,
                                          int &JF, int &KF) {
  IE = I; JE = J; KE = K; IF = I; JF = J; KF = K;
  if (N == 5) { KE = K + 1; KF = K - 1; }
  else if (N == 6) { KE = K - 1; KF = K + 1; }
  else if (N == 3) { JE = J + 1; JF = J - 1; }
  else if (N == 4) { JE = J - 1; JF = J + 1; }
  else if (N == 1) { IE = I + 1; IF = I - 1; }
  else if (N == 2) { IE = I - 1; IF = I + 1; }
}
__device__ __forceinline__ bool is_surf(int n) { return n >= 1 && n <= 6; }

// Neighbour offsets in ascending linear-index order and the NF value a
// surface cell at that offset must have for this cell to be its E or F.
// Offset (-K): the cell below; it points up at us if it is NF=5 (fluid
// below it, so we are its E) or NF=6 (we are its F).
struct NbSel { int di, dj, dk, nE, nF; };
__device__ constexpr NbSel c_nb[6] = {
    {0, 0, -1, 5, 6}, {0, -1, 0, 3, 4}, {-1, 0, 0, 1, 2},
    {1, 0, 0, 2, 1},  {0, 1, 0, 4, 3},  {0, 0, 1, 6, 5}};

__global__ void __launch_bounds__(CELL_THREADS) k_fmod1_count(Geo g, Fld f, int *NLIM) {
  CELL_LOOP_BEGIN(g)
  const long long c = cid(g, I, J, K);
  int n = 0;
  if (I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1) {
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      int nb = A(f.nf, I + c_nb[q].di, J + c_nb[q].dj, K + c_nb[q].dk);
      if (nb == c_nb[q].nE || nb == c_nb[q].nF) n++;
    }
  }
  NLIM[c] = n;
  CELL_LOOP_END
}

__device__ __forceinline__ double cellvol(const Geo &g, const double *GGV, int I, int J, int K) {
  return gx(g, 2, I) * gy(g, 2, J) * gz(g, 2, K) * GGV[cid(g, I, J, K)];
}

__global__ void __launch_bounds__(CELL_THREADS) k_fmod1_redist(Geo g, Fld f, const int *NLIM) {
  double *FF = f.ff;
  SCAN_LOOP_BEGIN(g, f.nf, n_ >= 1 && n_ <= 6)
  const long long s = cid(g, I, J, K);
  int N = f.nf[s];
  if (is_surf(N) && I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1) {
    int IE, JE, KE, IF, JF, KF;
    fmod_ends(N, I, J, K, IE, JE, KE, IF, JF, KF);
    const long long e = cid(g, IE, JE, KE), fc = cid(g, IF, JF, KF);
    double VE = cellvol(g, f.ggv, IE, JE, KE), VS = cellvol(g, f.ggv, I, J, K), VF = cellvol(g, f.ggv, IF, JF, KF);
    double SS = VS * FF[s];
    if (NLIM[e] == 1) SS = SS + VE * FF[e];
    if (NLIM[fc] == 1) SS = SS + VF * FF[fc];
    double DS;
    if (NLIM[fc] == 1) { DS = dmin(VF, SS); SS = SS - DS; FF[fc] = DS / VF; }
    DS = dmin(VS, SS); SS = SS - DS; FF[s] = DS / VS;
    if (NLIM[e] == 1) { DS = dmin(VE, SS); SS = SS - DS; FF[e] = DS / VE; }
    if (SS > 0.0) {
      if (NLIM[e] == 1) FF[e] = FF[e] + SS / VE;
      else FF[s] = FF[s] + SS / VS;
    }
  }
  SCAN_LOOP_END
}

// Loop 400 for E/F cells (non-surface), gathering from surface neighbours.
__global__ void __launch_bounds__(CELL_THREADS) k_fmod1_target(Geo g, Fld f) {
  double *FF = f.ff;
  CELL_LOOP_BEGIN(g)
  const long long c = cid(g, I, J, K);
  if (!is_surf(f.nf[c]) && I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1) {
    int nb[6];
    bool any = false;
#pragma unroll
    for (int q = 0; q < 6; ++q) nb[q] = ld_now(&A(f.nf, I + c_nb[q].di, J + c_nb[q].dj, K + c_nb[q].dk));
#pragma unroll
    for (int q = 0; q < 6; ++q) any = any || is_surf(nb[q]);
    if (!any) continue;  // away from the surface
    double v = FF[c];
    bool touched = false;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int Is = I + c_nb[q].di, Js = J + c_nb[q].dj, Ks = K + c_nb[q].dk;
      const long long s = cid(g, Is, Js, Ks);
      const int n = nb[q];
      if (n == c_nb[q].nE) {            // we are the E cell of s
        double fs = FF[s];
        if (fs > 1.0) {
          double VS = cellvol(g, f.ggv, Is, Js, Ks), VE = cellvol(g, f.ggv, I, J, K);
          v = v + VS * (fs - 1.0) / VE;
          touched = true;
        }
      } else if (n == c_nb[q].nF) {     // we are the F cell of s
        double fs = FF[s];
        if (!(fs > 1.0) && fs < 0.0) {
          double VS = cellvol(g, f.ggv, Is, Js, Ks), VF = cellvol(g, f.ggv, I, J, K);
          v = v + VS * fs / VF;
          touched = true;
        }
      }
    }
    if (touched) FF[c] = v;
  }
  CELL_LOOP_END
}

__global__ void __launch_bounds__(CELL_THREADS) k_fmod1_clamp(Geo g, Fld f) {
  SCAN_LOOP_BEGIN(g, f.nf, n_ >= 1 && n_ <= 6)
  const long long s = cid(g, I, J, K);
  if (is_surf(f.nf[s]) && I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1) {
    double v = f.ff[s];
    if (v > 1.0) v = 1.0;
    else if (v < 0.0) v = 0.0;
    f.ff[s] = v;
  }
  SCAN_LOOP_END
}

// ----------------------------------------------------------- VF_FCUT01
__global__ void k_fcut(Geo g, Fld f, Prm p, double *rb_sum, double *rb_cut) {
  double ssum = 0.0, scut = 0.0;
  const long long nrows = (long long)g.NJ * g.NK;
  ROW_LOOP_BEGIN(g)
  if (I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1) {
    const long long c = cid(g, I, J, K);
    if (f.nf[c] != -1) {
      double V = XX_(2, I) * YY_(2, J) * ZZ_(2, K) * f.ggv[c];
      double F = f.ff[c];
      if (F > p.fupper) { scut = scut + (F - 1.0) * V; F = 1.0; f.ff[c] = F; }
      else if (F < p.flower) { scut = scut + (F - 0.0) * V; F = 0.0; f.ff[c] = F; }
      ssum = ssum + F * V;
    }
  }
  ROW_LOOP_END
  const long long row = (long long)blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 5);
  row_store(ssum, rb_sum, row, nrows);
  row_store(scut, rb_cut, row, nrows);
}

// ----------------------------------------------------------- VF_FNFINI
// Phase 1+2: non-obstacle cells to fluid, then gas where F < FLOWER and no
// neighbour face carries F > FUPPER (vf_fnfini.f:39-103).
__global__ void __launch_bounds__(CELL_THREADS) k_fnf_init(Geo g, Fld f, Prm p) {
  const double FU = p.fupper;
  const double *FF = f.ff;
  CELL_LOOP_BEGIN(g)
  const long long c = cid(g, I, J, K);
  if (K >= 2 && K <= g.NK - 1) {
    const double F = ld_now(FF + c);
    int n = f.nf[c];
    if (n != -1) {
      n = 0;
      if (I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && F < p.flower) {
        int IX1 = f.indx[c], IX2 = A(f.indx, I + 1, J, K), IY1 = f.indy[c], IY2 = A(f.indy, I, J + 1, K);
        int IZ1 = f.indz[c], IZ2 = A(f.indz, I, J, K + 1);
        // a face with IND >= 1 does not count, whatever its boundary value
        const double FX1 = ld_now(&A(FF, I - 1, J, K)), FX2 = ld_now(&A(FF, I + 1, J, K));
        const double FY1 = ld_now(&A(FF, I, J - 1, K)), FY2 = ld_now(&A(FF, I, J + 1, K));
        const double FZ1 = ld_now(&A(FF, I, J, K - 1)), FZ2 = ld_now(&A(FF, I, J, K + 1));
        if (!(FZ1 > FU && IZ1 == 0) && !(FY1 > FU && IY1 == 0) && !(FY2 > FU && IY2 == 0) &&
            !(FX1 > FU && IX1 == 0) && !(FX2 > FU && IX2 == 0) && !(FZ2 > FU && IZ2 == 0))
          n = 8;
      }
      f.nf[c] = n;
    }
  }
  CELL_LOOP_END
}

__device__ __forceinline__ bool interior3(const Geo &g, int I, int J, int K) {
  return I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1;
}

// loop 1100: cells next to gas become surface (7).  A thread takes SCAN_K
// cells of a column: their flags and those above and below them at once,
// then the lateral ones of all that may change.
__global__ void __launch_bounds__(CELL_THREADS) k_fnf_mark7(Geo g, int *NF, const int *done) {
  if (*done) return;
  CELL_IJ(g)
    if (I < 2 || I > g.NI - 1 || J < 2 || J > g.NJ - 1) return;
    const long long sj = g.NI, sk = (long long)g.NI * g.NJ;
    for (int K0 = (int)blockIdx.y * SCAN_K + 1; K0 <= g.NK; K0 += (int)gridDim.y * SCAN_K) {
      int v[SCAN_K + 2];
      bool any = false;
#pragma unroll
      for (int u = 0; u < SCAN_K + 2; ++u) v[u] = NF[p_ + sk * (min(max(K0 + u - 1, 1), g.NK) - 1)];
#pragma unroll
      for (int u = 1; u <= SCAN_K; ++u) any = any || (v[u] != -1 && v[u] != 8);
      if (!any) continue;
      bool gas[SCAN_K];
#pragma unroll
      for (int u = 0; u < SCAN_K; ++u) {
        const int *q = NF + p_ + sk * (min(K0 + u, g.NK) - 1);
        const int a = q[-1], b = q[1], c = q[-sj], d = q[sj];
        gas[u] = (a == 8) | (b == 8) | (c == 8) | (d == 8) | (v[u] == 8) | (v[u + 2] == 8);
      }
#pragma unroll
      for (int u = 0; u < SCAN_K; ++u) {
        const int K = K0 + u;
        if (K >= 2 && K <= g.NK - 1 && v[u + 1] != -1 && v[u + 1] != 8 && gas[u]) NF[p_ + sk * (K - 1)] = 7;
      }
    }
  }
}
// loop 1200: surface cells without a fluid neighbour become gas
__global__ void __launch_bounds__(CELL_THREADS) k_fnf_to8(Geo g, int *NF, const int *done) {
  if (*done) return;
  SCAN_LOOP_BEGIN(g, NF, n_ == 7)
  const long long c = cid(g, I, J, K);
  if (interior3(g, I, J, K) && NF[c] == 7) {
    if (A(NF, I, J, K + 1) != 0 && A(NF, I, J + 1, K) != 0 && A(NF, I, J - 1, K) != 0 &&
        A(NF, I + 1, J, K) != 0 && A(NF, I - 1, J, K) != 0 && A(NF, I, J, K - 1) != 0)
      NF[c] = 8;
  }
  SCAN_LOOP_END
}
// loop 1300: surface cells not between fluid and gas along any axis -> -7
__global__ void __launch_bounds__(CELL_THREADS) k_fnf_markm7(Geo g, int *NF, int *nch, const int *done) {
  if (*done) return;
  int cnt = 0;
  SCAN_LOOP_BEGIN(g, NF, n_ == 7)
  const long long c = cid(g, I, J, K);
  if (interior3(g, I, J, K) && NF[c] == 7) {
    if (A(NF, I, J, K - 1) != 0 || A(NF, I, J, K + 1) != 8)
      if (A(NF, I - 1, J, K) != 0 || A(NF, I + 1, J, K) != 8)
        if (A(NF, I + 1, J, K) != 0 || A(NF, I - 1, J, K) != 8)
          if (A(NF, I, J - 1, K) != 0 || A(NF, I, J + 1, K) != 8)
            if (A(NF, I, J + 1, K) != 0 || A(NF, I, J - 1, K) != 8)
              if (A(NF, I, J, K + 1) != 0 || A(NF, I, J, K - 1) != 8) { NF[c] = -7; cnt++; }
  }
  SCAN_LOOP_END
  if (cnt) atomicAdd(nch, cnt);
}
// loop exit test: NCH = 0 ends the iteration; the counter is cleared for
// the next sweep.  Capped so that no input can keep the loop running.
__global__ void k_fnf_check(int *nch, int *done, int *iter, int cap, int *err) {
  if (*done) return;
  int n = *nch;
  *nch = 0;
  *iter = *iter + 1;
  if (n <= 0) *done = 1;
  else if (*iter >= cap) { *done = 1; atomicOr(err, ERR_CAP); }
}
// loop 1400: -7 -> gas
__global__ void __launch_bounds__(CELL_THREADS) k_fnf_m7to8(Geo g, int *NF, const int *done) {
  if (*done) return;
  SCAN_LOOP_BEGIN(g, NF, n_ == -7)
  const long long c = cid(g, I, J, K);
  if (NF[c] == -7) NF[c] = 8;
  SCAN_LOOP_END
}

// ----------------------------------------------------------- VF_FBUBUP
// One thread per (I,J) column walks K = NK-2 .. 2 over the levels whose
// timer fired (active[K] != 0, decided on the host from TBUB and TNOW).
__global__ void k_fbubup(Geo g, Fld f, Prm p, const unsigned char *active) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  int ni = g.NI - 2, nj = g.NJ - 2;
  if (t >= ni * nj) return;
  const int I = 2 + t % ni, J = 2 + t / ni;
  double *FF = f.ff;
  for (int K = g.NK - 2; K >= 2; --K) {
    if (!active[K]) continue;
    const int K1 = K + 1;
    const long long c = cid(g, I, J, K), u = cid(g, I, J, K1);
    if (FF[c] < p.fupper && f.nf[c] == 0 && f.nf[u] != -1) {
      double V0 = ZZ_(2, K) * f.ggv[c], V1 = ZZ_(2, K1) * f.ggv[u];
      double FMOVE = dmin((1.0 - FF[c]) * V0, FF[u] * V1);
      FF[u] = FF[u] - FMOVE / V1;
      FF[c] = FF[c] + FMOVE / V0;
    }
  }
}

// ----------------------------------------------------------- VF_FNFPRV
__device__ __forceinline__ double bcf_or(const Fld &f, int ind, double v) { return ind >= 1 ? f.bcf[ind - 1] : v; }

__global__ void __launch_bounds__(CELL_THREADS) k_fnfprv(Geo g, Fld f, int *err) {
  const double *FF = f.ff;
  int *NF = f.nf;
  SCAN_LOOP_BEGIN(g, f.nf, n_ == 7)
  const long long c = cid(g, I, J, K);
  if (interior3(g, I, J, K) && NF[c] == 7) {
    double FM = -1.0, FS;
    int res = 7;
    int KB = K - 1;
    if (A(NF, I, J, KB) == 0 && A(NF, I, J, K + 1) == 8) {
      FS = 2.0 * A(FF, I, J, KB);
      FS = FS + bcf_or(f, A(f.indx, I, J, KB), A(FF, I - 1, J, KB));
      FS = FS + bcf_or(f, A(f.indx, I + 1, J, KB), A(FF, I + 1, J, KB));
      FS = FS + bcf_or(f, A(f.indy, I, J, KB), A(FF, I, J - 1, KB));
      FS = FS + bcf_or(f, A(f.indy, I, J + 1, KB), A(FF, I, J + 1, KB));
      if (FS > FM) { res = 5; FM = FS; }
    }
    KB = K + 1;
    if (A(NF, I, J, KB) == 0 && A(NF, I, J, K - 1) == 8) {
      FS = 2.0 * A(FF, I, J, KB);
      FS = FS + bcf_or(f, A(f.indx, I, J, KB), A(FF, I - 1, J, KB));
      FS = FS + bcf_or(f, A(f.indx, I + 1, J, KB), A(FF, I + 1, J, KB));
      FS = FS + bcf_or(f, A(f.indy, I, J, KB), A(FF, I, J - 1, KB));
      FS = FS + bcf_or(f, A(f.indy, I, J + 1, KB), A(FF, I, J + 1, KB));
      if (FS > FM) { res = 6; FM = FS; }
    }
    int JB = J - 1;
    if (A(NF, I, JB, K) == 0 && A(NF, I, J + 1, K) == 8) {
      FS = 2.0 * A(FF, I, JB, K);
      FS = FS + bcf_or(f, A(f.indx, I, JB, K), A(FF, I - 1, JB, K));
      FS = FS + bcf_or(f, A(f.indx, I + 1, JB, K), A(FF, I + 1, JB, K));
      FS = FS + bcf_or(f, A(f.indz, I, JB, K), A(FF, I, JB, K - 1));
      FS = FS + bcf_or(f, A(f.indz, I, JB, K + 1), A(FF, I, JB, K + 1));
      if (FS > FM) { res = 3; FM = FS; }
    }
    JB = J + 1;
    if (A(NF, I, JB, K) == 0 && A(NF, I, J - 1, K) == 8) {
      FS = 2.0 * A(FF, I, JB, K);
      FS = FS + bcf_or(f, A(f.indx, I, JB, K), A(FF, I - 1, JB, K));
      FS = FS + bcf_or(f, A(f.indx, I + 1, JB, K), A(FF, I + 1, JB, K));
      FS = FS + bcf_or(f, A(f.indz, I, JB, K), A(FF, I, JB, K - 1));
      FS = FS + bcf_or(f, A(f.indz, I, JB, K + 1), A(FF, I, JB, K + 1));
      if (FS > FM) { res = 4; FM = FS; }
    }
    int IB = I - 1;
    if (A(NF, IB, J, K) == 0 && A(NF, I + 1, J, K) == 8) {
      FS = 2.0 * A(FF, IB, J, K);
      FS = FS + bcf_or(f, A(f.indy, IB, J, K), A(FF, IB, J - 1, K));
      FS = FS + bcf_or(f, A(f.indy, IB, J + 1, K), A(FF, IB, J + 1, K));
      FS = FS + bcf_or(f, A(f.indz, IB, J, K), A(FF, IB, J, K - 1));
      FS = FS + bcf_or(f, A(f.indz, IB, J, K + 1), A(FF, IB, J, K + 1));
      if (FS > FM) { res = 1; FM = FS; }
    }
    IB = I + 1;
    if (A(NF, IB, J, K) == 0 && A(NF, I - 1, J, K) == 8) {
      FS = 2.0 * A(FF, IB, J, K);
      FS = FS + bcf_or(f, A(f.indy, IB, J, K), A(FF, IB, J - 1, K));
      FS = FS + bcf_or(f, A(f.indy, IB, J + 1, K), A(FF, IB, J + 1, K));
      FS = FS + bcf_or(f, A(f.indz, IB, J, K), A(FF, IB, J, K - 1));
      FS = FS + bcf_or(f, A(f.indz, IB, J, K + 1), A(FF, IB, J, K + 1));
      if (FS > FM) { res = 2; FM = FS; }
    }
    NF[c] = res;
    if (res == 7) atomicOr(err, ERR_PG);
  }
  SCAN_LOOP_END
}

// ------------------------------------------------------------ VF_CINDC
__global__ void __launch_bounds__(CELL_THREADS) k_cindc(Geo g, Fld f, int *nums) {
  int cnt = 0;
  CELL_IJ(g)
    const long long sk = (long long)g.NI * g.NJ;
    if (I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1)
      for (int K0 = (int)blockIdx.y * SCAN_K + 1; K0 <= g.NK; K0 += (int)gridDim.y * SCAN_K) {
        int v[SCAN_K];
#pragma unroll
        for (int u = 0; u < SCAN_K; ++u) v[u] = f.nf[p_ + sk * (min(K0 + u, g.NK) - 1)];
#pragma unroll
        for (int u = 0; u < SCAN_K; ++u) {
          const int K = K0 + u, n = v[u];
          if (K < 2 || K > g.NK - 1) continue;
          f.indc[p_ + sk * (K - 1)] = (n == 8 || n == -1) ? -1 : 0;
          if (n >= 1 && n <= 7) cnt++;
        }
      }
  }
  if (cnt) atomicAdd(nums, cnt);
}

// ----------------------------------------------------------- VF_BSPPFL
__global__ void __launch_bounds__(CELL_THREADS) k_bsppfl(Geo g, Fld f, const double *PP0, double *PPN) {
  CELL_LOOP_BEGIN(g)
  const long long c = cid(g, I, J, K);
  double v = PP0[c];
  if (interior3(g, I, J, K) && f.nf[c] == 0 && f.nf0[c] == 8) {
    double SUMF = 0.0, SUMP = 0.0;
    for (int KP = -1; KP <= 1; ++KP)
      for (int JP = -1; JP <= 1; ++JP)
        for (int IP = -1; IP <= 1; ++IP) {
          const long long q = cid(g, I + IP, J + JP, K + KP);
          if (f.nf[q] == 0) { double F = f.ff[q]; SUMF = SUMF + F; SUMP = SUMP + F * PP0[q]; }
        }
    v = (SUMF < 1.0e-20) ? 0.0 : SUMP / SUMF;
  }
  PPN[c] = v;
  CELL_LOOP_END
}

#undef A
#undef XX_
#undef YY_
#undef ZZ_

// ------------------------------------------------------------ launchers
#define RL(kern, ...) (kern<<<row_blocks(g), ROW_THREADS, 0, s>>>(__VA_ARGS__), count_launch())
#define CL(kern, ...) (kern<<<cell_grid(g), CELL_THREADS, 0, s>>>(__VA_ARGS__), count_launch())
#define SCL(kern, ...) (kern<<<cell_grid(g, SCAN_K), CELL_THREADS, 0, s>>>(__VA_ARGS__), count_launch())
void launch_fconv(cudaStream_t s, const Geo &g, const Fld &f, const Prm &p, double *a, double *b, double *c) { CL(k_fconv, g, f, p, a, b, c); }
void launch_feuler(cudaStream_t s, const Geo &g, const Fld &f, const Prm &p, const double *a, const double *b, const double *c) { CL(k_feuler, g, f, p, a, b, c); }
void launch_fmod1(cudaStream_t s, const Geo &g, const Fld &f, int *nlim) {
  CL(k_fmod1_count, g, f, nlim);
  SCL(k_fmod1_redist, g, f, nlim);
  CL(k_fmod1_target, g, f);
  SCL(k_fmod1_clamp, g, f);
}
void launch_fcut(cudaStream_t s, const Geo &g, const Fld &f, const Prm &p, double *rbs, double *rbc) { RL(k_fcut, g, f, p, rbs, rbc); }
void launch_fnf_init(cudaStream_t s, const Geo &g, const Fld &f, const Prm &p) { CL(k_fnf_init, g, f, p); }
void launch_fnf_sweep(cudaStream_t s, const Geo &g, int *nf, int *nch, int *done, int *iter, int cap, int *err) {
  SCL(k_fnf_mark7, g, nf, done);
  SCL(k_fnf_to8, g, nf, done);
  SCL(k_fnf_markm7, g, nf, nch, done);
  k_fnf_check<<<1, 1, 0, s>>>(nch, done, iter, cap, err);
  count_launch();
  SCL(k_fnf_m7to8, g, nf, done);
}
void launch_fbubup(cudaStream_t s, const Geo &g, const Fld &f, const Prm &p, const unsigned char *active) {
  int n = (g.NI - 2) * (g.NJ - 2);
  k_fbubup<<<(n + 255) / 256, 256, 0, s>>>(g, f, p, active);
  count_launch();
}
void launch_fnfprv(cudaStream_t s, const Geo &g, const Fld &f, int *err) { SCL(k_fnfprv, g, f, err); }
void launch_cindc(cudaStream_t s, const Geo &g, const Fld &f, int *nums) { SCL(k_cindc, g, f, nums); }
void launch_bsppfl(cudaStream_t s, const Geo &g, const Fld &f, const double *pp0, double *ppn) { CL(k_bsppfl, g, f, pp0, ppn); }
#undef RL
#undef CL
#undef SCL

}  // namespace cadmas
