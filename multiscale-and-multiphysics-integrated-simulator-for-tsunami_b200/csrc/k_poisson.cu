// k_poisson.cu -- pressure-Poisson assembly, MILU-BiCGSTAB and correction.
//
//   k_vpcoef            VF_VPCOEF (vf_vpcoef.f:117-437)
//   k_dcmp  (tile)      VF_MZDCMP (vf_mzdcmp.f:53-67)
//   k_sweep_cp, k_sweep VF_MZFRWD (vf_mzfrwd.f:37-48), optionally fused with
//    (tile)             the SpMV VF_MZAX (vf_mzax.f:42-56) of its input, and
//                       VF_MZBKWD (vf_mzbkwd.f:37-47)
//   slab, flat kernels  the vector updates and VF_MZIP dot products of
//                       VF_M1BCGS (vf_m1bcgs.f:76-266)
//   k_vmodif            VF_VMODIF (vf_vmodif.f:58-215)
//
// MILU is a lexicographic recurrence.  A tile of TI x TJ z-columns is one
// thread block; thread (ti,tj) owns column (is+ti, js+tj) and at wavefront
// step s processes k = 2 + s - ti - tj, so X(i-1,j,k) and X(i,j-1,k) were
// produced by the neighbouring threads at step s-1 and X(i,j,k-1) by the
// thread itself.  Every cell is evaluated with exactly the expression and
// operand order of the sequential loop, so a single tile covering the
// interior reproduces the serial reference bit for bit.  Several tiles form
// the block-Jacobi preconditioner that the reference itself applies when it
// runs on NPI x NPJ MPI ranks (each rank factors and sweeps its own x-y
// block; neighbour terms outside the block are coef*0*0 because the rank's
// halo DD and coefficients are zero).
#include <mutex>
#include "cadmas_dev.cuh"
#include "kernels.h"
#include "sweep_cp.cuh"
#include <algorithm>

namespace cadmas {

#define A(a, i, j, k) a[cid(g, i, j, k)]
#define XX_(m, i) gx(g, m, i)
#define YY_(m, j) gy(g, m, j)
#define ZZ_(m, k) gz(g, m, k)

// ------------------------------------------------------------- VF_VPCOEF
// A fluid cell loads its flags and the 26 values of its faces together: with
// the loads in the branches that use them 917 us on 1026x130x130 cells (1.8
// GB), 610 us with 116 registers, 509 us with 64.
__global__ void __launch_bounds__(CELL_THREADS, 8) k_vpcoef(Geo g, Fld f, Prm p, SysPtr A_, int *err) {
  const double DTI = 1.0 / p.dtnow, TR = p.dtnow / p.rho0, PPS = 0.0;
  const double *GGV = f.ggv, *GLV = f.glv, *FF = f.ff, *PP = f.pp;
  CELL_LOOP_BEGIN(g)
  const long long c = cid(g, I, J, K);
  double AD = 0.0, ALI = 0.0, ALJ = 0.0, ALK = 0.0, AUI = 0.0, AUJ = 0.0, AUK = 0.0, BB = 0.0;
  const int N = ld_now(f.nf + c), IC = ld_now(f.indc + c);
  if (IC == -1) {
    AD = 1.0;
  } else if (N == 0) {
    const int IM = I - 1, IP = I + 1, JM = J - 1, JP = J + 1, KM = K - 1, KP = K + 1;
    double AXY = XX_(2, I) * YY_(2, J), AXZ = XX_(2, I) * ZZ_(2, K), AYZ = YY_(2, J) * ZZ_(2, K);
    double AVL = XX_(2, I) * YY_(2, J) * ZZ_(2, K);
    double AIM, AIP, AJM, AJP, AKM, AKP, GV;
    // everything that a fluid cell may use, loaded together
    const long long sk = (long long)g.NI * g.NJ, last = g.N - 1;
    const long long xm = max(c - 1, 0LL), xp = min(c + 1, last), ym = max(c - g.NI, 0LL), yp = min(c + g.NI, last),
                    zm = max(c - sk, 0LL), zp = min(c + sk, last);
    const int ix = ld_now(f.indx + c), ixp = ld_now(f.indx + xp), iy = ld_now(f.indy + c), iyp = ld_now(f.indy + yp),
              iz = ld_now(f.indz + c), izp = ld_now(f.indz + zp);
    const double gc = ld_now(GGV + c), gxm = ld_now(GGV + xm), gxp = ld_now(GGV + xp), gym = ld_now(GGV + ym),
                 gyp = ld_now(GGV + yp), gzm = ld_now(GGV + zm), gzp = ld_now(GGV + zp);
    const double lc = ld_now(GLV + c), lxm = ld_now(GLV + xm), lxp = ld_now(GLV + xp), lym = ld_now(GLV + ym),
                 lyp = ld_now(GLV + yp), lzm = ld_now(GLV + zm), lzp = ld_now(GLV + zp);
    const double ax = ld_now(f.ggx + c), axp = ld_now(f.ggx + xp), ay = ld_now(f.ggy + c), ayp = ld_now(f.ggy + yp),
                 az = ld_now(f.ggz + c), azp = ld_now(f.ggz + zp);
    const double uc = ld_now(f.uu + c), up = ld_now(f.uu + xp), vc = ld_now(f.vv + c), vp = ld_now(f.vv + yp),
                 wc = ld_now(f.ww + c), wp = ld_now(f.ww + zp);
    int IS = ix;
    if (IS == 0) {
      GV = XX_(6, I) * (XX_(2, I) * gc / lc + XX_(2, IM) * gxm / lxm);
      AIM = AYZ * XX_(5, I) * ax * GV; ALI = -AIM;
    } else if (IS >= 1) {
      if (indb(f, 3, IS) == 4 || (indb(f, 3, IS) == 5 && I == 2 && p.fixlvl[0]))  // vf_vpcoef.f:158-175
        AIM = 2.0 * AYZ * XX_(4, I) * ax * gc / lc;
      else AIM = 0.0;
    } else { AIM = 0.0; atomicOr(err, ERR_PG); }
    IS = ixp;
    if (IS == 0) {
      GV = XX_(6, IP) * (XX_(2, IP) * gxp / lxp + XX_(2, I) * gc / lc);
      AIP = AYZ * XX_(5, IP) * axp * GV; AUI = -AIP;
    } else if (IS >= 1) {
      if (indb(f, 3, IS) == 4 || (indb(f, 3, IS) == 5 && IP == g.NI && p.fixlvl[1]))
        AIP = 2.0 * AYZ * XX_(4, I) * axp * gc / lc;
      else AIP = 0.0;
    } else { AIP = 0.0; atomicOr(err, ERR_PG); }
    IS = iy;
    if (IS == 0) {
      GV = YY_(6, J) * (YY_(2, J) * gc / lc + YY_(2, JM) * gym / lym);
      AJM = AXZ * YY_(5, J) * ay * GV; ALJ = -AJM;
    } else if (IS >= 1) {
      if (indb(f, 3, IS) == 4 || (indb(f, 3, IS) == 5 && J == 2 && p.fixlvl[2]))
        AJM = 2.0 * AXZ * YY_(4, J) * ay * gc / lc;
      else AJM = 0.0;
    } else { AJM = 0.0; atomicOr(err, ERR_PG); }
    IS = iyp;
    if (IS == 0) {
      GV = YY_(6, JP) * (YY_(2, JP) * gyp / lyp + YY_(2, J) * gc / lc);
      AJP = AXZ * YY_(5, JP) * ayp * GV; AUJ = -AJP;
    } else if (IS >= 1) {
      if (indb(f, 3, IS) == 4 || (indb(f, 3, IS) == 5 && JP == g.NJ && p.fixlvl[3]))
        AJP = 2.0 * AXZ * YY_(4, J) * ayp * gc / lc;
      else AJP = 0.0;
    } else { AJP = 0.0; atomicOr(err, ERR_PG); }
    IS = iz;
    if (IS == 0) {
      GV = ZZ_(6, K) * (ZZ_(2, K) * gc / lc + ZZ_(2, KM) * gzm / lzm);
      AKM = AXY * ZZ_(5, K) * az * GV; ALK = -AKM;
    } else if (IS >= 1) {
      if (indb(f, 3, IS) != 4) AKM = 0.0;
      else AKM = 2.0 * AXY * ZZ_(4, K) * az * gc / lc;
    } else { AKM = 0.0; atomicOr(err, ERR_PG); }
    IS = izp;
    if (IS == 0) {
      GV = ZZ_(6, KP) * (ZZ_(2, KP) * gzp / lzp + ZZ_(2, K) * gc / lc);
      AKP = AXY * ZZ_(5, KP) * azp * GV; AUK = -AKP;
    } else if (IS >= 1) {
      if (indb(f, 3, IS) != 4) AKP = 0.0;
      else AKP = 2.0 * AXY * ZZ_(4, K) * azp * gc / lc;
    } else { AKP = 0.0; atomicOr(err, ERR_PG); }
    AD = AKM + AJM + AIM + AIP + AJP + AKP;
    double VD = AYZ * (axp * up - ax * uc) +
                AXZ * (ayp * vp - ay * vc) +
                AXY * (azp * wp - az * wc);
    double VQ = -(gc - gc) * DTI * AVL;
    // wave source line (vf_vpcoef.f:349-350)
    if (p.iws == I) VQ = 2.0 * ZZ_(2, K) * f.srcuv[(J - 1) + (long long)g.NJ * (K - 1)] * YY_(2, J);
    if (p.jws == J) VQ = 2.0 * ZZ_(2, K) * f.srcuv[(I - 1) + (long long)g.NI * (K - 1)] * XX_(2, I);
    BB = VD - VQ;
  } else if (N == 5) {
    double PSI = ZZ_(3, K) / (0.5 * ZZ_(2, K - 1) + FF[c] * ZZ_(2, K));
    AD = 1.0; ALK = PSI - 1.0;
    BB = -TR * ((1.0 - PSI) * A(PP, I, J, K - 1) + PSI * PPS - PP[c]);
  } else if (N == 6) {
    double PSI = ZZ_(3, K + 1) / (0.5 * ZZ_(2, K + 1) + FF[c] * ZZ_(2, K));
    AD = 1.0; AUK = PSI - 1.0;
    BB = -TR * ((1.0 - PSI) * A(PP, I, J, K + 1) + PSI * PPS - PP[c]);
  } else if (N == 3) {
    double PSI = YY_(3, J) / (0.5 * YY_(2, J - 1) + FF[c] * YY_(2, J));
    AD = 1.0; ALJ = PSI - 1.0;
    BB = -TR * ((1.0 - PSI) * A(PP, I, J - 1, K) + PSI * PPS - PP[c]);
  } else if (N == 4) {
    double PSI = YY_(3, J + 1) / (0.5 * YY_(2, J + 1) + FF[c] * YY_(2, J));
    AD = 1.0; AUJ = PSI - 1.0;
    BB = -TR * ((1.0 - PSI) * A(PP, I, J + 1, K) + PSI * PPS - PP[c]);
  } else if (N == 1) {
    double PSI = XX_(3, I) / (0.5 * XX_(2, I - 1) + FF[c] * XX_(2, I));
    AD = 1.0; ALI = PSI - 1.0;
    BB = -TR * ((1.0 - PSI) * A(PP, I - 1, J, K) + PSI * PPS - PP[c]);
  } else if (N == 2) {
    double PSI = XX_(3, I + 1) / (0.5 * XX_(2, I + 1) + FF[c] * XX_(2, I));
    AD = 1.0; AUI = PSI - 1.0;
    BB = -TR * ((1.0 - PSI) * A(PP, I + 1, J, K) + PSI * PPS - PP[c]);
  } else {
    atomicOr(err, ERR_PG);
  }
  A_.ad[c] = AD; A_.ali[c] = ALI; A_.alj[c] = ALJ; A_.alk[c] = ALK;
  A_.aui[c] = AUI; A_.auj[c] = AUJ; A_.auk[c] = AUK; A_.bb[c] = BB;
  CELL_LOOP_END
}

// ----------------------------------------------------------- tile sweeps
struct TileGeo {
  int is, js, wi, wj;  // tile origin and width in cells
  int ti, tj;          // thread coordinates
  bool valid;
};
__device__ __forceinline__ TileGeo tile_geo(const Geo &g, const SkewGeo &q, int bx, int by) {
  TileGeo t;
  t.is = 2 + bx * q.TI;
  t.js = 2 + by * q.TJ;
  t.wi = min(q.TI, g.NI - t.is);  // interior cells is..NI-1
  t.wj = min(q.TJ, g.NJ - t.js);
  t.ti = threadIdx.x % q.TIp;
  t.tj = threadIdx.x / q.TIp;
  t.valid = (t.ti < t.wi) && (t.tj < t.wj);  // also false on the padding column ti = TI
  return t;
}

// ---------------------------------------------------------------------------
// Column prefetch.  Each thread streams its own column through a ring of R
// shared-memory slots with cp.async, D wavefront steps ahead of use, so a
// step only waits for shared memory and one barrier.  Values of the
// neighbouring columns at the same plane are read from the neighbours' ring
// slots: the left/lower neighbour handled plane k one step earlier (slot
// s-1), the right/upper one handles it one step later (slot s+1, prefetched
// long before).  R = D+3: at step s a thread refills slot s+D before the
// step's barrier, while a slower neighbour may still read slot s-2.
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <typename V> __device__ __forceinline__ void cp_async_v(V *smem, const V *gmem) {
  if (sizeof(V) == 8) cp_async8(smem, gmem);
  else cp_async4(smem, gmem);
}

// Ring layout in dynamic shared memory: V r[R][NV][T], then the exchange
// buffers V xb[2][T], then int ri[R][T].
template <int NV, typename V> struct Ring {
  V *r;
  int *ri;
  V *xb;
  int T, R;
  __device__ __forceinline__ V &v(int slot, int q, int t) const { return r[((slot * NV) + q) * T + t]; }
  __device__ __forceinline__ int &ind(int slot, int t) const { return ri[slot * T + t]; }
};
template <int NV, typename V> __device__ __forceinline__ Ring<NV, V> ring_setup(int T, int R) {
  extern __shared__ __align__(16) double sm[];
  Ring<NV, V> g;
  g.T = T; g.R = R;
  g.r = reinterpret_cast<V *>(sm);
  g.xb = g.r + (size_t)R * NV * T;
  g.ri = (int *)(g.xb + 2 * T);
  return g;
}
inline size_t ring_bytes(int NV, int T, int R, size_t es = sizeof(double)) {
  return (size_t)R * NV * T * es + 2 * (size_t)T * es + (size_t)R * T * sizeof(int);
}

// ----------------------------------------------------- tile-skewed layout
// The MILU kernels visit, at wavefront step s, cell (is+ti, js+tj,
// k = 2+s-ti-tj) with thread t = ti + TIp*tj.  The arrays that stay constant
// through a solve (7 coefficients, DD, INDC), the right-hand side and the
// BiCGSTAB vectors are stored tile by tile in that visiting order,
//     sl(b, w, t) = (b*WS + w)*T + t,   w = (k-2) + ti + tj,
// b = tile index, w = 0 .. W-1 (SkewGeo says how tiles overlap), so the T
// values a block needs at one step are contiguous and every load of the
// sweep coalesces.
__device__ __forceinline__ long long sl_index(const SkewGeo &q, int b, int w, int t) {
  return ((long long)b * skew_stride(q) + w) * q.T + t;
}

// Store the coefficients AD, ALI, ALJ, ALK, AUI, AUJ, AUK of column t of a
// slab as chunks, DD = 0.
__device__ __forceinline__ void sys_put(double *sys, long long slab, int T, int t, const double *v) {
  const double e[8] = {v[4], v[5], v[6], 0.0, v[1], v[2], v[3], v[0]};
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<double2 *>(sys + sys_chunk<double>(slab, c, T, t)) = make_double2(e[2 * c], e[2 * c + 1]);
}

// Copy the Poisson system (7 coefficients, interleaved per slab; DD set to
// 0 for MZDCMP to fill), INDC, BB and X0 into the skewed layout (e counts
// the nb*W*T wavefront entries).  Columns of a tile past the grid get 0
// (INDC -1).  warm: keep the
// previous solution already in xsl as the initial guess (0 where INDC is
// now -1) instead of X0.
__device__ __forceinline__ void to_skew_elem(const Geo &g, const SkewGeo &q, const SysPtr &A_, const int *INDC,
                                             const SkewSys &S, const double *X0, double *bsl, double *xsl, int warm,
                                             long long e) {
  {
    const int t = (int)(e % q.T);
    const long long bw = e / q.T;
    const int w = (int)(bw % q.W), b = (int)(bw / q.W);
    const int ti = t % q.TIp, tj = t / q.TIp;
    const int I = 2 + (b % q.ntx) * q.TI + ti, J = 2 + (b / q.ntx) * q.TJ + tj, k = 2 + w - ti - tj;
    if (ti >= q.TI || k < 2 || k > g.NK - 1) return;  // the entry is not this tile's
    const long long slab = (long long)b * skew_stride(q) + w, x = slab * q.T + t;
    double v[7] = {0, 0, 0, 0, 0, 0, 0}, bv = 0.0, xv = 0.0;
    int ic = -1;
    if (I <= g.NI - 1 && J <= g.NJ - 1) {
      const long long c = cid(g, I, J, k);
      v[0] = A_.ad[c]; v[1] = A_.ali[c]; v[2] = A_.alj[c]; v[3] = A_.alk[c];
      v[4] = A_.aui[c]; v[5] = A_.auj[c]; v[6] = A_.auk[c];
      ic = INDC[c];
      bv = A_.bb[c];
      xv = warm ? (ic != -1 ? xsl[x] : 0.0) : X0[c];
    }
    sys_put(S.sys, slab, q.T, t, v);
    S.sys[sys_t(slab, q.T, t)] = 0.0;
    S.indc[x] = ic;
    bsl[x] = bv;
    xsl[x] = xv;
  }
}
__global__ void k_to_skew(Geo g, SkewGeo q, SysPtr A_, const int *INDC, SkewSys S, const double *X0,
                          double *bsl, double *xsl, int warm) {
  pdl_enter();
  const long long n = (long long)q.nb * q.W * q.T;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    to_skew_elem(g, q, A_, INDC, S, X0, bsl, xsl, warm, e);
}

// The same conversion, one block per row tj of a layout tile b: the row's
// interior cells of all layers, (NK-2) x TI values of two arrays at a
// time, are staged in shared memory with coalesced loads and then written
// slab by slab (TIp consecutive entries of a slab per row): the two arrays
// of a chunk of the system together, then BB with X0 (or, warm, BB alone).
// Same values as to_skew_elem; used when two panels fit in shared memory.
__global__ void k_to_skew_rows(Geo g, SkewGeo q, SysPtr A_, const int *INDC, SkewSys S, const double *X0,
                               double *bsl, double *xsl, int warm) {
  extern __shared__ __align__(16) double pan[];  // [2][(NK-2) * TI]
  pdl_enter();
  const int b = blockIdx.x / q.TJ, tj = blockIdx.x % q.TJ;
  const int TI = q.TI, TIp = q.TIp, T = q.T, nk = g.NK - 2;
  const int is = 2 + (b % q.ntx) * TI, J = 2 + (b / q.ntx) * q.TJ + tj;
  const int wi = (J <= g.NJ - 1) ? min(TI, g.NI - is) : 0;  // columns of the row inside the interior
  const int npan = nk * TI, nent = (nk + TI - 1) * TIp;  // the row's slabs tj .. tj+nk+TI-2
  const long long slab0 = (long long)b * skew_stride(q) + tj;
  int *ipan = reinterpret_cast<int *>(pan);
  // INDC, then T = 0, INDC and the warm guess
#pragma unroll 4
  for (int x = threadIdx.x; x < npan; x += blockDim.x) {
    const int k = 2 + x / TI, ti = x % TI;
    ipan[x] = ti < wi ? INDC[cid(g, is + ti, J, k)] : -1;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < nent; x += blockDim.x) {
    const int w = x / TIp, ti = x % TIp, t = ti + TIp * tj;
    if (ti >= TI || (unsigned)(w - ti) >= (unsigned)nk) continue;  // the entry is not this tile's
    const int ic = ipan[(w - ti) * TI + ti];
    const long long e = (slab0 + w) * T + t;
    S.indc[e] = ic;
    S.sys[sys_t(slab0 + w, T, t)] = 0.0;
    if (warm) xsl[e] = ic != -1 ? xsl[e] : 0.0;
  }
  // chunks {AUI,AUJ}, {AUK,DD = 0}, {ALI,ALJ}, {ALK,AD}; BB and X0
  const double *src[10] = {A_.aui, A_.auj, A_.auk, nullptr, A_.ali, A_.alj, A_.alk, A_.ad, A_.bb, warm ? nullptr : X0};
#pragma unroll 1
  for (int a = 0; a < 5; ++a) {
    __syncthreads();
    const double *s0 = src[2 * a], *s1 = src[2 * a + 1];
#pragma unroll 4
    for (int x = threadIdx.x; x < npan; x += blockDim.x) {
      const int k = 2 + x / TI, ti = x % TI;
      const long long c = cid(g, is + ti, J, k);
      pan[x] = ti < wi ? s0[c] : 0.0;
      pan[npan + x] = ti < wi && s1 ? s1[c] : 0.0;
    }
    __syncthreads();
    for (int x = threadIdx.x; x < nent; x += blockDim.x) {
      const int w = x / TIp, ti = x % TIp, t = ti + TIp * tj;
      if (ti >= TI || (unsigned)(w - ti) >= (unsigned)nk) continue;
      const int p = (w - ti) * TI + ti;
      const double v0 = pan[p], v1 = pan[npan + p];
      if (a < 4) {
        *reinterpret_cast<double2 *>(S.sys + sys_chunk<double>(slab0 + w, a, T, t)) = make_double2(v0, v1);
      } else {
        bsl[(slab0 + w) * T + t] = v0;
        if (!warm) xsl[(slab0 + w) * T + t] = v1;
      }
    }
  }
}
// Shared memory of k_to_skew_rows (0: the panels do not fit, k_to_skew).
static size_t to_skew_rows_bytes(const Geo &g, const SkewGeo &q) {
  const size_t b = 2 * (size_t)(g.NK - 2) * q.TI * sizeof(double);
  return b <= 64 * 1024 ? b : 0;
}

// Value of a skewed vector at the cell (ti,tj,k) of tile (bx,by), where ti
// and tj may step one past the tile into the neighbouring tile; cells
// outside the interior are the zero ghost layer of the reference vectors.
__device__ __forceinline__ long long skew_nb(const Geo &g, const SkewGeo &q, int bx, int by, int ti, int tj,
                                             int k) {
  if (ti < 0) { bx -= 1; ti += q.TI; } else if (ti >= q.TI) { bx += 1; ti -= q.TI; }
  if (tj < 0) { by -= 1; tj += q.TJ; } else if (tj >= q.TJ) { by += 1; tj -= q.TJ; }
  const int I = 2 + bx * q.TI + ti, J = 2 + by * q.TJ + tj;
  if (bx < 0 || by < 0 || I > g.NI - 1 || J > g.NJ - 1 || k < 2 || k > g.NK - 1) return -1;
  return sl_index(q, bx + q.ntx * by, (k - 2) + ti + tj, ti + q.TIp * tj);
}
__device__ __forceinline__ double skew_at(const Geo &g, const SkewGeo &q, const double *X, int bx, int by,
                                          int ti, int tj, int k) {
  const long long e = skew_nb(g, q, bx, by, ti, tj, k);
  return e < 0 ? 0.0 : X[e];
}
// Asynchronous copy of a neighbour value into shared memory (0 for ghosts).
__device__ __forceinline__ void skew_fetch(double *dst, const Geo &g, const SkewGeo &q, const double *X, int bx,
                                           int by, int ti, int tj, int k) {
  const long long e = skew_nb(g, q, bx, by, ti, tj, k);
  if (e < 0) *dst = 0.0;
  else cp_async8(dst, X + e);
}

// ------------------------------------------------------------ VF_MZDCMP
// One thread block per preconditioner block (TI x TJ*split columns; with
// split = 2 the block's columns live in two layout tiles), one thread per
// column, wavefront step s at k = 2+s-ti-tj.  Ring values: 0 AD, 1 ALI,
// 2 ALJ, 3 ALK, 4 AUI, 5 AUJ, 6 AUK; DD is written in the skewed layout.
template <int D, typename V>
__device__ __forceinline__ void dcmp_body(const Geo &g, const SkewGeo &q, V U, const SkewSysT<V> &S, int *pivot_bad,
                                          int bx, int by) {
  constexpr int NV = 7, R = D + 3;
  const int TIp = q.TIp, TJl = q.TJ, Tl = q.T;      // layout tile
  const int TJb = TJl * q.split, Tb = TIp * TJb;    // preconditioner block
  Ring<NV, V> rg = ring_setup<NV, V>(Tb, R);
  const int tid = threadIdx.x;
  const int ti = tid % TIp, tj = tid / TIp;
  const int is = 2 + bx * q.TI, js = 2 + by * TJb;
  const int wi = min(q.TI, g.NI - is), wj = min(TJb, g.NJ - js);
  const bool valid = ti < wi && tj < wj;
  const int r = tj / TJl, tjl = tj % TJl;
  const long long bl = bx + (long long)q.ntx * (by * q.split + r);  // layout tile
  // slab of step s: w = (k-2) + ti + tjl = s - r*TJl
  const long long slab0 = bl * skew_stride(q) - (long long)r * TJl;
  const int tl = ti + TIp * tjl;
  const int nsteps = (g.NK - 2) + (wi - 1) + (wj - 1);
  auto prefetch = [&](int s) {
    const int k = 2 + s - ti - tj;
    if (valid && k >= 2 && k <= g.NK - 1) {
      const long long slab = slab0 + s, e = slab * Tl + tl;
      const int sl = s % R;
      constexpr int cs[7] = {SYS_AD, SYS_ALI, SYS_ALJ, SYS_ALK, SYS_AUI, SYS_AUJ, SYS_AUK};
#pragma unroll
      for (int c = 0; c < 7; ++c) cp_async_v(&rg.v(sl, c, tid), S.sys + sys_at<V>(slab, cs[c], Tl, tl));
      cp_async4(&rg.ind(sl, tid), S.indc + e);
    }
    cp_commit();
  };
#pragma unroll 1
  for (int s = 0; s < D; ++s) prefetch(s);
  V dk1 = V(0), au3 = V(0);  // DD(i,j,k-1) and AU3 of (i,j,k-1); k-1 = 1 is the zero ghost layer
  const V z = V(0), one = V(1);
  bool bad = false;
  const int T = Tb;
  for (int s = 0; s < nsteps; ++s) {
    prefetch(s + D);
    cp_wait<D - 1>();
    __syncthreads();
    const int k = 2 + s - ti - tj;
    const int sl = s % R, slp = (s + R - 1) % R, cur = s & 1, prv = cur ^ 1;
    if (valid && k >= 2 && k <= g.NK - 1) {
      V dd = z;
      if (rg.ind(sl, tid) != -1) {
        V d1 = z, a1, d2 = z, a2;
        if (ti > 0) {
          d1 = rg.xb[prv * T + tid - 1];
          a1 = rg.v(slp, 4, tid - 1) + U * (rg.v(slp, 5, tid - 1) + rg.v(slp, 6, tid - 1));
        } else {
          a1 = z + U * (z + z);
        }
        if (tj > 0) {
          d2 = rg.xb[prv * T + tid - TIp];
          a2 = rg.v(slp, 5, tid - TIp) + U * (rg.v(slp, 4, tid - TIp) + rg.v(slp, 6, tid - TIp));
        } else {
          a2 = z + U * (z + z);
        }
        dd = one / (rg.v(sl, 0, tid) - rg.v(sl, 1, tid) * d1 * a1 - rg.v(sl, 2, tid) * d2 * a2 -
                    rg.v(sl, 3, tid) * dk1 * au3);
        if (dd <= z) bad = true;
      }
      S.sys[sys_at<V>(slab0 + s, SYS_DD, Tl, tl)] = dd;
      rg.xb[cur * T + tid] = dd;
      dk1 = dd;
      au3 = rg.v(sl, 6, tid) + U * (rg.v(sl, 4, tid) + rg.v(sl, 5, tid));
    }
  }
  cp_wait<0>();
  if (bad) atomicOr(pivot_bad, 1);
}
template <int D, typename V>
__global__ void k_dcmp(Geo g, SkewGeo q, V U, SkewSysT<V> S, int *pivot_bad) {
  pdl_enter();
  dcmp_body<D, V>(g, q, U, S, pivot_bad, (int)blockIdx.x, (int)blockIdx.y);
}

// ------------------------------------------------ bulk-copy slab pipeline
// The sweeps read, at every wavefront step, one contiguous slab of T
// values from each of 5 or 9 skewed arrays.  A producer warp moves those
// slabs into a ring of R = D+2 shared-memory slots with cp.async.bulk, D
// steps ahead, each slot completing on its own mbarrier (transaction
// count); the T consumer threads wait on the mbarrier of the step they
// need and then work purely from shared memory.  One block barrier per
// step orders the exchange of the sweep values between neighbouring
// columns and frees the slot of step s-2 for the producer.  launch_sweep says
// which sweeps run in this form.
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}
// Wait for the phase `parity` of an mbarrier, giving up after limit_ns.
__device__ __noinline__ bool mbar_wait_slow(unsigned bar, unsigned parity, unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (mbar_try(bar, parity)) return true;
    if (global_ns() - t0 > limit_ns) return false;
  }
}
// Non-blocking test of a phase: its latency overlaps the instructions that
// follow until the predicate is used.
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The limit comes from the solve state, read only once a wait has to
// spin, so that it occupies no register in the sweeps' step loop.
__device__ __noinline__ bool mbar_wait_st(unsigned bar, unsigned parity, const SolveState *st) {
  return mbar_wait_slow(bar, parity, (unsigned long long)st->wait_ns);
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, const SolveState *st) {
  return mbar_try(bar, parity) || mbar_wait_st(bar, parity, st);
}

// ------------------------------------- cluster exchange (precond_split 2)
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Store into another CTA of the cluster and credit the stored bytes to an
// mbarrier there (transaction count); no release of earlier stores.
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];\n" ::"r"(addr), "d"(v),
               "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, float v, unsigned mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];\n" ::"r"(addr), "f"(v),
               "r"(mbar)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_cluster(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait (limit_ns) acquiring what other CTAs of the cluster released.
__device__ __noinline__ bool mbar_wait_cluster_slow(unsigned bar, unsigned parity, unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (mbar_try_cluster(bar, parity)) return true;
    if (global_ns() - t0 > limit_ns) return false;
  }
}
__device__ __noinline__ bool mbar_wait_cluster_st(unsigned bar, unsigned parity, const SolveState *st) {
  return mbar_wait_cluster_slow(bar, parity, (unsigned long long)st->wait_ns);
}
__device__ __forceinline__ bool mbar_wait_cluster(unsigned bar, unsigned parity, const SolveState *st) {
  return mbar_try_cluster(bar, parity) || mbar_wait_cluster_st(bar, parity, st);
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}

// ------------------------------------ VF_MZFRWD (+VF_MZAX) and VF_MZBKWD
// One block per tile: T consumer threads (thread t = ti + TIp*tj owns
// column (ti,tj)) and one producer warp.  MODE (SweepMode):
//   SWEEP_FWD     T = MINV_L * Y, Y given (skewed);  vf_mzfrwd.f
//   SWEEP_FWD_AX  T = MINV_L * (A*P), A*P formed on the fly (VF_MZAX
//                 then VF_MZFRWD: vf_mzax.f:46-53, vf_mzfrwd.f)
//   SWEEP_BWD     X = MINV_U * T;  vf_mzbkwd.f
// The forward sweeps write T into the system block (SYS_T), where the
// backward sweep's one bulk copy per step finds it with AUI..DD; the
// backward sweep writes X in the skewed layout.  Forward step s visits
// k = 2+s-ti-tj, backward step s visits k = NK-1-(s-ri-rj) (ri, rj the
// distances from the far corner), so step s of every thread is one slab.
// A cell is computed where DD != 0: MZDCMP gives DD = 0 exactly on
// INDC = -1 and a positive (or NaN) DD elsewhere, and a zero or negative
// pivot ends the solve before any sweep runs.
//
// Between two block barriers lie the recurrence of step s (the neighbours'
// results of step s-1 are read, combined in five dependent operations and
// published) and the preparation of step s+1, which does not depend on it:
// the ring loads, the 7-term product A*P and the products ALI*DD(i-1) etc.
// of the recurrence.  Both are straight-line and scheduled into one another;
// a column without a cell at a step computes on what its slot holds and
// stores nothing.  A warp of the fused forward sweep whose columns have
// nothing to compute (air, obstacles) skips the preparation: 1024x128x128
// cells with 1 % water, split 16x16 blocks, forward sweeps 63.7 -> 56.5 ms a
// step, for 1 % more on the 512x32x96 flume.  The expressions and their evaluation order are those of
// the reference loops, so the results do not change.  The depth D is a
// run-time value: with D = 8 compiled in a step of the cluster form takes
// between 1 % less and 1 % more.
template <int MODE, typename V, int CS>
__device__ __forceinline__ void sweep_body(const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *vin,
                                           V *vout, SolveState *st, const V *vin2, double *rb, int bx, int by,
                                           const int D) {
  constexpr bool BWD = MODE >= SWEEP_BWD;
  constexpr int NDOT = sweep_ndot(MODE);
  // CS = 2: the thread blocks of a cluster are the two layout tiles of one
  // preconditioner block; every block of a cluster runs through the two
  // cluster barriers below, so none returns early.
  const bool skip = st->done || (CS == 2 && by >= q.nb / q.ntx);
  if (CS == 1 && skip) return;
  if (CS == 2 && skip) {
    cluster_barrier();
    cluster_barrier();
    return;
  }
  const int R = D + 2;
  constexpr int AHEAD = (MODE == SWEEP_FWD_AX) ? 2 : 1;  // preparing step s+1 reads the slot of step s+AHEAD
  extern __shared__ __align__(16) double sm[];
  const int T = q.T, TIp = q.TIp;
  const int Tc = (T + 31) & ~31;
  constexpr int ES = (int)sizeof(V);
  const int SS = sweep_slot(q, MODE, ES);
  // position in a slot of the coefficients' run, and in it of a column's coefficient
  constexpr int RUN = MODE == SWEEP_FWD_AX ? 0 : 1;  // in units of T (after Y or T)
  auto co = [&](const V *slot, int c, int tt) { return slot[RUN * T + sys_in_run<V>(c, T, tt)]; };
  // The coefficients of a column, e[c - SYS_AUI] of those that the mode uses,
  // as 16-byte loads of their chunks: one coefficient at a time a warp's
  // loads have two-way (FP64) or four-way (FP32) bank conflicts.  Fused
  // forward sweeps of 16x16 blocks split over clusters, ms per step: 512x32x96
  // FP64 15.2 -> 14.2; 1024x128x128 FP64 139.7 -> 136.2, FP32 99.3 -> 89.8.
  constexpr int G = 16 / ES;
  struct alignas(16) Chunk { V v[G]; };
  struct Coef { V e[8]; };
  auto coefs = [&](const V *slot, int tt) {
    Coef f;
#pragma unroll
    for (int c = 0; c < (BWD ? 4 : 8) / G; ++c) {
      const Chunk k = *reinterpret_cast<const Chunk *>(slot + RUN * T + (c * T + tt) * G);
#pragma unroll
      for (int i = 0; i < G; ++i) f.e[c * G + i] = k.v[i];
    }
    return f;
  };
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(sm);
  V *ring = reinterpret_cast<V *>(sm + ((R + 1) & ~1));
  V *xb = ring + (size_t)R * SS;
  const int tid = threadIdx.x, b = bx + q.ntx * by;
  TileGeo t = tile_geo(g, q, bx, by);
  const int nsteps = (g.NK - 2) + (t.wi - 1) + (t.wj - 1);
  const bool producer = tid >= Tc;
  const int lane = tid & 31;

  // Cluster exchange (CS = 2).  The forward sweeps need, on row 0 of the
  // upper tile, the result and DD of row TJ-1 of the lower tile at the
  // same k; the backward sweep needs the reverse.  The sending row stores
  // its values of step u into slot u of the receiver's xin/din with
  // st.async, each store crediting its bytes to the receiver's xfull[u],
  // which the receiver armed at start-up for one full row (TIp values of x,
  // and of DD for the forward sweeps); a slot is written once per sweep.
  const int NX = q.W;                                   // slots: steps of a tile at most
  unsigned long long *xfull = reinterpret_cast<unsigned long long *>(xb + 2 * T);
  V *xin = reinterpret_cast<V *>(xfull + NX);
  V *din = xin + (size_t)NX * TIp;
  const int crank = (CS == 2) ? (by & 1) : 0;
  const int nty = q.nb / q.ntx;
  const bool has_up = CS == 2 && crank == 0 && by + 1 < nty;
  const bool has_lo = CS == 2 && crank == 1;
  const bool recv = BWD ? has_up : has_lo;
  const bool send = BWD ? has_lo : has_up;
  const bool srow = send && (BWD ? t.tj == 0 : t.tj == q.TJ - 1) && !producer;
  const bool rrow = recv && (BWD ? t.tj == t.wj - 1 : t.tj == 0) && !producer;
  // receiver's step lag: rows of the sending tile minus one
  const int lag = BWD ? min(q.TJ, g.NJ - (2 + (by + 1) * q.TJ)) - 1 : q.TJ - 1;
  unsigned r_xin = 0, r_din = 0, r_full = 0;            // the partner's xin, din, xfull
  if (CS == 2 && send) {
    const unsigned peer = cluster_rank() ^ 1u;
    r_xin = mapa(smem_u32(xin), peer);
    r_din = mapa(smem_u32(din), peer);
    r_full = mapa(smem_u32(xfull), peer);
  }

  // s_abort[c & 1]: a wait of some thread ran out of time during ring
  // cycle c.  Written during a cycle, read after its last barrier; the two
  // entries keep those reads apart from the writes of the next cycle.
  __shared__ int s_abort[2];
  if (tid == 0) {
    for (int r = 0; r < R; ++r) mbar_init(smem_u32(bar + r), 1);
    s_abort[0] = s_abort[1] = 0;
  }
  if (CS == 2 && recv) {
    const unsigned row_bytes = (unsigned)(TIp * ES * (BWD ? 1 : 2));
    for (int u = tid; u < NX; u += blockDim.x) {
      mbar_init(smem_u32(xfull + u), 1u);
      mbar_expect_tx(smem_u32(xfull + u), row_bytes);
    }
  }
  if (MODE == SWEEP_FWD_AX) {  // halo values of absent neighbours stay 0 (ghost layer)
    const int nh = 2 * halo_span(q, ES) + 2 * TIp;
    for (int r = 0; r < R; ++r)
      for (int i = tid; i < nh; i += blockDim.x) ring[(size_t)r * SS + halo_left(q, ES) + i] = V(0);
  }
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  if (CS == 2) cluster_barrier();  // partner's barriers initialised before any remote arrival
  else __syncthreads();

  // Producer: lane l issues copy l of every step (at most 6); its fixed
  // part is worked out once here.
  const V *src0 = nullptr;
  SweepLane l0;
  l0.dlo = 1; l0.dhi = 0; l0.bytes = 0; l0.dst = 0; l0.wstride = 0;  // empty range: no copy
  if (producer && lane < sweep_ncopy(q, MODE) && sweep_lane(q, MODE, b, lane, l0, ES))
    src0 = (l0.arr == 0 ? S.sys : (l0.arr == 1 ? vin : vin2)) + l0.base;
  else { l0.dlo = 1; l0.dhi = 0; l0.bytes = 0; }
  const unsigned bar0 = smem_u32(bar), ring0 = smem_u32(ring);
  const int stall_from = producer ? st->stall_from : 0;  // read by the producer warp only
  auto issue = [&](int u, int slot) {
    if (u >= nsteps || u >= stall_from) return;
    const int w = BWD ? nsteps - 1 - u : u;
    const unsigned bslot = bar0 + 8u * slot;
    const unsigned dslot = ring0 + (unsigned)ES * (unsigned)(slot * SS);
    const bool v0 = (w >= l0.dlo && w <= l0.dhi);
    const unsigned bytes = __reduce_add_sync(0xffffffffu, v0 ? l0.bytes : 0);
    if (lane == 0) mbar_expect_tx(bslot, bytes);
    __syncwarp();
    if (v0) bulk_load(dslot + (unsigned)ES * l0.dst, src0 + (long long)w * l0.wstride, l0.bytes, bslot);
  };
  // data of step u sits in slot u % R, phase (u / R) & 1
  auto wait_data = [&](int u, int slot, unsigned parity) -> bool {
    return u >= nsteps || mbar_wait(bar0 + 8u * slot, parity, st);
  };

  if (producer) {
#pragma unroll 1
    for (int u = 0; u < D; ++u) issue(u, u);
  }

  // Column geometry: active steps slo..shi (k inside 2..NK-1).
  const int ri = t.wi - 1 - t.ti, rj = t.wj - 1 - t.tj;
  const bool ex0 = (t.ti == 0), ex1 = (t.ti == t.wi - 1), ey0 = (t.tj == 0), ey1 = (t.tj == t.wj - 1);
  const int slo = BWD ? ri + rj : t.ti + t.tj, shi = slo + g.NK - 3;
  const bool col = t.valid && !producer;
  const int hti = col ? t.ti : 0, htj = col ? t.tj : 0;  // in range for threads without a column too
  const int hl = halo_left(q, ES) + TIp * htj + halo_lofs(q, ES), hr = halo_right(q, ES) + TIp * htj,
            hd = halo_down(q, ES) + hti, hu = halo_up(q, ES) + hti;
  // forward: T into the system block; backward: X
  V *vp = BWD ? vout + ((long long)b * skew_stride(q) + nsteps - 1) * T + tid
                              : S.sys + sys_t((long long)b * skew_stride(q), T, tid);
  const long long vstep = BWD ? -(long long)T : (long long)SYS_N * T;

  // Neighbouring column's entry of the exchange buffer and of the ring
  // (the own entry where the tile has none; the value is then replaced).
  const int tr = min(tid, T - 1);  // threads past the layout's T columns read entry T-1 and store nothing
  const bool hx = BWD ? ri > 0 : t.ti > 0, hy = BWD ? rj > 0 : t.tj > 0;
  const int ox = col && hx ? tr + (BWD ? 1 : -1) : tr, oy = col && hy ? tr + (BWD ? TIp : -TIp) : tr;
  // P neighbours on the far side (inside the tile, else the halo)
  const int oxp = col && !ex1 ? tr + 1 : tr, oyp = col && !ey1 ? tr + TIp : tr;
  // first active step; a column that has no cells (or gave up waiting) never becomes active
  int sfirst = col ? slo : (1 << 29);
  const unsigned nact = (unsigned)(g.NK - 3);

  // Prepared values of the next step.
  bool act = false;             // the column has a cell at this step
  V dd = V(0);              // DD of the cell (0: not computed)
  V y0 = V(0);              // FWD: Y or A*P;  BWD: T
  V c1 = V(0), c2 = V(0), c3 = V(0);  // FWD: ALI*DD(i-1), ALJ*DD(j-1), ALK*DD(k-1); BWD: AUI, AUJ, AUK
  V dk1 = V(0), pk1 = V(0);  // DD and P of this column at the previous step (FWD; 0 below the interior)
  V pcol = V(0);             // P of this column at the step to prepare (FWD_AX)
  V ddn = V(0);              // DD of this column there
  V xk1 = V(0);             // result of this column at the previous step
  V q0 = V(0), q1 = V(0);   // NDOT: R0 and RR of the cell
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, a4 = 0.0;  // NDOT: this column's sums
  // Prepare step s: cs = slot of s, ps = slot of s-1, ns = slot of s+1.
  // Straight-line: every thread loads and computes whether or not it has a
  // cell at this step (all addresses lie in the ring), and `act` decides
  // what is stored.
  auto prepare = [&](int s, const V *cs, const V *ps, const V *ns) {
    act = (unsigned)(s - sfirst) <= nact;
    if (MODE == SWEEP_FWD_AX) {
      // DD, read a step ahead, says whether the warp has anything to compute
      dd = ddn;
      ddn = co(ns, SYS_DD, tr);
      if (!__any_sync(0xffffffffu, act && dd != V(0))) {
        dk1 = V(0);
        pk1 = act ? pcol : V(0);
        pcol = ns[8 * T + tr];
        return;
      }
    }
    const Coef f = coefs(cs, tr);
    auto k = [&](int c) { return f.e[c - SYS_AUI]; };
    dd = k(SYS_DD);
    if (MODE == SWEEP_FWD_AX) {
      const V pc = pcol;
      const V pn = ns[8 * T + tr];
      const V pxm = *(ex0 ? cs + hl : ps + 8 * T + ox);
      const V pym = *(ey0 ? cs + hd : ps + 8 * T + oy);
      const V pzm = pk1;
      const V pxp = *(ex1 ? cs + hr : ns + 8 * T + oxp);
      const V pyp = *(ey1 ? cs + hu : ns + 8 * T + oyp);
      const V pzp = (s < shi) ? pn : V(0);
      const V ali = k(SYS_ALI), alj = k(SYS_ALJ), alk = k(SYS_ALK);
      const V d1 = hx ? co(ps, SYS_DD, ox) : V(0);
      const V d2 = hy ? co(ps, SYS_DD, oy) : (CS == 2 && rrow && act ? din[(size_t)(s + lag) * TIp + t.ti] : V(0));
      y0 = k(SYS_AD) * pc + ali * pxm + alj * pym + alk * pzm + k(SYS_AUI) * pxp + k(SYS_AUJ) * pyp + k(SYS_AUK) * pzp;
      c1 = ali * d1;
      c2 = alj * d2;
      c3 = alk * dk1;
      dk1 = act ? dd : V(0);
      pk1 = act ? pc : V(0);
      pcol = pn;
    } else if (MODE == SWEEP_FWD) {
      const V d1 = hx ? co(ps, SYS_DD, ox) : V(0);
      const V d2 = hy ? co(ps, SYS_DD, oy) : (CS == 2 && rrow && act ? din[(size_t)(s + lag) * TIp + t.ti] : V(0));
      y0 = cs[tr];
      c1 = k(SYS_ALI) * d1;
      c2 = k(SYS_ALJ) * d2;
      c3 = k(SYS_ALK) * dk1;
      dk1 = act ? dd : V(0);
    } else {
      y0 = cs[tr];
      c1 = k(SYS_AUI);
      c2 = k(SYS_AUJ);
      c3 = k(SYS_AUK);
      if (NDOT > 0) q0 = cs[5 * T + tr];
      if (NDOT == 5) q1 = cs[6 * T + tr];
    }
  };
  bool ok = true;
  // slots of steps s, s+1 and s+2 (R >= 3), the exchange buffers of steps
  // s and s-1, and the slot of step s+1+AHEAD with its phase
  const V *ps = ring, *cs = ring + SS, *ns = ring + 2 * (size_t)SS;
  const V *const rend = ring + (size_t)R * SS;
  V *xc = xb, *xp = xb + T;
  int ru = AHEAD;
  unsigned pu = 0;
  // whether the newest data that preparing step s+1 reads has arrived;
  // tested a step ahead, so the test's latency is hidden
  bool ready = true;
  if (!producer) {
    for (int u = 0; u < AHEAD; ++u) if (ok) ok = wait_data(u, u, 0u);
    if (CS == 2 && ok && rrow && col && 0 >= slo && 0 <= shi) ok = mbar_wait_cluster(smem_u32(xfull + lag), 0u, st);
    if (!ok) { sfirst = 1 << 29; s_abort[0] = 1; }
    if (MODE == SWEEP_FWD_AX) { pcol = ring[8 * T + tr]; ddn = co(ring, SYS_DD, tr); }
    prepare(0, ring, rend - SS, ring + SS);
    ready = !ok || ru >= nsteps || mbar_test(bar0 + 8u * ru, 0u);
  }
  bool aborted = false;
  int issued = min(min(D, nsteps), stall_from) - 1;  // last step whose copies were issued (producer)
  int rs = 0, rd = D;               // slots of steps s and s+D
  unsigned ph = 0;                  // parity of the ring cycle s / R: its s_abort entry
#pragma unroll 1
  for (int s = 0; s < nsteps; ++s) {
    if (producer) {
      issue(s + D, rd);
      if (s + D < nsteps && s + D < stall_from) issued = s + D;
      if (++rd == R) rd = 0;
    } else {
      // newest data that preparing step s+1 reads: step s+AHEAD, slot ru
      if (!ready) {
        ok = mbar_wait_st(bar0 + 8u * ru, pu, st);
        if (!ok) { sfirst = 1 << 29; act = false; s_abort[ph] = 1; }
      }
      if (++ru == R) { ru = 0; pu ^= 1u; }
      // Straight-line from here to the stores: the recurrence of step s
      // (a chain of dependent operations) and the preparation of step
      // s+1 (independent of it) are scheduled into one another.
      const V xl1 = xp[ox], xl2 = xp[oy];
      const V xr = (CS == 2 && rrow && act) ? xin[(size_t)(s + lag) * TIp + t.ti] : V(0);  // partner tile's row
      const V x1 = hx ? xl1 : V(0), x2 = hy ? xl2 : xr;
      const bool a = act;
      const V d = dd, z0 = q0, z1 = q1;
      V x = y0 - c1 * x1 - c2 * x2 - c3 * xk1;
      if (BWD) x = x * d;
      if (CS == 2 && ok && rrow && col && s + 1 >= slo && s + 1 <= shi) {
        ok = mbar_wait_cluster(smem_u32(xfull + (s + 1 + lag)), 0u, st);
        if (!ok) { sfirst = 1 << 29; s_abort[ph] = 1; }
      }
      prepare(s + 1, cs, ps, ns);
      x = (a && d != V(0)) ? x : V(0);
      if (a) {
        xc[tid] = x;
        *vp = x;
      }
      xk1 = x;
      vp += vstep;
      // products of two single-precision values are exact in double;
      // outside the column's cells x is 0 and so are the other factors
      if (NDOT == 1) a0 += (double)(a ? z0 : V(0)) * (double)x;
      if (NDOT == 5) {
        const double rv = (double)(a ? z1 : V(0)), e = (double)x, z = (double)(a ? z0 : V(0));
        a0 += rv * e;
        a1 += e * e;
        a2 += rv * rv;
        a3 += z * rv;
        a4 += z * e;
      }
      if (CS == 2 && srow) {  // this step's boundary-row values to the partner tile
        const unsigned off = (unsigned)(((size_t)s * TIp + t.ti) * ES), fb = r_full + 8u * (unsigned)s;
        st_async(r_xin + off, x, fb);
        if (!BWD) st_async(r_din + off, a ? d : V(0), fb);
      }
      ready = !ok || s + 1 + AHEAD >= nsteps || mbar_test(bar0 + 8u * ru, pu);
      ps = cs; cs = ns; ns += SS;
      if (ns == rend) ns = ring;
      V *const xs = xc; xc = xp; xp = xs;
    }
    __syncthreads();
    if (++rs == R) {
      // A timed-out wait stops the sweep at the end of this ring cycle; the
      // threads that gave up skip their remaining waits and work meanwhile.
      rs = 0;
      if (s_abort[ph]) { aborted = true; break; }
      ph ^= 1u;
    }
  }
  if (s_abort[ph]) aborted = true;  // the last, partial cycle
  if (aborted && producer) {
    // Let the copies already issued land (bounded) before the block exits.
    if (lane == 0)
      for (int u = max(0, issued - R + 1); u <= issued; ++u)
        mbar_wait_slow(bar0 + 8u * (u % R), (unsigned)((u / R) & 1), 100000000ull);
    if (lane == 0) { st->timeout = 1; st->done = 1; }
  }
  if (NDOT > 0) {
    const double a[5] = {a0, a1, a2, a3, a4};
    sweep_sums<NDOT>(a, rb, q.nb, b);
  }
  if (CS == 2) cluster_barrier();  // the partner may still write into this block's shared memory
}
template <int MODE, int MAXT, typename V, int CS>
__global__ void __launch_bounds__(MAXT, 1)
    k_sweep(Geo g, SkewGeo q, SkewSysT<V> S, const V *vin, V *vout, SolveState *st, const V *vin2, double *rb, int D) {
  pdl_enter();
  sweep_body<MODE, V, CS>(g, q, S, vin, vout, st, vin2, rb, (int)blockIdx.x, (int)blockIdx.y, D);
}

// ---------------------------------------------- slab and flat kernels
// The BiCGSTAB vectors live in the skewed layout.  A kernel that forms
// sums (or needs a cell's place) maps one warp to one wavefront slab (b,w)
// of T entries and lets lane l visit t = l, l+32, ..., skipping the entries
// that are not the tile's (they hold cells of another tile).  The dot
// products (VF_MZIP) sum in that order: lane partials, warp tree per slab,
// then the 1024-thread tree over the slab partials (block_final).
// Every vector is zero wherever INDC = -1 and where an entry holds no cell
// (the sweeps write 0 for non-computed cells), so sums need no INDC, and
// the kernels without sums pass over the whole arrays (FLAT_LOOP): an update
// leaves a zero entry zero.
// What is not the tile's: k = 2 + w - ti - tj outside 2 .. NK-1.
// The loops stand in two parts, all loads of several entries, then their
// arithmetic and stores: the compiler may not move a load above the stores of
// an earlier entry by itself, and one entry's loads in flight per thread
// left the passes at half the memory's rate.
// Slab numbers fit 32 bits (a slab has at least four entries of some 130
// bytes): with 64-bit divisions the sums of small tiles took up to 8 % more
// (256x32x64 cells in blocks of 16x1: 11.1 against 10.3 ms a step).
#define SLAB_BEGIN(g, q)                                                            \
  const int lane_ = threadIdx.x & 31;                                               \
  const long long slab_ = (long long)BX_ * ROWS_PER_BLOCK + (threadIdx.x >> 5);      \
  if (slab_ < (long long)(q).nb * (q).W) {                                          \
    const int b_ = (int)((unsigned)slab_ / (unsigned)(q).W), w_ = (int)((unsigned)slab_ - (unsigned)b_ * (unsigned)(q).W); \
    const long long e0_ = ((long long)b_ * skew_stride(q) + w_) * (q).T;             \
    const unsigned nk_ = (unsigned)((g).NK - 2);
#define SLAB_END }
// the U entries t = t0, t0+32, ... of a lane: in[u] whether the tile has it
#define SLAB_ENTRIES(q, U)                                                          \
  bool in[U];                                                                       \
  _Pragma("unroll")                                                                 \
  for (int u = 0; u < U; ++u) {                                                     \
    const int t = t0 + 32 * u, tj = (int)((unsigned)t / (unsigned)(q).TIp);          \
    in[u] = t < (q).T && (unsigned)(w_ - (t - tj * (q).TIp) - tj) < nk_;             \
  }                                                                                 \
  const long long e = e0_ + t0;
#define SLAB_LOOP_BEGIN(g, q)                                                       \
  SLAB_BEGIN(g, q)                                                                  \
  _Pragma("unroll 4")                                                               \
  for (int t_ = lane_; t_ < (q).T; t_ += 32) {                                      \
    const int tj_ = (int)((unsigned)t_ / (unsigned)(q).TIp), ti_ = t_ - tj_ * (q).TIp; \
    const bool in_ = (unsigned)(w_ - ti_ - tj_) < nk_;                               \
    const long long e = e0_ + t_;
#define SLAB_LOOP_END \
  }                   \
  SLAB_END
// FLAT_BLOCK entries per block of 256 threads, `per` entries (16 bytes) at a
// time, U of them loaded together; the arrays' lengths are multiples of 4
#define FLAT_LOOP_BEGIN(q, per, U)                                                  \
  const long long n_ = skew_entries(q) / (per), i0_ = (long long)BX_ * (FLAT_BLOCK / (per)) + threadIdx.x; \
  for (int j_ = 0; j_ < FLAT_BLOCK / (per) / 256; j_ += U) {                        \
    long long e[U];                                                                 \
    bool in[U];                                                                     \
    _Pragma("unroll")                                                               \
    for (int u = 0; u < U; ++u) { e[u] = i0_ + (j_ + u) * 256; in[u] = e[u] < n_; }
#define FLAT_LOOP_END }
#define EACH(U) _Pragma("unroll") for (int u = 0; u < U; ++u) if (in[u])

// Partial of one block of a slab sum: each warp's slab sum (warp tree),
// then the block's ROWS_PER_BLOCK slabs added in slab order by thread 0,
// into rb[bx] (bx the block's index).  The finaliser then reduces one
// partial per block (nslab / 8 of them) instead of one per slab.  Every
// thread of the block calls it (it holds block barriers).
__device__ __forceinline__ void slab_store(double s, double *rb, long long nslab, unsigned bx) {
  __shared__ double ws[ROWS_PER_BLOCK];
  s = warp_tree(s);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    const long long first = (long long)bx * ROWS_PER_BLOCK;
    double t = 0.0;
    for (int i = 0; i < ROWS_PER_BLOCK; ++i)
      if (first + i < nslab) t = t + ws[i];
    rb[bx] = t;
  }
  __syncthreads();
}

__device__ __forceinline__ bool interior(const Geo &g, int I, int J, int K) {
  return I >= 2 && I <= g.NI - 1 && J >= 2 && J <= g.NJ - 1 && K >= 2 && K <= g.NK - 1;
}

// A*X at entry e, column (ti,tj) of tile b, layer k (VF_MZAX expression,
// vf_mzax.f:46-53).
template <typename V>
__device__ __forceinline__ V skew_ax(const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *X, long long e,
                                     int b, int ti, int tj, int k) {
  const long long slab = e / q.T;
  const int t = (int)(e - slab * q.T);
  const int bx = b % q.ntx, by = b / q.ntx;
  const V *s = S.sys + sys_chunk<V>(slab, 0, q.T, 0);
  auto a = [&](int c) { return s[sys_in_run<V>(c, q.T, t)]; };
  auto at = [&](int di, int dj, int dk) -> V {
    const long long n = skew_nb(g, q, bx, by, ti + di, tj + dj, k + dk);
    return n < 0 ? V(0) : X[n];
  };
  return a(SYS_AD) * X[e] + a(SYS_ALI) * at(-1, 0, 0) + a(SYS_ALJ) * at(0, -1, 0) + a(SYS_ALK) * at(0, 0, -1) +
         a(SYS_AUI) * at(1, 0, 0) + a(SYS_AUJ) * at(0, 1, 0) + a(SYS_AUK) * at(0, 0, 1);
}

// Y = A X on INDC != -1 (VF_MZAX), 0 elsewhere.
template <typename V>
__global__ void k_spmv(Geo g, SkewGeo q, SkewSysT<V> S, const V *X, V *Y, const SolveState *st) {
  pdl_enter();
  const unsigned BX_ = blockIdx.x;
  if (st && st->done) return;
  SLAB_LOOP_BEGIN(g, q)
  if (in_) Y[e] = S.indc[e] != -1 ? skew_ax(g, q, S, X, e, b_, ti_, tj_, 2 + w_ - ti_ - tj_) : V(0);
  SLAB_LOOP_END
}

// Y = B - A X on INDC != -1 (vf_m1bcgs.f:117-132), 0 elsewhere; with rb0
// also the slab partials of (B,B) and (Y,Y) over INDC != -1.
__device__ __forceinline__ void resid_body(const Geo &g, const SkewGeo &q, const SkewSys &S, const double *B,
                                           const double *X, double *Y, double *rb0, double *rb1,
                                           const SolveState *st, unsigned BX_) {
  if (st && st->done) return;
  double s0 = 0.0, s1 = 0.0;
  const long long nslab = (long long)q.nb * q.W;
  SLAB_LOOP_BEGIN(g, q)
  if (in_) {
    double y = 0.0;
    if (S.indc[e] != -1) {
      const double bv = B[e];
      y = bv - skew_ax(g, q, S, X, e, b_, ti_, tj_, 2 + w_ - ti_ - tj_);
      s0 = s0 + bv * bv;
      s1 = s1 + y * y;
    }
    Y[e] = y;
  }
  SLAB_LOOP_END
  if (rb0) {
    slab_store(s0, rb0, nslab, BX_);
    slab_store(s1, rb1, nslab, BX_);
  }
}
__global__ void k_resid(Geo g, SkewGeo q, SkewSys S, const double *B, const double *X, double *Y, double *rb0,
                        double *rb1, const SolveState *st) {
  pdl_enter();
  resid_body(g, q, S, B, X, Y, rb0, rb1, st, blockIdx.x);
}

// The BiCGSTAB vector kernels below serve the FP64 solve (V = double) and
// the FP32 inner solves of the mixed solver (V = float).  With float
// vectors the arithmetic runs in double (the scalars are double) and is
// rounded once on the store; dot products always accumulate in double.

// Slab partials of up to two dot products (VF_MZIP).
template <typename V>
__device__ __forceinline__ void dot_body(const Geo &g, const SkewGeo &q, const V *x0, const V *y0, const V *x1, const V *y1,
                      double *rb0, double *rb1, const SolveState *st, unsigned BX_) {
  if (st && st->done) return;
  double s0 = 0.0, s1 = 0.0;
  const long long nslab = (long long)q.nb * q.W;
  SLAB_BEGIN(g, q)
  for (int t0 = lane_; t0 < q.T; t0 += 128) {
    SLAB_ENTRIES(q, 4)
    V a[4], c[4], a1[4], c1[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = c[u] = a1[u] = c1[u] = V(0);
    EACH(4) { a[u] = x0[e + 32 * u]; c[u] = y0[e + 32 * u]; }
    if (x1) EACH(4) { a1[u] = x1[e + 32 * u]; c1[u] = y1[e + 32 * u]; }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s0 = s0 + (double)a[u] * (double)c[u];
      s1 = s1 + (double)a1[u] * (double)c1[u];
    }
  }
  SLAB_END
  slab_store(s0, rb0, nslab, BX_);
  if (x1) slab_store(s1, rb1, nslab, BX_);
}
template <typename V>
__global__ void k_dot(Geo g, SkewGeo q, const V *x0, const V *y0, const V *x1, const V *y1,
                      double *rb0, double *rb1, const SolveState *st) {
  pdl_enter();
  dot_body<V>(g, q, x0, y0, x1, y1, rb0, rb1, st, blockIdx.x);
}

// RR = R0, PP = R0
template <typename V>
__device__ __forceinline__ void copy2_body(const SkewGeo &q, const V *R0, V *RR, V *PP, const SolveState *st, unsigned BX_) {
  if (st->done) return;
  constexpr int G = 16 / (int)sizeof(V);
  const uint4 *r0 = reinterpret_cast<const uint4 *>(R0);
  uint4 *rr = reinterpret_cast<uint4 *>(RR), *pp = reinterpret_cast<uint4 *>(PP);
  FLAT_LOOP_BEGIN(q, G, 4)
  uint4 r[4];
  EACH(4) r[u] = r0[e[u]];
  EACH(4) { rr[e[u]] = r[u]; pp[e[u]] = r[u]; }
  FLAT_LOOP_END
}
template <typename V>
__global__ void __launch_bounds__(256) k_copy2(SkewGeo q, const V *R0, V *RR, V *PP, const SolveState *st) {
  pdl_enter();
  copy2_body<V>(q, R0, RR, PP, st, blockIdx.x);
}

// Whether a value's bits change.  The FP64 updates store only those: what is
// not computed (air, obstacles) stays 0.  Updates of a step on 1024x128x128
// cells, 16x16 blocks: 1 % water 19.9 -> 14.7 ms, the solitary beach 38.9 ->
// 31.8 ms.
__device__ __forceinline__ bool changed(double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); }

// RR = RR - ALPHA*AP (vf_m1bcgs.f:181-189)
__global__ void __launch_bounds__(256) k_axpy_rr(SkewGeo q, const double *AP, double *RR, const SolveState *st) {
  pdl_enter();
  const unsigned BX_ = blockIdx.x;
  if (st->done) return;
  const double alpha = st->alpha;
  const double2 *ap = reinterpret_cast<const double2 *>(AP);
  double2 *rr = reinterpret_cast<double2 *>(RR);
  FLAT_LOOP_BEGIN(q, 2, 4)
  double2 r[4], a[4];
  EACH(4) { r[u] = rr[e[u]]; a[u] = ap[e[u]]; }
  EACH(4) {
    const double2 n = make_double2(r[u].x - alpha * a[u].x, r[u].y - alpha * a[u].y);
    if (changed(n.x, r[u].x) || changed(n.y, r[u].y)) rr[e[u]] = n;
  }
  FLAT_LOOP_END
}

// XW = XW + (ALPHA*PP + OMEGA*RR); RR = RR - OMEGA*AE; slab partials of
// (RR,RR) and (R0,RR) on the updated RR (vf_m1bcgs.f:206-225).
__global__ void k_upd_xr(Geo g, SkewGeo q, const double *PP, const double *AE, const double *R0, double *XW, double *RR,
                         double *rb0, double *rb1, const SolveState *st) {
  pdl_enter();
  const unsigned BX_ = blockIdx.x;
  if (st->done) return;
  const double alpha = st->alpha, omega = st->omega;
  double s0 = 0.0, s1 = 0.0;
  const long long nslab = (long long)q.nb * q.W;
  SLAB_BEGIN(g, q)
  for (int t0 = lane_; t0 < q.T; t0 += 128) {
    SLAB_ENTRIES(q, 4)
    double xw[4], pp[4], rr[4], ae[4], r0[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) xw[u] = pp[u] = rr[u] = ae[u] = r0[u] = 0.0;
    EACH(4) { xw[u] = XW[e + 32 * u]; pp[u] = PP[e + 32 * u]; rr[u] = RR[e + 32 * u]; ae[u] = AE[e + 32 * u]; r0[u] = R0[e + 32 * u]; }
    EACH(4) {
      const double x = xw[u] + (alpha * pp[u] + omega * rr[u]);
      if (changed(x, xw[u])) XW[e + 32 * u] = x;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double r = in[u] ? rr[u] - omega * ae[u] : 0.0;
      if (in[u] && changed(r, rr[u])) RR[e + 32 * u] = r;
      s0 = s0 + r * r;
      s1 = s1 + r0[u] * r;
    }
  }
  SLAB_END
  slab_store(s0, rb0, nslab, BX_);
  slab_store(s1, rb1, nslab, BX_);
}

// PP = RR + BETA*(PP - OMEGA*AP) (vf_m1bcgs.f:229-238)
__global__ void __launch_bounds__(256) k_upd_p(SkewGeo q, const double *RR, const double *AP, double *PP,
                                               const SolveState *st) {
  pdl_enter();
  const unsigned BX_ = blockIdx.x;
  if (st->done) return;
  const double beta = st->beta, omega = st->omega;
  const double2 *rr = reinterpret_cast<const double2 *>(RR), *ap = reinterpret_cast<const double2 *>(AP);
  double2 *pp = reinterpret_cast<double2 *>(PP);
  FLAT_LOOP_BEGIN(q, 2, 4)
  double2 r[4], a[4], p[4];
  EACH(4) { r[u] = rr[e[u]]; a[u] = ap[e[u]]; p[u] = pp[e[u]]; }
  EACH(4) {
    const double2 n = make_double2(r[u].x + beta * (p[u].x - omega * a[u].x), r[u].y + beta * (p[u].y - omega * a[u].y));
    if (changed(n.x, p[u].x) || changed(n.y, p[u].y)) pp[e[u]] = n;
  }
  FLAT_LOOP_END
}

// --------------------------------- FP32 inner solves of the mixed solver
// The inner BiCGSTAB of the mixed solver (V = float) runs a regrouped
// iteration with fewer passes over the vectors; it is the same method and
// ends on the same criterion, but its sums are not those of VF_M1BCGS,
// whose FP64 form (above) keeps the reference's order.
//   * After the second sweep pair one pass forms the five sums (RR,AE),
//     (AE,AE), (RR,RR), (R0,RR), (R0,AE); OMEGA, the new |RR|^2 =
//     (RR,RR) - 2 OMEGA (RR,AE) + OMEGA^2 (AE,AE), the new (R0,RR) =
//     (R0,RR) - OMEGA (R0,AE), the convergence test and BETA follow from
//     them (k_fin5), and one pass updates XW, RR and PP together (k_upd3f).
//     Per iteration a sum drops by about 25 times, so the expansion loses
//     nothing to cancellation at the tolerances used (FP64 sums).
// Four consecutive entries per lane of a slab, as 16-byte loads; keep4
// clears those that are not the tile's.
#define SLAB4_LOOP_BEGIN(g, q)                                                      \
  const int lane_ = threadIdx.x & 31;                                               \
  const long long slab_ = (long long)BX_ * ROWS_PER_BLOCK + (threadIdx.x >> 5);      \
  if (slab_ < (long long)(q).nb * (q).W) {                                          \
    const int b_ = (int)((unsigned)slab_ / (unsigned)(q).W), w_ = (int)((unsigned)slab_ - (unsigned)b_ * (unsigned)(q).W); \
    const int T4_ = (q).T >> 2;                                                     \
    const unsigned nk_ = (unsigned)((g).NK - 2);                                     \
    _Pragma("unroll 2")                                                             \
    for (int t_ = lane_; t_ < T4_; t_ += 32) {                                      \
      const int tj_ = (int)(4u * (unsigned)t_ / (unsigned)(q).TIp), s_ = w_ - (4 * t_ - tj_ * (q).TIp) - tj_;     \
      const long long e4 = ((long long)b_ * skew_stride(q) + w_) * T4_ + t_;
#define SLAB4_LOOP_END \
    }                  \
  }
__device__ __forceinline__ float4 keep4(const float4 &a, int s, unsigned nk) {
  return make_float4((unsigned)s < nk ? a.x : 0.0f, (unsigned)(s - 1) < nk ? a.y : 0.0f,
                     (unsigned)(s - 2) < nk ? a.z : 0.0f, (unsigned)(s - 3) < nk ? a.w : 0.0f);
}
__device__ __forceinline__ double dot4(const float4 &a, const float4 &b) {
  return (double)a.x * (double)b.x + (double)a.y * (double)b.y + (double)a.z * (double)b.z +
         (double)a.w * (double)b.w;
}
// slab partials of (R0,AP)
__global__ void k_dot2f(Geo g, SkewGeo q, const float *R0, const float *AP, double *rb, const SolveState *st) {
  pdl_enter();
  const unsigned BX_ = blockIdx.x;
  if (st->done) return;
  const float4 *r0 = reinterpret_cast<const float4 *>(R0), *ap = reinterpret_cast<const float4 *>(AP);
  double s0 = 0.0;
  const long long nslab = (long long)q.nb * q.W;
  SLAB4_LOOP_BEGIN(g, q)
  s0 += dot4(keep4(r0[e4], s_, nk_), keep4(ap[e4], s_, nk_));
  SLAB4_LOOP_END
  slab_store(s0, rb, nslab, BX_);
}
// RR = RR - ALPHA*AP
__device__ __forceinline__ void axpyf_body(const SkewGeo &q, const float *AP, float *RR, const SolveState *st, unsigned BX_) {
  if (st->done) return;
  const double alpha = st->alpha;
  const float4 *ap = reinterpret_cast<const float4 *>(AP);
  float4 *rr = reinterpret_cast<float4 *>(RR);
  FLAT_LOOP_BEGIN(q, 4, 4)
  float4 r[4], a[4];
  EACH(4) { r[u] = rr[e[u]]; a[u] = ap[e[u]]; }
  EACH(4) {
    r[u].x = (float)(r[u].x - alpha * a[u].x); r[u].y = (float)(r[u].y - alpha * a[u].y);
    r[u].z = (float)(r[u].z - alpha * a[u].z); r[u].w = (float)(r[u].w - alpha * a[u].w);
    rr[e[u]] = r[u];
  }
  FLAT_LOOP_END
}
__global__ void __launch_bounds__(256) k_axpyf(SkewGeo q, const float *AP, float *RR, const SolveState *st) {
  pdl_enter();
  axpyf_body(q, AP, RR, st, blockIdx.x);
}
// block partials of (RR,AE), (AE,AE), (RR,RR), (R0,RR), (R0,AE) into
// rb + c*nrb, c = 0..4 (nrb = blocks of the launch)
__global__ void k_dot5f(Geo g, SkewGeo q, const float *R0, const float *RR, const float *AE, double *rb,
                        const SolveState *st) {
  pdl_enter();
  const unsigned BX_ = blockIdx.x;
  if (st->done) return;
  const float4 *r0 = reinterpret_cast<const float4 *>(R0), *rr = reinterpret_cast<const float4 *>(RR),
               *ae = reinterpret_cast<const float4 *>(AE);
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0, s4 = 0.0;
  const long long nslab = (long long)q.nb * q.W;
  SLAB4_LOOP_BEGIN(g, q)
  const float4 a = keep4(r0[e4], s_, nk_), r = keep4(rr[e4], s_, nk_), e = keep4(ae[e4], s_, nk_);
  s0 += dot4(r, e);
  s1 += dot4(e, e);
  s2 += dot4(r, r);
  s3 += dot4(a, r);
  s4 += dot4(a, e);
  SLAB4_LOOP_END
  const long long nrb = gridDim.x;  // block partials of each sum
  slab_store(s0, rb, nslab, BX_);
  slab_store(s1, rb + nrb, nslab, BX_);
  slab_store(s2, rb + 2 * nrb, nslab, BX_);
  slab_store(s3, rb + 3 * nrb, nslab, BX_);
  slab_store(s4, rb + 4 * nrb, nslab, BX_);
}
// XW = XW + (ALPHA*PP + OMEGA*RR); RR' = RR - OMEGA*AE;
// PP = RR' + BETA*(PP - OMEGA*AP); RR = RR'
__device__ __forceinline__ void upd3f_body(const SkewGeo &q, const float *AE, const float *AP, float *XW, float *RR, float *PP,
                        const SolveState *st, unsigned BX_) {
  if (st->done) return;
  const double alpha = st->alpha, omega = st->omega, beta = st->beta;
  const float4 *ae = reinterpret_cast<const float4 *>(AE), *ap = reinterpret_cast<const float4 *>(AP);
  float4 *xw = reinterpret_cast<float4 *>(XW), *rr = reinterpret_cast<float4 *>(RR),
         *pp = reinterpret_cast<float4 *>(PP);
  FLAT_LOOP_BEGIN(q, 4, 2)
  float4 d[2], a[2], r[2], p[2], x[2];
  EACH(2) { d[u] = ae[e[u]]; a[u] = ap[e[u]]; r[u] = rr[e[u]]; p[u] = pp[e[u]]; x[u] = xw[e[u]]; }
  EACH(2) {
    float4 rn, pn;
#define UPD3_(c)                                                              \
    x[u].c = (float)(x[u].c + (alpha * p[u].c + omega * r[u].c));             \
    rn.c = (float)(r[u].c - omega * d[u].c);                                  \
    pn.c = (float)(rn.c + beta * (p[u].c - omega * a[u].c));
    UPD3_(x) UPD3_(y) UPD3_(z) UPD3_(w)
#undef UPD3_
    xw[e[u]] = x[u];
    rr[e[u]] = rn;
    pp[e[u]] = pn;
  }
  FLAT_LOOP_END
}
__global__ void __launch_bounds__(256) k_upd3f(SkewGeo q, const float *AE, const float *AP, float *XW, float *RR,
                                               float *PP, const SolveState *st) {
  pdl_enter();
  upd3f_body(q, AE, AP, XW, RR, PP, st, blockIdx.x);
}
// OMEGA, the new |RR|^2 and (R0,RR), convergence and BETA from the five
// sums (vf_m1bcgs.f:196-241 regrouped).  A finished solve sets `stop`;
// k_commit turns it into `done` once the last update has run.
__device__ __forceinline__ void fin5_body(const double *rb, long long nrows, SolveState *st, double epsa2,
                                          double epsr2, double div2, int icgmax) {
  if (st->done) return;
  const double *const b[5] = {rb, rb + nrows, rb + 2 * nrows, rb + 3 * nrows, rb + 4 * nrows};
  double t[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  block_final_n<5>(b, nrows, t);
  if (threadIdx.x != 0) return;
  const double rae = t[0], aeae = t[1], rrrr = t[2], r0rr = t[3], r0ae = t[4];
  const double omega = rae / aeae;
  st->omega = omega;
  st->w1 = rae;
  st->w2 = aeae;
  const double xn = rrrr - 2.0 * omega * rae + omega * omega * aeae;
  st->xnorm = xn;
  if (xn <= st->bnorm * epsr2 + epsa2) { st->stop = 1; st->beta = 0.0; return; }
  if (xn > div2) { st->iter = -2; st->stop = 1; st->beta = 0.0; return; }
  const double W1 = r0rr - omega * r0ae;
  st->beta = W1 * st->alpha / (st->S * omega);
  st->S = W1;
  st->iter = st->iter + 1;
  if (st->iter > icgmax) st->stop = 1;
}
__global__ void k_fin5(const double *rb, long long nrows, SolveState *st, double epsa2, double epsr2, double div2,
                       int icgmax) {
  pdl_enter();
  fin5_body(rb, nrows, st, epsa2, epsr2, div2, icgmax);
}
__global__ void k_commit(SolveState *st) {
  pdl_enter();
  if (st->stop) st->done = 1;
}

// ------------------------------------------- mixed-precision conversions
// FP32 copy of the 7 coefficients (DD comes from the FP32 factorisation,
// T from the FP32 forward sweeps).
__device__ __forceinline__ void sys_to_f_elem(const SkewGeo &q, const double *sys, float *sysf, long long e) {
  const long long slab = e / q.T;
  const int t = (int)(e - slab * q.T);
  float v[8];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const double2 d = *reinterpret_cast<const double2 *>(sys + sys_chunk<double>(slab, c, q.T, t));
    v[2 * c] = (float)d.x;
    v[2 * c + 1] = (float)d.y;
  }
  v[SYS_DD - SYS_AUI] = 0.0f;  // filled by the FP32 factorisation
#pragma unroll
  for (int c = 0; c < 2; ++c)
    *reinterpret_cast<float4 *>(sysf + sys_chunk<float>(slab, c, q.T, t)) =
        make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
}
__global__ void k_sys_to_f(SkewGeo q, const double *sys, float *sysf) {
  pdl_enter();
  const long long n = skew_entries(q);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    sys_to_f_elem(q, sys, sysf, e);
}
// RF = R * scale (the right-hand side of an inner solve)
__device__ __forceinline__ void scale_to_f_body(const SkewGeo &q, const double *R, double scale, float *RF, unsigned BX_) {
  const double2 *r2 = reinterpret_cast<const double2 *>(R);
  float4 *rf = reinterpret_cast<float4 *>(RF);
  FLAT_LOOP_BEGIN(q, 4, 4)
  double2 a[4], b[4];
  EACH(4) { a[u] = r2[2 * e[u]]; b[u] = r2[2 * e[u] + 1]; }
  EACH(4) rf[e[u]] = make_float4((float)(a[u].x * scale), (float)(a[u].y * scale), (float)(b[u].x * scale), (float)(b[u].y * scale));
  FLAT_LOOP_END
}
__global__ void __launch_bounds__(256) k_scale_to_f(SkewGeo q, const double *R, double scale, float *RF) {
  pdl_enter();
  scale_to_f_body(q, R, scale, RF, blockIdx.x);
}
// X = X + D * inv_scale (the correction of an inner solve)
__device__ __forceinline__ void add_f_body(const SkewGeo &q, const float *D, double inv_scale, double *X, unsigned BX_) {
  const float4 *d4 = reinterpret_cast<const float4 *>(D);
  double2 *x2 = reinterpret_cast<double2 *>(X);
  FLAT_LOOP_BEGIN(q, 4, 2)
  float4 d[2];
  double2 a[2], b[2];
  EACH(2) { d[u] = d4[e[u]]; a[u] = x2[2 * e[u]]; b[u] = x2[2 * e[u] + 1]; }
  EACH(2) {
    a[u].x = a[u].x + (double)d[u].x * inv_scale; a[u].y = a[u].y + (double)d[u].y * inv_scale;
    b[u].x = b[u].x + (double)d[u].z * inv_scale; b[u].y = b[u].y + (double)d[u].w * inv_scale;
    x2[2 * e[u]] = a[u];
    x2[2 * e[u] + 1] = b[u];
  }
  FLAT_LOOP_END
}
__global__ void __launch_bounds__(256) k_add_f(SkewGeo q, const float *D, double inv_scale, double *X) {
  pdl_enter();
  add_f_body(q, D, inv_scale, X, blockIdx.x);
}

// X0 = XW on INDC != -1 when ITER >= 0 (vf_m1bcgs.f:251-261), back to the
// standard layout.
__device__ __forceinline__ void x0_body(Geo g, SkewGeo q, const int *INDC, const double *XW, double *X0, const SolveState *st, unsigned BX_) {
  if (st->iter < 0) return;
  SLAB_LOOP_BEGIN(g, q)
  if (in_ && INDC[e] != -1) {
    const int I = 2 + (b_ % q.ntx) * q.TI + ti_, J = 2 + (b_ / q.ntx) * q.TJ + tj_;
    X0[cid(g, I, J, 2 + w_ - ti_ - tj_)] = XW[e];
  }
  SLAB_LOOP_END
}
__global__ void k_x0(Geo g, SkewGeo q, const int *INDC, const double *XW, double *X0, const SolveState *st) {
  pdl_enter();
  x0_body(g, q, INDC, XW, X0, st, blockIdx.x);
}

// ||b-Ax||^2 and ||b||^2 slab partials (diagnostic of the metric)
__global__ void k_relres(Geo g, SkewGeo q, SkewSys S, const double *B, const double *X, double *rb0,
                         double *rb1) {
  pdl_enter();
  const unsigned BX_ = blockIdx.x;
  double s0 = 0.0, s1 = 0.0;
  const long long nslab = (long long)q.nb * q.W;
  SLAB_LOOP_BEGIN(g, q)
  if (in_ && S.indc[e] != -1) {
    double r = B[e] - skew_ax(g, q, S, X, e, b_, ti_, tj_, 2 + w_ - ti_ - tj_);
    s0 = s0 + r * r;
    s1 = s1 + B[e] * B[e];
  }
  SLAB_LOOP_END
  slab_store(s0, rb0, nslab, BX_);
  slab_store(s1, rb1, nslab, BX_);
}

// ------------------------------------------------------------- finalisers
// One block of 1024 threads: reduce the row partials and advance the
// BiCGSTAB scalars exactly as the host code of vf_m1bcgs.f would.
__device__ __forceinline__ void fin_body(int mode, const double *rb0, const double *rb1, long long nrows,
                                         SolveState *st, double *out, double epsa2, double epsr2, double div2,
                                         int icgmax) {
  if (mode < FIN_ALPHA && mode != FIN_STORE && mode != FIN_RELRES && st->done) return;
  if (mode >= FIN_ALPHA && st->done) return;
  double a, b = 0.0;
  if (rb1) {
    const double *const bufs[2] = {rb0, rb1};
    double t[2] = {0.0, 0.0};
    block_final_n<2>(bufs, nrows, t);
    a = t[0];
    b = t[1];
  } else {
    a = block_final(rb0, nrows);
  }
  if (threadIdx.x != 0) return;
  switch (mode) {
    case FIN_BNORM:
      st->bnorm = a;
      break;
    case FIN_START:  // S=(R0,R0), first convergence test (vf_m1bcgs.f:140-144)
      st->S = a;
      st->xnorm = a;
      st->iter = 0;
      if (st->xnorm <= st->bnorm * epsr2 + epsa2) { st->done = 1; st->status = 0; }
      else {
        st->iter = 1;
        if (st->iter > icgmax) { st->done = 1; }
      }
      break;
    case FIN_ALPHA:
      st->w1 = a;
      st->alpha = st->S / a;
      break;
    case FIN_OMEGA:
      st->w1 = a;
      st->w2 = b;
      st->omega = a / b;
      break;
    case FIN_CONV: {  // vf_m1bcgs.f:218-241
      st->xnorm = a;
      if (st->xnorm <= st->bnorm * epsr2 + epsa2) { st->done = 1; break; }
      if (st->xnorm > div2) { st->iter = -2; st->done = 1; break; }
      double W1 = b;
      st->beta = W1 * st->alpha / (st->S * st->omega);
      st->S = W1;
      st->iter = st->iter + 1;
      if (st->iter > icgmax) st->done = 1;
    } break;
    case FIN_RELRES:
      st->rn = a;
      st->bn = b;
      break;
    case FIN_STORE:
      out[0] = a;
      out[1] = b;
      break;
    default:
      break;
  }
}
__global__ void k_fin(int mode, const double *rb0, const double *rb1, long long nrows,
                      SolveState *st, double *out, double epsa2, double epsr2, double div2,
                      int icgmax) {
  pdl_enter();
  fin_body(mode, rb0, rb1, nrows, st, out, epsa2, epsr2, div2, icgmax);
}

// Factorisation failure ends the solve with ITER = -1 (vf_m1bcgs.f:101-102).
__global__ void k_pivot_check(SolveState *st) {
  pdl_enter();
  if (st->pivot_bad) { st->iter = -1; st->done = 1; }
}

// ------------------------------------------------------------- VF_VMODIF
// 453 us on 1026x130x130 cells with a row per warp, 274 us with a cell per
// thread and its flags, then its values loaded together.
__global__ void __launch_bounds__(CELL_THREADS) k_vmodif(Geo g, Fld f, Prm p, const double *PT) {
  const double *GGV = f.ggv, *GLV = f.glv;
  const int *NF = f.nf;
  const double RT = p.rho0 / p.dtnow;
  CELL_LOOP_BEGIN(g)
  const long long c = cid(g, I, J, K);
  const int NI = g.NI, NJ = g.NJ, NK = g.NK;
  if (I < 2 || J < 2 || K < 2) continue;
  // the flags, then the values, each in flight together
  const long long sj = NI, sk = (long long)NI * NJ;
  const int n0 = ld_now(NF + c), nx = ld_now(NF + c - 1), ny = ld_now(NF + c - sj), nz = ld_now(NF + c - sk);
  const int ix = ld_now(f.indx + c), iy = ld_now(f.indy + c), iz = ld_now(f.indz + c), in = ld_now(f.indc + c);
  const bool pres = interior(g, I, J, K) && in != -1;
  const bool dox = K <= NK - 1 && J <= NJ - 1 && nx * n0 == 0, doy = K <= NK - 1 && I <= NI - 1 && ny * n0 == 0,
             doz = J <= NJ - 1 && I <= NI - 1 && nz * n0 == 0;
  if (!dox && !doy && !doz && !pres) continue;
  const double gv0 = ld_now(GGV + c), gvx = ld_now(GGV + c - 1), gvy = ld_now(GGV + c - sj), gvz = ld_now(GGV + c - sk);
  const double lv0 = ld_now(GLV + c), lvx = ld_now(GLV + c - 1), lvy = ld_now(GLV + c - sj), lvz = ld_now(GLV + c - sk);
  const double p0 = ld_now(PT + c), px = ld_now(PT + c - 1), py = ld_now(PT + c - sj), pz = ld_now(PT + c - sk);
  const double u0 = ld_now(f.uu + c), v0 = ld_now(f.vv + c), w0 = ld_now(f.ww + c), pp0 = ld_now(f.pp + c);
  if (dox) {
    const int IS = ix;
    if (IS == 0) {
      double GV = XX_(6, I) * (XX_(2, I) * gv0 / lv0 + XX_(2, I - 1) * gvx / lvx);
      f.uu[c] = u0 + XX_(5, I) * GV * (p0 - px);
    } else if (IS > 0 && (indb(f, 3, IS) == 4 || (indb(f, 3, IS) == 5 && fixlvl_face(g, p, indb(f, 2, IS), I, J)))) {
      if (indb(f, 2, IS) == 1) f.uu[c] = u0 + 2.0 * XX_(4, I) * gv0 / lv0 * p0;
      else f.uu[c] = u0 - 2.0 * XX_(4, I - 1) * gvx / lvx * px;
      f.bcu[IS - 1] = f.uu[c];
    }
  }
  if (doy) {
    const int IS = iy;
    if (IS == 0) {
      double GV = YY_(6, J) * (YY_(2, J) * gv0 / lv0 + YY_(2, J - 1) * gvy / lvy);
      f.vv[c] = v0 + YY_(5, J) * GV * (p0 - py);
    } else if (IS > 0 && (indb(f, 3, IS) == 4 || (indb(f, 3, IS) == 5 && fixlvl_face(g, p, indb(f, 2, IS), I, J)))) {
      if (indb(f, 2, IS) == 3) f.vv[c] = v0 + 2.0 * YY_(4, J) * gv0 / lv0 * p0;
      else f.vv[c] = v0 - 2.0 * YY_(4, J - 1) * gvy / lvy * py;
      f.bcv[IS - 1] = f.vv[c];
    }
  }
  if (doz) {
    const int IS = iz;
    if (IS == 0) {
      double GV = ZZ_(6, K) * (ZZ_(2, K) * gv0 / lv0 + ZZ_(2, K - 1) * gvz / lvz);
      f.ww[c] = w0 + ZZ_(5, K) * GV * (p0 - pz);
    } else if (IS > 0 && indb(f, 3, IS) == 4) {
      if (indb(f, 2, IS) == 5) f.ww[c] = w0 + 2.0 * ZZ_(4, K) * gv0 / lv0 * p0;
      else f.ww[c] = w0 - 2.0 * ZZ_(4, K - 1) * gvz / lvz * pz;
      f.bcw[IS - 1] = f.ww[c];
    }
  }
  if (pres) f.pp[c] = pp0 - RT * p0;
  CELL_LOOP_END
}

#undef A
#undef XX_
#undef YY_
#undef ZZ_

// ------------------------------------------------------------- launchers
void launch_vpcoef(cudaStream_t s, const Geo &g, const Fld &f, const Prm &p, const SysPtr &a, int *err) {
  k_vpcoef<<<cell_grid(g), CELL_THREADS, 0, s>>>(g, f, p, a, err);
  count_launch();
}
// Prefetch depth: the largest of 8, 4, 2, 1 whose ring fits the shared
// memory a block may use (200 KB here).
static int ring_depth(int NV, int T, size_t es) {
  const size_t cap = 200 * 1024;
  for (int d : {8, 4, 2, 1})
    if (ring_bytes(NV, T, d + 3, es) <= cap) return d;
  return 0;
}
// Launch a kernel that starts with pdl_enter() with programmatic stream
// serialisation (cluster dimensions optional).
template <typename... KArgs, typename... Args>
static void launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, int cluster_y,
                       Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  int na = 1;
  if (cluster_y > 1) {
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = (unsigned)cluster_y; at[1].val.clusterDim.z = 1;
    na = 2;
  }
  cfg.attrs = at; cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, kern, ((KArgs)args)...);
  count_launch();
}
// The kernel's dynamic shared-memory limit, raised to the bytes of this
// launch and never lowered: handles stepped from several host threads at
// once (cadmas_step_ensemble) with different tile shapes then never lower
// it under one another's launches.
template <class K> static void set_smem(K kern, size_t bytes) {
  raise_dynamic_smem((const void *)kern, bytes);
}

void launch_to_skew(cudaStream_t s, const Geo &g, const SkewGeo &q, const SysPtr &a, const int *indc,
                    const SkewSys &S, const double *x0, double *bsl, double *xsl, int warm) {
  const size_t rb = to_skew_rows_bytes(g, q);
  if (rb > 0) {
    raise_dynamic_smem((const void *)k_to_skew_rows, rb);
    launch_pdl(k_to_skew_rows, dim3((unsigned)(q.nb * q.TJ)), dim3(256), rb, s, 1, g, q, a, indc, S, x0, bsl, xsl,
               warm);
    return;
  }
  const long long n = (long long)q.nb * q.W * q.T;
  const int blocks = (int)std::min<long long>((n + 255) / 256, 148LL * 16);
  launch_pdl(k_to_skew, dim3(blocks), dim3(256), 0, s, 1, g, q, a, indc, S, x0, bsl, xsl, warm);
}
template <typename V>
static void launch_dcmp_t(cudaStream_t s, const Geo &g, const SkewGeo &q, V U, const SkewSysT<V> &S, int *pivot_bad) {
  const int T = q.T * q.split, d = ring_depth(7, T, sizeof(V));  // one thread per block column
  const size_t bytes = ring_bytes(7, T, d + 3, sizeof(V));
  const int TJb = q.TJ * q.split, nby = (g.NJ - 2 + TJb - 1) / TJb;
  const dim3 grid((unsigned)q.ntx, (unsigned)nby);
  switch (d) {
#define DCMP_CASE(DD)                                                                    \
  case DD:                                                                               \
    set_smem(k_dcmp<DD, V>, bytes);                                                      \
    launch_pdl(k_dcmp<DD, V>, grid, dim3(T), bytes, s, 1, g, q, U, S, pivot_bad);              \
    break;
    DCMP_CASE(8) DCMP_CASE(4) DCMP_CASE(2)
    default: DCMP_CASE(1)
#undef DCMP_CASE
  }
}
void launch_dcmp(cudaStream_t s, const Geo &g, const SkewGeo &q, double U, const SkewSys &S, int *pivot_bad) {
  launch_dcmp_t<double>(s, g, q, U, S, pivot_bad);
}
void launch_dcmp_f(cudaStream_t s, const Geo &g, const SkewGeo &q, double U, const SkewSysF &S, int *pivot_bad) {
  launch_dcmp_t<float>(s, g, q, (float)U, S, pivot_bad);
}
// Bulk-copy ring: prefetch depth D in {8, 6, 4, 3, 2, 1}, the largest whose ring
// (R = D+2 slots, mbarriers, exchange buffers) fits the 227 KB of shared
// memory a block may use.
static size_t sweep_bytes(const SkewGeo &q, int mode, int D, int es) {
  const int R = D + 2;
  size_t b = (size_t)((R + 1) & ~1) * 8 + (size_t)R * sweep_slot(q, mode, es) * es + 2 * (size_t)q.T * es;
  if (q.split == 2)  // cluster exchange: xfull[W] barriers, xin (and din) [W][TIp]
    b += (size_t)q.W * 8 + (size_t)q.W * q.TIp * es * (mode >= SWEEP_BWD ? 1 : 2);
  return b;
}
static int sweep_depth(const SkewGeo &q, int mode, int es) {
  if (sweep_threads(q.T) > (q.split == 2 ? 512 : 1024)) return 0;
  // (depth 1 would starve the fused sweep, which reads two steps ahead)
  for (int d : {8, 6, 4, 3, 2, 1})
    if (sweep_bytes(q, mode, d, es) <= 227 * 1024 && (d > 1 || mode != SWEEP_FWD_AX)) return d;
  return 0;
}
// ---- dispatch.  The sweeps run in the thread-copy form (k_sweep_cp); the
// bulk-copy ring (k_sweep) serves clusters (split 2), tiles too large for the
// other and handles with the stall injection on (SkewGeo::ring), whose
// subject is the ring's waits.
static int sweep_form_depth(const SkewGeo &q, int mode, int es) {  // 0: the ring
  return q.ring ? 0 : sweep_cp_depth(q, mode, es);
}
template <int D, int MODE, int MAXT, typename V, int MINB, bool ONE = false>
static void sweep_cp_go(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *vin, V *vout,
                        SolveState *st, const V *vin2, double *rb) {
  const size_t bytes = sweep_cp_bytes(MODE, D, sweep_cp_unrolled(q, MODE, (int)sizeof(V)), q.T, q.TIp, q.TI, q.TJ, (int)sizeof(V));
  const dim3 grid((unsigned)q.ntx, (unsigned)(q.nb / q.ntx)), block((unsigned)sweep_cp_threads(q.T));
#define SWEEP_GO(CT, CI)                                                                                        \
  {                                                                                                             \
    set_smem(k_sweep_cp<D, MODE, MAXT, V, MINB, CT, CI, ONE>, bytes);                                           \
    launch_pdl(k_sweep_cp<D, MODE, MAXT, V, MINB, CT, CI, ONE>, grid, block, bytes, s, 1, g, q, S, vin, vout, st, vin2, rb); \
    return;                                                                                                     \
  }
  if constexpr (MAXT == 128) {
    if (q.T == 128 && q.TIp == 8) SWEEP_GO(128, 8)
    if (q.T == 128 && q.TIp == 16) SWEEP_GO(128, 16)
  }
  if constexpr (MAXT == 256) {
    if (q.T == 256 && q.TIp == 16) SWEEP_GO(256, 16)
  }
  SWEEP_GO(0, 0)
#undef SWEEP_GO
}
template <int MODE, typename V, int MAXT, int CS>
static void sweep_ring_go(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *vin, V *vout,
                          SolveState *st, const V *vin2, double *rb) {
  const int d = sweep_depth(q, MODE, (int)sizeof(V));
  if (d == 0) return;  // rejected by cadmas_create (sweep_supported)
  const size_t bytes = sweep_bytes(q, MODE, d, (int)sizeof(V));
  const int nty = q.nb / q.ntx;
  const dim3 grid((unsigned)q.ntx, (unsigned)(CS == 2 ? (nty + 1) & ~1 : nty)), block((unsigned)sweep_threads(q.T));
  set_smem(k_sweep<MODE, MAXT, V, CS>, bytes);
  launch_pdl(k_sweep<MODE, MAXT, V, CS>, grid, block, bytes, s, CS, g, q, S, vin, vout, st, vin2, rb, d);
}
// The sweep MODE of a grid.  vin2 and rb: the inner products' second
// vector and partials (modes 3, 4).
template <int MODE, typename V>
static void launch_sweep(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *vin,
                         V *vout, SolveState *st, const V *vin2 = nullptr, double *rb = nullptr) {
  const int d = sweep_form_depth(q, MODE, (int)sizeof(V)), nt = sweep_cp_threads(q.T);
#define CP_GO(D, MT, MB)                                                       \
  {                                                                            \
    sweep_cp_go<D, MODE, MT, V, MB>(s, g, q, S, vin, vout, st, vin2, rb);      \
    return;                                                                    \
  }
  // two blocks' registers for FP32, whose rings leave room for two blocks
  constexpr int MB = sizeof(V) == 4 ? 2 : 1;
  if constexpr (MODE == SWEEP_FWD_AX) {
#define CP_ONE(D, MT)                                                          \
  {                                                                            \
    sweep_cp_go<D, MODE, MT, V, 1, true>(s, g, q, S, vin, vout, st, vin2, rb); \
    return;                                                                    \
  }
    if (d > 0 && q.one) {
      if (d == 8) CP_ONE(8, 576)
      if (d == 4) CP_ONE(4, 576)
      CP_ONE(2, 576)
    }
#undef CP_ONE
    if (d > 0) {
      if (nt <= 128) {
        if (d == 12) CP_GO(12, 128, 1)
        if (d == 8) CP_GO(8, 128, 1)
        if (d == 6) CP_GO(6, 128, 1)
        if (d == 4) CP_GO(4, 128, 1)
        CP_GO(2, 128, 1)
      } else if (nt <= 256) {
        if (d == 8) CP_GO(8, 256, MB)
        if (d == 6) CP_GO(6, 256, MB)
        if (d == 4) CP_GO(4, 256, MB)
        CP_GO(2, 256, MB)
      } else if (nt <= 576) {
        if (d == 8) CP_GO(8, 576, 1)
        if (d == 6) CP_GO(6, 576, 1)
        if (d == 4) CP_GO(4, 576, 1)
        CP_GO(2, 576, 1)
      } else if constexpr (sizeof(V) == 4) {  // (FP64: never, sweep_cp_depth)
        if (d == 8) CP_GO(8, 1024, 1)
        if (d == 6) CP_GO(6, 1024, 1)
        if (d == 4) CP_GO(4, 1024, 1)
        if (d == 2) CP_GO(2, 1024, 1)
        CP_GO(1, 1024, 1)
      }
    }
  } else if (d > 0) {
    if (nt <= 128) {
      if (d == 15) CP_GO(15, 128, 1)
      if (d == 9) CP_GO(9, 128, 1)
      CP_GO(3, 128, 1)
    } else if (nt <= 256) {
      if (d == 9) CP_GO(9, 256, 2)
      CP_GO(3, 256, 2)
    } else if (nt <= 576) {
      if (d == 9) CP_GO(9, 576, 1)
      CP_GO(3, 576, 1)
    } else {
      if (d == 9) CP_GO(9, 1024, 1)
      if (d == 3) CP_GO(3, 1024, 1)
      CP_GO(1, 1024, 1)
    }
  }
#undef CP_GO
  if (q.split == 2) sweep_ring_go<MODE, V, 512, 2>(s, g, q, S, vin, vout, st, vin2, rb);
  else if (sweep_threads(q.T) <= 512) sweep_ring_go<MODE, V, 512, 1>(s, g, q, S, vin, vout, st, vin2, rb);
  else sweep_ring_go<MODE, V, 1024, 1>(s, g, q, S, vin, vout, st, vin2, rb);
}
bool sweep_supported(const SkewGeo &q) {
  const int tb = q.T * q.split;  // threads of the factorisation kernel
  return sweep_depth(q, SWEEP_FWD, 8) > 0 && sweep_depth(q, SWEEP_BWD, 8) > 0 &&
         (q.split == 1 || sweep_depth(q, SWEEP_FWD_AX, 8) > 0) && tb <= 1024 && ring_depth(7, tb, 8) > 0;
}
bool sweep_supported_f(const SkewGeo &q) {
  const int tb = q.T * q.split;
  return sweep_depth(q, SWEEP_FWD, 4) > 0 && sweep_depth(q, SWEEP_BWD, 4) > 0 &&
         (q.split == 1 || sweep_depth(q, SWEEP_FWD_AX, 4) > 0) && tb <= 1024 && ring_depth(7, tb, 4) > 0;
}
template <typename V>
static void launch_fwd_t(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *y,
                         const V *spmv_x, SolveState *st, V *ybuf) {
  const int es = (int)sizeof(V);
  const bool ring = q.ring || q.split == 2;
  if (spmv_x && (ring ? sweep_depth(q, SWEEP_FWD_AX, es) : sweep_cp_depth(q, SWEEP_FWD_AX, es)) == 0) {
    // No fused sweep for this tile: SpMV first.
    launch_spmv_t<V>(s, g, q, S, spmv_x, ybuf, st);
    y = ybuf;
    spmv_x = nullptr;
  }
  if (spmv_x) launch_sweep<SWEEP_FWD_AX, V>(s, g, q, S, spmv_x, nullptr, st);
  else launch_sweep<SWEEP_FWD, V>(s, g, q, S, y, nullptr, st);
}
void launch_fwd(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSys &S, const double *y,
                const double *spmv_x, SolveState *st, double *ybuf) {
  launch_fwd_t<double>(s, g, q, S, y, spmv_x, st, ybuf);
}
void launch_fwd_f(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysF &S, const float *y,
                  const float *spmv_x, SolveState *st, float *ybuf) {
  launch_fwd_t<float>(s, g, q, S, y, spmv_x, st, ybuf);
}
void launch_bwd(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSys &S, double *x, SolveState *st) {
  launch_sweep<SWEEP_BWD, double>(s, g, q, S, nullptr, x, st);
}
void launch_bwd_f(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysF &S, float *x, SolveState *st) {
  launch_sweep<SWEEP_BWD, float>(s, g, q, S, nullptr, x, st);
}
// The FP32 backward sweep with the inner products that follow it summed
// on the way (mode 3: (R0,X); mode 4: the five sums of k_dot5f), one
// partial per tile into rb (rb + c*nb for sum c).  One layout tile per
// preconditioner block, blocks of up to 512 threads; false (nothing
// launched) where that does not hold.
template <int MODE>
static bool launch_bwd_dots(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysF &S, const float *r0,
                            const float *rr, float *x, double *rb, SolveState *st) {
  if (q.split != 1 || sweep_threads(q.T) > 512 || sweep_depth(q, MODE, 4) < 2) return false;
  launch_sweep<MODE, float>(s, g, q, S, r0, x, st, rr, rb);
  return true;
}
bool launch_bwd_f_dot1(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysF &S, const float *r0, float *x,
                       double *rb, SolveState *st) {
  return launch_bwd_dots<SWEEP_BWD1>(s, g, q, S, r0, nullptr, x, rb, st);
}
bool launch_bwd_f_dot5(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysF &S, const float *r0,
                       const float *rr, float *x, double *rb, SolveState *st) {
  return launch_bwd_dots<SWEEP_BWD5>(s, g, q, S, r0, rr, x, rb, st);
}
static inline unsigned slab_blocks(const SkewGeo &q) { return (unsigned)slab_partials(q); }
#define SL(kern, ...) launch_pdl(kern, dim3(slab_blocks(q)), dim3(ROW_THREADS), 0, s, 1, __VA_ARGS__)
static inline unsigned flat_blocks(const SkewGeo &q) { return (unsigned)((skew_entries(q) + FLAT_BLOCK - 1) / FLAT_BLOCK); }
#define FL(kern, ...) launch_pdl(kern, dim3(flat_blocks(q)), dim3(256), 0, s, 1, __VA_ARGS__)
template <typename V>
void launch_spmv_t(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSysT<V> &S, const V *x, V *y,
                   const SolveState *st) { SL(k_spmv<V>, g, q, S, x, y, st); }
void launch_resid(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSys &S, const double *b, const double *x,
                  double *y, double *rb0, double *rb1, const SolveState *st) {
  SL(k_resid, g, q, S, b, x, y, rb0, rb1, st);
}
template <typename V>
void launch_dot_t(cudaStream_t s, const Geo &g, const SkewGeo &q, const V *x0, const V *y0, const V *x1,
                  const V *y1, double *rb0, double *rb1, const SolveState *st) {
  SL(k_dot<V>, g, q, x0, y0, x1, y1, rb0, rb1, st);
}
template <typename V>
void launch_copy2_t(cudaStream_t s, const SkewGeo &q, const V *r0, V *rr, V *pp,
                    const SolveState *st) { FL(k_copy2<V>, q, r0, rr, pp, st); }
template void launch_spmv_t<double>(cudaStream_t, const Geo &, const SkewGeo &, const SkewSysT<double> &,
                                    const double *, double *, const SolveState *);
template void launch_spmv_t<float>(cudaStream_t, const Geo &, const SkewGeo &, const SkewSysT<float> &,
                                   const float *, float *, const SolveState *);
template void launch_dot_t<double>(cudaStream_t, const Geo &, const SkewGeo &, const double *, const double *,
                                   const double *, const double *, double *, double *, const SolveState *);
template void launch_dot_t<float>(cudaStream_t, const Geo &, const SkewGeo &, const float *, const float *,
                                  const float *, const float *, double *, double *, const SolveState *);
template void launch_copy2_t<double>(cudaStream_t, const SkewGeo &, const double *, double *, double *,
                                     const SolveState *);
template void launch_copy2_t<float>(cudaStream_t, const SkewGeo &, const float *, float *, float *,
                                    const SolveState *);
void launch_axpy_rr(cudaStream_t s, const SkewGeo &q, const double *ap, double *rr,
                    const SolveState *st) { FL(k_axpy_rr, q, ap, rr, st); }
void launch_upd_xr(cudaStream_t s, const Geo &g, const SkewGeo &q, const double *pp, const double *ae,
                   const double *r0, double *xw, double *rr, double *rb0, double *rb1, const SolveState *st) {
  SL(k_upd_xr, g, q, pp, ae, r0, xw, rr, rb0, rb1, st);
}
void launch_upd_p(cudaStream_t s, const SkewGeo &q, const double *rr, const double *ap,
                  double *pp, const SolveState *st) { FL(k_upd_p, q, rr, ap, pp, st); }
void launch_x0(cudaStream_t s, const Geo &g, const SkewGeo &q, const int *indc, const double *xw, double *x0,
               const SolveState *st) { SL(k_x0, g, q, indc, xw, x0, st); }
void launch_relres(cudaStream_t s, const Geo &g, const SkewGeo &q, const SkewSys &S, const double *b,
                   const double *x, double *rb0, double *rb1) { SL(k_relres, g, q, S, b, x, rb0, rb1); }
void launch_dot2f(cudaStream_t s, const Geo &g, const SkewGeo &q, const float *r0, const float *ap, double *rb,
                  const SolveState *st) { SL(k_dot2f, g, q, r0, ap, rb, st); }
void launch_axpyf(cudaStream_t s, const SkewGeo &q, const float *ap, float *rr, const SolveState *st) {
  FL(k_axpyf, q, ap, rr, st);
}
void launch_dot5f(cudaStream_t s, const Geo &g, const SkewGeo &q, const float *r0, const float *rr, const float *ae,
                  double *rb, const SolveState *st) { SL(k_dot5f, g, q, r0, rr, ae, rb, st); }
void launch_upd3f(cudaStream_t s, const SkewGeo &q, const float *ae, const float *ap, float *xw, float *rr,
                  float *pp, const SolveState *st) { FL(k_upd3f, q, ae, ap, xw, rr, pp, st); }
void launch_fin5(cudaStream_t s, const double *rb, long long nrows, SolveState *st, double epsa2, double epsr2,
                 double div2, int icgmax) {
  launch_pdl(k_fin5, dim3(1), dim3(1024), 0, s, 1, rb, nrows, st, epsa2, epsr2, div2, icgmax);
}
void launch_commit(cudaStream_t s, SolveState *st) { launch_pdl(k_commit, dim3(1), dim3(1), 0, s, 1, st); }
void launch_sys_to_f(cudaStream_t s, const SkewGeo &q, const double *sys, float *sysf) {
  const long long n = skew_entries(q);
  launch_pdl(k_sys_to_f, dim3((unsigned)std::min<long long>((n + 255) / 256, 148LL * 16)), dim3(256), 0, s, 1, q, sys,
             sysf);
}
void launch_scale_to_f(cudaStream_t s, const SkewGeo &q, const double *r, double scale, float *rf) {
  FL(k_scale_to_f, q, r, scale, rf);
}
void launch_add_f(cudaStream_t s, const SkewGeo &q, const float *d, double inv_scale, double *x) {
  FL(k_add_f, q, d, inv_scale, x);
}
#undef FL
#undef SL
void launch_fin(cudaStream_t s, int mode, const double *rb0, const double *rb1, long long nrows,
                SolveState *st, double *out, double epsa2, double epsr2, double div2, int icgmax) {
  launch_pdl(k_fin, dim3(1), dim3(1024), 0, s, 1, mode, rb0, rb1, nrows, st, out, epsa2, epsr2, div2, icgmax);
}
void launch_pivot_check(cudaStream_t s, SolveState *st) {
  launch_pdl(k_pivot_check, dim3(1), dim3(1), 0, s, 1, st);
}
void launch_vmodif(cudaStream_t s, const Geo &g, const Fld &f, const Prm &p, const double *pt) {
  k_vmodif<<<cell_grid(g), CELL_THREADS, 0, s>>>(g, f, p, pt);
  count_launch();
}


// ---------------------------------------------------- batched solves
// A block's member: the largest m with pre[m] <= blk (pre ascending).
__device__ __forceinline__ int batch_member(const int *pre, int nm, int blk) {
  int lo = 0, hi = nm - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= blk) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
#define BATCH_BLOCK(range)                                                     \
  const int *pr_ = pre + (range) * (nm + 1);                                   \
  const int m_ = batch_member(pr_, nm, (int)blockIdx.x);                       \
  const BatchMember &M = bm[m_];                                               \
  const unsigned lb_ = blockIdx.x - (unsigned)pr_[m_];

__global__ void kb_to_skew(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_ELEM)
  if (!M.active) return;
  const long long e = (long long)lb_ * BATCH_ELEM + threadIdx.x;
  if (e < (long long)M.q.nb * M.q.W * M.q.T)
    to_skew_elem(M.g, M.q, M.a, M.indc, M.S, M.pt, M.vd[BD_B], M.vd[BD_X], M.warm, e);
}
__global__ void kb_sys_to_f(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_ELEM)
  if (!M.active) return;
  const long long e = (long long)lb_ * BATCH_ELEM + threadIdx.x;
  if (e < skew_entries(M.q)) sys_to_f_elem(M.q, M.S.sys, M.Sf.sys, e);
}
template <int D>
__global__ void kb_dcmp_f(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_TILE)
  if (!M.active) return;
  dcmp_body<D, float>(M.g, M.q, (float)M.U, M.Sf, M.pivot_bad, (int)(lb_ % M.q.ntx), (int)(lb_ / M.q.ntx));
}
template <int D, int MODE, int MAXT, int MINB, int CT, int CTIP, bool ONE = false>
__global__ void __launch_bounds__(MAXT, MINB) kb_sweep(const BatchMember *bm, const int *pre, int nm, int vin,
                                                       int vout, int vin2, int rb5) {
  pdl_enter();
  BATCH_BLOCK(BR_TILE)
  sweep_cp_body<D, MODE, float, CT, CTIP, ONE>(M.g, M.q, M.Sf, vin >= 0 ? M.vf[vin] : nullptr,
                                               vout >= 0 ? M.vf[vout] : nullptr, M.st,
                                               vin2 >= 0 ? M.vf[vin2] : nullptr, rb5 ? M.rb5 : M.rb0,
                                               (int)(lb_ % M.q.ntx), (int)(lb_ / M.q.ntx));
}
// the bulk-copy ring: a member's stall is on
template <int MODE>
__global__ void __launch_bounds__(512, 1) kb_sweep_ring(const BatchMember *bm, const int *pre, int nm, int vin,
                                                        int vout, int vin2, int rb5, int D) {
  pdl_enter();
  BATCH_BLOCK(BR_TILE)
  sweep_body<MODE, float, 1>(M.g, M.q, M.Sf, vin >= 0 ? M.vf[vin] : nullptr, vout >= 0 ? M.vf[vout] : nullptr, M.st,
                             vin2 >= 0 ? M.vf[vin2] : nullptr, rb5 ? M.rb5 : M.rb0, (int)(lb_ % M.q.ntx),
                             (int)(lb_ / M.q.ntx), D);
}
// the solve state of every member cleared up to the wait limit; members
// outside the pass marked done, so every solver kernel skips them
__global__ void kb_clear(const BatchMember *bm, int nm) {
  pdl_enter();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= nm) return;
  unsigned char *p = reinterpret_cast<unsigned char *>(bm[m].st);
  for (int i = 0; i < (int)SOLVE_CLEAR_BYTES; ++i) p[i] = 0;
  bm[m].st->done = bm[m].active ? 0 : 1;
  if (bm[m].pivot_bad) *bm[m].pivot_bad = 0;
}
__global__ void kb_gather(const BatchMember *bm, int nm, double *out) {
  pdl_enter();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= nm) return;
  const SolveState *st = bm[m].st;
  double *o = out + (long long)m * BATCH_GATHER;
  o[0] = st->done; o[1] = st->timeout; o[2] = st->iter; o[3] = st->pivot_bad;
  o[4] = bm[m].dres[6]; o[5] = bm[m].dres[7];
}
// r = b - A x in FP64 and the slab partials of (b,b) and (r,r)
__global__ void kb_residual(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_SLAB)
  resid_body(M.g, M.q, M.S, M.vd[BD_B], M.vd[BD_X], M.vd[BD_Y2], M.rb0, M.rb1, M.st, lb_);
}
// one block per member: the finaliser of its sums (tile partials after a
// backward sweep with sums, slab-block partials otherwise)
__global__ void kb_fin(const BatchMember *bm, int nm, int mode, int tile_partials) {
  pdl_enter();
  const BatchMember &M = bm[blockIdx.x];
  if (mode == FIN_STORE && !M.active) return;
  const long long nrows = tile_partials ? (long long)M.q.nb : M.nrb;
  fin_body(mode, M.rb0, mode == FIN_STORE ? M.rb1 : nullptr, nrows, M.st, M.dres + 6, M.epsa2, M.eps2, M.div2,
           M.icgmax);
}
__global__ void kb_fin5(const BatchMember *bm, int nm) {
  pdl_enter();
  const BatchMember &M = bm[blockIdx.x];
  fin5_body(M.rb5, (long long)M.q.nb, M.st, M.epsa2, M.eps2, M.div2, M.icgmax);
}
__global__ void kb_commit(const BatchMember *bm, int nm) {
  pdl_enter();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < nm && bm[m].st->stop) bm[m].st->done = 1;
}
// the inner solve's start: BF = R/|r|, D = 0
__global__ void __launch_bounds__(256) kb_start_f(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_FLAT)
  if (!M.active) return;
  scale_to_f_body(M.q, M.vd[BD_Y2], M.scale, M.vf[BF_B], lb_);
  const unsigned BX_ = lb_;
  float4 *x = reinterpret_cast<float4 *>(M.vf[BF_X]);
  FLAT_LOOP_BEGIN(M.q, 4, 4)
  EACH(4) x[e[u]] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  FLAT_LOOP_END
}
__global__ void kb_dot_r0f(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_SLAB)
  dot_body<float>(M.g, M.q, M.vf[BF_R0], M.vf[BF_R0], nullptr, nullptr, M.rb0, nullptr, M.st, lb_);
}
__global__ void __launch_bounds__(256) kb_copy2_f(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_FLAT)
  copy2_body<float>(M.q, M.vf[BF_R0], M.vf[BF_RR], M.vf[BF_PV], M.st, lb_);
}
__global__ void __launch_bounds__(256) kb_axpyf(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_FLAT)
  axpyf_body(M.q, M.vf[BF_AP], M.vf[BF_RR], M.st, lb_);
}
__global__ void __launch_bounds__(256) kb_upd3f(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_FLAT)
  upd3f_body(M.q, M.vf[BF_AE], M.vf[BF_AP], M.vf[BF_X], M.vf[BF_RR], M.vf[BF_PV], M.st, lb_);
}
// XW += |r| D on the members whose inner solve ended within ICGMAX
__global__ void __launch_bounds__(256) kb_add_f(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_FLAT)
  if (!M.active || M.st->iter < 0 || M.st->iter > M.icgmax) return;
  add_f_body(M.q, M.vf[BF_X], M.rn, M.vd[BD_X], lb_);
}
__global__ void kb_x0(const BatchMember *bm, const int *pre, int nm) {
  pdl_enter();
  BATCH_BLOCK(BR_SLAB)
  if (!M.active) return;
  x0_body(M.g, M.q, M.S.indc, M.vd[BD_X], M.pt, M.st, lb_);
}
#undef BATCH_BLOCK

static inline dim3 bgrid(long long n) { return dim3((unsigned)n); }
void launch_b_to_skew(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nblk) {
  launch_pdl(kb_to_skew, bgrid(nblk), dim3(BATCH_ELEM), 0, s, 1, bm, pre, nm);
}
void launch_b_sys_to_f(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nblk) {
  launch_pdl(kb_sys_to_f, bgrid(nblk), dim3(BATCH_ELEM), 0, s, 1, bm, pre, nm);
}
bool launch_b_dcmp_f(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long ntiles, int T) {
  const int d = ring_depth(7, T, sizeof(float));
  const size_t bytes = ring_bytes(7, T, d + 3, sizeof(float));
  switch (d) {
#define BDCMP(DD)                                                                          \
  case DD:                                                                                 \
    set_smem(kb_dcmp_f<DD>, bytes);                                                        \
    launch_pdl(kb_dcmp_f<DD>, bgrid(ntiles), dim3(T), bytes, s, 1, bm, pre, nm);          \
    return true;
    BDCMP(8) BDCMP(4) BDCMP(2) BDCMP(1)
#undef BDCMP
    default: return false;
  }
}
// The batched FP32 sweeps: the form and depth of launch_sweep, by the tile
// shape that the members share (qref; qref.ring for the bulk-copy ring).
bool b_sweeps_supported(const SkewGeo &q) {
  if (q.split != 1 || sweep_threads(q.T) > 512) return false;
  for (int mode : {(int)SWEEP_FWD, (int)SWEEP_FWD_AX, (int)SWEEP_BWD, (int)SWEEP_BWD1, (int)SWEEP_BWD5})
    if (sweep_depth(q, mode, 4) < 2) return false;
  return true;
}
template <int MODE>
static bool launch_b_sweep_t(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long ntiles,
                             const SkewGeo &q, int vin, int vout, int vin2, int rb5) {
  SkewGeo qa = q;  // the depth by the tiles of all members
  qa.nb = (int)std::min<long long>(ntiles, 1 << 30);
  const int d = q.ring ? 0 : sweep_cp_depth(qa, MODE, 4), nt = sweep_cp_threads(q.T);
  if (d == 0) {
    const int dr = sweep_depth(q, MODE, 4);
    if (dr < 2) return false;
    const size_t bytes = sweep_bytes(q, MODE, dr, 4);
    set_smem(kb_sweep_ring<MODE>, bytes);
    launch_pdl(kb_sweep_ring<MODE>, bgrid(ntiles), dim3((unsigned)sweep_threads(q.T)), bytes, s, 1, bm, pre, nm, vin,
               vout, vin2, rb5, dr);
    return true;
  }
  const size_t bytes = sweep_cp_bytes(MODE, d, sweep_cp_unrolled(q, MODE, 4), q.T, q.TIp, q.TI, q.TJ, 4);
  const dim3 block((unsigned)nt);
#define BSWEEP_F(D, MT, MB, CT, CI, ONE)                                                                      \
  {                                                                                                           \
    set_smem(kb_sweep<D, MODE, MT, MB, CT, CI, ONE>, bytes);                                                  \
    launch_pdl(kb_sweep<D, MODE, MT, MB, CT, CI, ONE>, bgrid(ntiles), block, bytes, s, 1, bm, pre, nm, vin, vout, vin2, rb5); \
    return true;                                                                                              \
  }
#define BSWEEP(D, MT, MB, CT, CI) BSWEEP_F(D, MT, MB, CT, CI, false)
#define BSWEEP_128(D)                                            \
  {                                                              \
    if (q.T == 128 && q.TIp == 8) BSWEEP(D, 128, 1, 128, 8)      \
    if (q.T == 128 && q.TIp == 16) BSWEEP(D, 128, 1, 128, 16)    \
    BSWEEP(D, 128, 1, 0, 0)                                      \
  }
#define BSWEEP_D(D)                                              \
  {                                                              \
    if (nt <= 128) BSWEEP_128(D)                                 \
    if (nt <= 256) {                                             \
      if (q.T == 256 && q.TIp == 16) BSWEEP(D, 256, 2, 256, 16)  \
      BSWEEP(D, 256, 2, 0, 0)                                    \
    }                                                            \
    BSWEEP(D, 576, 1, 0, 0)                                      \
  }
  if constexpr (MODE == SWEEP_FWD_AX) {
    if (q.one) {
      if (d == 8) BSWEEP_F(8, 576, 1, 0, 0, true)
      if (d == 4) BSWEEP_F(4, 576, 1, 0, 0, true)
      BSWEEP_F(2, 576, 1, 0, 0, true)
    }
    if (d == 12) BSWEEP_128(12)
    if (d == 8) BSWEEP_D(8)
    if (d == 6) BSWEEP_D(6)
    if (d == 4) BSWEEP_D(4)
    BSWEEP_D(2)
  } else {
    if (d == 15) BSWEEP_128(15)
    if (d == 9) BSWEEP_D(9)
    BSWEEP_D(3)
  }
#undef BSWEEP_D
#undef BSWEEP_128
#undef BSWEEP
#undef BSWEEP_F
}
bool launch_b_sweep(cudaStream_t s, int mode, const BatchMember *bm, const int *pre, int nm, long long ntiles,
                    const SkewGeo &q, int vin, int vout, int vin2, bool rb5) {
  switch (mode) {
    case SWEEP_FWD: return launch_b_sweep_t<SWEEP_FWD>(s, bm, pre, nm, ntiles, q, vin, vout, vin2, rb5);
    case SWEEP_FWD_AX: return launch_b_sweep_t<SWEEP_FWD_AX>(s, bm, pre, nm, ntiles, q, vin, vout, vin2, rb5);
    case SWEEP_BWD: return launch_b_sweep_t<SWEEP_BWD>(s, bm, pre, nm, ntiles, q, vin, vout, vin2, rb5);
    case SWEEP_BWD1: return launch_b_sweep_t<SWEEP_BWD1>(s, bm, pre, nm, ntiles, q, vin, vout, vin2, rb5);
    case SWEEP_BWD5: return launch_b_sweep_t<SWEEP_BWD5>(s, bm, pre, nm, ntiles, q, vin, vout, vin2, rb5);
    default: return false;
  }
}
// one thread per member
static inline dim3 bmem(int nm) { return dim3((unsigned)((nm + 255) / 256)); }
void launch_b_clear(cudaStream_t s, const BatchMember *bm, int nm) {
  launch_pdl(kb_clear, bmem(nm), dim3(256), 0, s, 1, bm, nm);
}
void launch_b_gather(cudaStream_t s, const BatchMember *bm, int nm, double *out) {
  launch_pdl(kb_gather, bmem(nm), dim3(256), 0, s, 1, bm, nm, out);
}
void launch_b_residual(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nslab) {
  launch_pdl(kb_residual, bgrid(nslab), dim3(ROW_THREADS), 0, s, 1, bm, pre, nm);
}
void launch_b_fin(cudaStream_t s, int mode, const BatchMember *bm, int nm, bool tile_partials) {
  launch_pdl(kb_fin, dim3((unsigned)nm), dim3(1024), 0, s, 1, bm, nm, mode, tile_partials ? 1 : 0);
}
void launch_b_fin5(cudaStream_t s, const BatchMember *bm, int nm) {
  launch_pdl(kb_fin5, dim3((unsigned)nm), dim3(1024), 0, s, 1, bm, nm);
}
void launch_b_commit(cudaStream_t s, const BatchMember *bm, int nm) {
  launch_pdl(kb_commit, bmem(nm), dim3(256), 0, s, 1, bm, nm);
}
#define BSL(kern, n) launch_pdl(kern, bgrid(n), dim3(ROW_THREADS), 0, s, 1, bm, pre, nm)
void launch_b_start_f(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nflat) { BSL(kb_start_f, nflat); }
void launch_b_dot_r0f(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nslab) { BSL(kb_dot_r0f, nslab); }
void launch_b_copy2_f(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nflat) { BSL(kb_copy2_f, nflat); }
void launch_b_axpyf(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nflat) { BSL(kb_axpyf, nflat); }
void launch_b_upd3f(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nflat) { BSL(kb_upd3f, nflat); }
void launch_b_add_f(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nflat) { BSL(kb_add_f, nflat); }
void launch_b_x0(cudaStream_t s, const BatchMember *bm, const int *pre, int nm, long long nslab) { BSL(kb_x0, nslab); }
#undef BSL

}  // namespace cadmas
