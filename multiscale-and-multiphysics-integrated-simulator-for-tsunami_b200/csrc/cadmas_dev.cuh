// cadmas_dev.cuh -- device-side definitions shared by the kernels of
// libcadmas_gpu.so (B200, sm_100a, FP64).
//
// Arithmetic rule for the whole library: every expression is written in the
// operand order of the Fortran routine it restates and compiled with
// --fmad=false, with IEEE division and square root, so that each cell value
// is bit-identical to a sequential evaluation of the same expression.
// Global sums use one fixed tree (row_reduce below); no atomics touch a
// floating-point value.
#pragma once
#include <cstddef>
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/cadmas_gpu.h"

namespace cadmas {

// ----------------------------------------------------------------- geometry
struct Geo {
  int NI, NJ, NK, NB;
  long long N;                 // NI*NJ*NK
  const double *XX, *YY, *ZZ;  // (6,N*) metrics
};

__device__ __forceinline__ long long cid(const Geo &g, int i, int j, int k) {
  return (long long)(i - 1) + (long long)g.NI * ((long long)(j - 1) + (long long)g.NJ * (long long)(k - 1));
}
// The metrics are constant: read-only loads, which stay valid across the
// kernels' stores.
__device__ __forceinline__ double gx(const Geo &g, int m, int i) { return __ldg(g.XX + (m - 1) + 6 * (i - 1)); }
__device__ __forceinline__ double gy(const Geo &g, int m, int j) { return __ldg(g.YY + (m - 1) + 6 * (j - 1)); }
__device__ __forceinline__ double gz(const Geo &g, int m, int k) { return __ldg(g.ZZ + (m - 1) + 6 * (k - 1)); }

// MAX/MIN with the comparison the oracle uses (first operand on ties).
__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }

// libgfortran's integer power (square and multiply), as x**n compiles.
__device__ __forceinline__ double ipow(double x, int n) {
  double p = 1.0;
  if (n != 0) {
    unsigned u;
    if (n < 0) { u = (unsigned)(-n); x = p / x; } else { u = (unsigned)n; }
    for (;;) {
      if (u & 1u) p *= x;
      u >>= 1;
      if (u) x *= x; else break;
    }
  }
  return p;
}

// -------------------------------------------------------------- parameters
struct Prm {
  double rho0, grz0, vvmax, cgpara, cgepsa, cgepsr, cgdiv, flower, fupper,
      plower, scmvp, wvlvl, wbub, glxmin, glxmax, glymin, glymax;
  double dtnow, tnow;
  int icgtyp, icgmax, ibsuw0;
  // sponge (vf_veuler.f:77-113), precomputed on the host
  int ipa, ip[4];
  double sw[4], spx[4], spz[4];
  // log-law and rough walls (IB 6, 8): kappa, A, ANU0; loglaw = 1 when the
  // grid has such faces
  double akk0, aka0, anu0;
  int loglaw;
  // fixlvl[JD-1] = 1: side JD is a wave side whose table fixes the water
  // level (MTBTYP 3); its faces then act as free faces
  int fixlvl[4];
  // wave source (ISCTYP(1)): IWS > 0 the x source's column I, JWS > 0 the
  // y source's row J (0: none); SRCUV in Fld::srcuv
  int iws, jws;
};

// A boundary face of a fixed-water-level side: on the domain boundary of
// the side its NS names (vf_bwuwn.f:161-216, vf_vmodif.f:89-112,
// vf_bwuwt.f:80-115).
__device__ __forceinline__ bool fixlvl_face(const Geo &g, const Prm &p, int NS, int I, int J) {
  if (NS < 1 || NS > 4 || !p.fixlvl[NS - 1]) return false;
  return NS == 1 ? I == 2 : NS == 2 ? I == g.NI : NS == 3 ? J == 2 : J == g.NJ;
}

// ---------------------------------------------------------- device arrays
struct Fld {
  // static
  const double *ggv, *ggx, *ggy, *ggz, *glv, *glx, *gly, *glz, *cd0, *anu;
  const int *indx, *indy, *indz, *indb;
  // state
  double *uu, *vv, *ww, *pp, *ff;
  int *nf, *indc, *nf0;
  double *bcu, *bcv, *bcw, *bcp, *bcf;
  const double *bcvi;  // BCVI roughness of rough-wall faces
  // SRCUV(NUMIJ,NUMK) of the wave source (NUMIJ = NUMJ for an x source,
  // NUMI for a y source); read only where Prm::iws or jws is set
  const double *srcuv;
};

// DROPTX, DROPTY, DROPTZ, DROPUU, DROPVV, DROPWW of the droplet model
struct DropArrays {
  double *tx, *ty, *tz, *uu, *vv, *ww;
};

// k-epsilon state (AK, AE, ANUT per cell; BCK, BCE and the types INDBK,
// INDBE per boundary face) and the constants of /VF_APHYSR/
struct KeArrays {
  double *ak, *ae, *anut, *bck, *bce;
  const int *indbk, *indbe;
};
struct KeConst {
  double anu0, scmk, akmink, akmine, akinik, akinie, akcmu, aksgk, aksge, akc1, akc2, akc3;
};

__device__ __forceinline__ int indb(const Fld &f, int m, int l) { return f.indb[(m - 1) + 4 * (l - 1)]; }

__device__ __forceinline__ void decode(const Geo &g, int ijk, int &i, int &j, int &k) {
  k = (ijk - 1) / (g.NI * g.NJ) + 1;
  ijk = ijk - g.NI * g.NJ * (k - 1);
  j = (ijk - 1) / g.NI + 1;
  i = ijk - g.NI * (j - 1);
}

// ------------------------------------------------------------ row kernels
// A "row kernel" maps one warp to one x-row (J,K) of the padded grid and
// lets lane l visit I = l+1, l+33, ...  Coalesced for the I-fastest layout,
// and the order in which each lane visits cells is the order of the global
// sums below.
constexpr int ROWS_PER_BLOCK = 8;
constexpr int ROW_THREADS = 32 * ROWS_PER_BLOCK;

inline unsigned row_blocks(const Geo &g) {
  long long rows = (long long)g.NJ * g.NK;
  return (unsigned)((rows + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK);
}

#define ROW_LOOP_BEGIN(g)                                                   \
  const int lane_ = threadIdx.x & 31;                                       \
  const long long row_ = (long long)blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 5); \
  if (row_ < (long long)(g).NJ * (g).NK) {                                  \
    const int J = (int)(row_ % (g).NJ) + 1;                                 \
    const int K = (int)(row_ / (g).NJ) + 1;                                 \
    for (int I = lane_ + 1; I <= (g).NI; I += 32) {
#define ROW_LOOP_END \
    }                \
  }

// A "cell kernel" (no sum over the grid) gives every thread one cell: the
// threads of a block take consecutive cells of an x-y plane, blockIdx.y the
// plane.  No lane walks a row on its own, so a row costs one cell's latency
// and not NI/32 of them, a small grid fills the chip (66x10x34 cells: 204
// blocks instead of 43) and a ragged row leaves no lanes idle.
constexpr int CELL_THREADS = 128;
inline dim3 cell_grid(const Geo &g, int kper = 1) {
  const int ny = (g.NK + kper - 1) / kper;
  return dim3(((unsigned)g.NI * (unsigned)g.NJ + CELL_THREADS - 1) / CELL_THREADS, (unsigned)(ny < 65535 ? ny : 65535));
}
#define CELL_IJ(g)                                             \
  const unsigned p_ = blockIdx.x * CELL_THREADS + threadIdx.x; \
  if (p_ < (unsigned)(g).NI * (unsigned)(g).NJ) {              \
    const int J = (int)(p_ / (unsigned)(g).NI) + 1;            \
    const int I = (int)(p_ % (unsigned)(g).NI) + 1;
#define CELL_LOOP_BEGIN(g) \
  CELL_IJ(g)               \
    for (int K = (int)blockIdx.y + 1; K <= (g).NK; K += (int)gridDim.y) {
#define CELL_LOOP_END \
    }                 \
  }
// A "scan kernel" acts on the few cells whose flag n_ satisfies `pred`:
// a thread reads the flags of SCAN_K planes at once and visits its hits.
// (The kernels that change the flags in place change a cell's flag only
// from its own thread.)
constexpr int SCAN_K = 4;
#define SCAN_LOOP_BEGIN(g, NF_, pred)                                                             \
  CELL_IJ(g)                                                                                      \
    const long long plane_ = (long long)(g).NI * (g).NJ;                                          \
    for (int K0_ = (int)blockIdx.y * SCAN_K + 1; K0_ <= (g).NK; K0_ += (int)gridDim.y * SCAN_K) { \
      unsigned m_ = 0;                                                                            \
      int v_[SCAN_K];                                                                             \
      _Pragma("unroll") for (int u_ = 0; u_ < SCAN_K; ++u_)                                       \
        v_[u_] = (NF_)[p_ + plane_ * (min(K0_ + u_, (g).NK) - 1)];                                \
      _Pragma("unroll") for (int u_ = 0; u_ < SCAN_K; ++u_) {                                     \
        const int n_ = v_[u_];                                                                    \
        if (K0_ + u_ <= (g).NK && (pred)) m_ |= 1u << u_;                                         \
      }                                                                                           \
      for (; m_; m_ &= m_ - 1) {                                                                  \
        const int K = K0_ + __ffs((int)m_) - 1;
#define SCAN_LOOP_END \
      }               \
    }                 \
  }
// Loads that stay where they are written, so that those of a cell are all in
// flight together (left to itself the compiler sinks each into the branch
// that uses it).  Not for arrays that the kernel writes.
__device__ __forceinline__ double ld_now(const double *p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int ld_now(const int *p) {
  int v;
  asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Programmatic dependent launch.  The solver's kernels are launched with
// programmatic stream serialisation (launch_pdl), so a kernel may be
// scheduled while the previous kernel of the stream still runs.  Each of
// them starts here: wait until the previous kernel has completed and its
// writes are visible, then let the next kernel be scheduled.  Without a
// programmatic dependency the wait returns at once.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// Warp tree: lane 0 ends with ((s0+s16)+(s8+s24))+... via shfl_down.
__device__ __forceinline__ double warp_tree(double s) {
  for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, off);
  return s;
}

// Store the row partial of a row kernel: call with every lane of the warp
// (lanes of an absent row store nothing).
__device__ __forceinline__ void row_store(double s, double *rowbuf, long long row, long long nrows) {
  s = warp_tree(s);
  if ((threadIdx.x & 31) == 0 && row < nrows) rowbuf[row] = s;
}

// Second stage: one block of 1024 threads sums the row partials of N
// buffers (together, so that one sum's latencies hide the others').
template <int N>
__device__ __forceinline__ void block_final_n(const double *const (&rowbuf)[N], long long nrows, double (&out)[N]) {
  __shared__ double w[N][32];
  // thread t sums rows t, t+1024, t+2048, ... in that order; the loads of
  // eight of them are issued before their additions
  double s[N];
#pragma unroll
  for (int c = 0; c < N; ++c) s[c] = 0.0;
  constexpr int L = N > 2 ? 2 : 8;
  for (long long r0 = threadIdx.x; r0 < nrows; r0 += L * 1024) {
    double v[N][L];
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int j = 0; j < L; ++j) v[c][j] = (r0 + j * 1024 < nrows) ? rowbuf[c][r0 + j * 1024] : 0.0;
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int j = 0; j < L; ++j)
        if (r0 + j * 1024 < nrows) s[c] = s[c] + v[c][j];
  }
#pragma unroll
  for (int c = 0; c < N; ++c) s[c] = warp_tree(s[c]);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int c = 0; c < N; ++c) w[c][threadIdx.x >> 5] = s[c];
  __syncthreads();
  if (threadIdx.x < 32)
#pragma unroll
    for (int c = 0; c < N; ++c) out[c] = warp_tree(w[c][threadIdx.x]);  // valid in thread 0
  __syncthreads();
}
__device__ __forceinline__ double block_final(const double *rowbuf, long long nrows) {
  const double *const b[1] = {rowbuf};
  double t[1] = {0.0};
  block_final_n<1>(b, nrows, t);
  return t[0];  // valid in thread 0
}

// -------------------------------------------------------- solver scalars
struct SolveState {
  double S, alpha, omega, beta, bnorm, xnorm, w1, w2, rn, bn;
  int iter, done, status, pivot_bad;
  int timeout;  // a bulk-copy wait of a sweep ran out of time
  int stop;     // regrouped FP32 iteration: finished, `done` after its last update
  // Set once per handle, kept when a solve clears the fields above (they
  // are read only where a sweep starts to wait, or by its producer warp,
  // so they add nothing to the sweeps' register load):
  //   wait_ns     an mbarrier wait of the sweeps gives up after this long
  //               and the solve ends with CADMAS_ETIMEOUT;
  //   stall_from  the producer warp issues no bulk copy for wavefront
  //               steps >= stall_from (failure injection for tests,
  //               cadmas_test_stall_sweeps; 2^30 otherwise).
  long long wait_ns;
  int stall_from, pad_;
};
// Bytes of SolveState that a new solve clears (everything before wait_ns).
#define SOLVE_CLEAR_BYTES offsetof(cadmas::SolveState, wait_ns)

// Error flags raised by kernels (bitmask in a device int).
enum : int {
  ERR_PG = 1,       // P.G ERROR (unexpected NF in VPCOEF, undetermined direction)
  ERR_CAP = 2,      // iteration cap
  ERR_UNSUP = 4,    // boundary type outside the implemented set
  ERR_NOTCONV = 8,  // the log-law friction velocity did not converge (VF_CLOGLW)
};

}  // namespace cadmas
