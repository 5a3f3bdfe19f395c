// k_unet.cu -- kernels of the learned warm start: a 3-level 3-D U-Net
// (BF16 weights and activations, FP32 accumulation) that maps (right-hand
// side, F, porosity, computed-cell mask) to an initial pressure correction.
//
// The 3x3x3 convolutions are implicit GEMMs on the tcgen05 tensor cores:
//   k_conv   D[voxel, cout] = sum over 27 taps and cin of X[voxel+tap, cin]
//            * W[cout, tap, cin].  A CTA owns a tile of bx x by voxels of
//            one z layer and all Cout (N).  For each of the three layers
//            z-1, z, z+1 it stages the tile with its halo once in shared
//            memory, as 16-byte rows of 8 channels per voxel in the linear
//            order of the padded tile; the nine taps of the layer then read
//            it through descriptors that start 16 bytes x (the tap's
//            offset) further on.  A row block of the MMA (M = 128) is 128
//            consecutive voxels of the padded tile; what falls on the
//            padding is computed and dropped.  The epilogue reads TMEM
//            (tcgen05.ld), adds the bias, applies ReLU or a ReLU-backward
//            mask and stores BF16 or FP32.  The input-gradient of a
//            convolution is the same kernel with the weights flipped and
//            transposed.
//   k_wgrad  dW[(tap,cin), cout] = sum over voxels of X[voxel+tap, cin] *
//            dY[voxel, cout]: M = 27*Cin rows in tiles of 128, N = Cout,
//            K = a slice of voxels in chunks of 64, both operands MN-major
//            (8 channels of a voxel are 16 consecutive bytes in memory and
//            in the tile); each CTA writes its slice's partial sums, which
//            k_wgrad_reduce adds in a fixed order.
// The rest are elementwise or gather kernels on CUDA cores.
//
// Layouts: activations channels-last, voxel v = x + X*(y + Y*(z + Z*b)),
// value [v*C + c]; FP32 weights [cout][tap][cin] with tap = (dz+1)*9 +
// (dy+1)*3 + (dx+1), their BF16 copies [tap][cin/8][cout][cin%8], the order
// of k_conv's tiles.  Every wait on an mbarrier is bounded: on a timeout the CTA
// records an error, waits once more for its MMAs, frees its TMEM and ends.
#include <algorithm>
#include <cuda_bf16.h>
#include "cadmas_dev.cuh"
#include "kernels.h"
#include "umma.cuh"

namespace cadmas {

using bf16 = __nv_bfloat16;

struct Vol {
  int X, Y, Z, B;
  __host__ __device__ __forceinline__ long long n() const { return (long long)X * Y * Z * B; }
};

// neighbour voxel of v at (dx,dy,dz), or -1 outside the volume
__device__ __forceinline__ long long nbr(const Vol &g, int x, int y, int z, int b, int dx, int dy, int dz) {
  const int xx = x + dx, yy = y + dy, zz = z + dz;
  if (xx < 0 || xx >= g.X || yy < 0 || yy >= g.Y || zz < 0 || zz >= g.Z) return -1;
  return (long long)xx + (long long)g.X * ((long long)yy + (long long)g.Y * ((long long)zz + (long long)g.Z * b));
}

__device__ __forceinline__ void decomp(const Vol &g, long long v, int &x, int &y, int &z, int &b) {
  x = (int)(v % g.X);
  long long r = v / g.X;
  y = (int)(r % g.Y);
  r /= g.Y;
  z = (int)(r % g.Z);
  b = (int)(r / g.Z);
}

// Every thread waits (bounded) for the phase of the given parity; the CTA
// goes on only if all of them saw it, so that no thread is left at a later
// barrier.
__device__ __forceinline__ bool cta_wait(uint64_t *bar, uint32_t parity) {
  const bool w = umma::mbar_wait(bar, parity);
  return __syncthreads_and(w) != 0;
}

// ------------------------------------------------------------- k_conv
constexpr int CONV_T = 256;  // threads: eight warps share the copies and the epilogue's row blocks
__global__ void __launch_bounds__(CONV_T) k_conv(Vol g, const bf16 *__restrict__ X, int Cin,
                                              const bf16 *__restrict__ W, const float *__restrict__ bias,
                                              int Cout, int mode, const bf16 *__restrict__ mask, void *Y,
                                              int *err, ConvPlan p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int N = Cout, C8 = Cin >> 3, P = p.P, PL = p.PL;
  const uint32_t st_bytes = p.a_bytes + p.b_bytes;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + (size_t)p.NST * st_bytes);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 2);
  const int tid = threadIdx.x, warp = tid >> 5;
  const uint32_t ncols = umma::tmem_cols(p.MT * N);
  // Issuing one MMA takes one thread longer than its 128 x 16 x 16 product
  // takes the tensor core: lane 0 of warp w issues those of row blocks w,
  // w + NI, ... (each accumulator's MMAs stay in one thread, in order).
  const int NI = min(CONV_T / 32, p.MT);
  const bool issuer = (tid & 31) == 0 && warp < NI;
  if (warp == 0) umma::tmem_alloc(tslot, ncols);
  if (tid == 0) {
    umma::mbar_init(&bar[0], NI);
    umma::mbar_init(&bar[1], NI);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const uint32_t sm0 = umma::smem_u32(smem);
  unsigned t = blockIdx.x;
  const int xt = (int)(t % p.nxt);
  t /= p.nxt;
  const int yt = (int)(t % p.nyt);
  t /= p.nyt;
  const int z = (int)(t % g.Z), b = (int)(t / g.Z);
  const int x0 = xt * p.bx, y0 = yt * p.by;
  // layer z + gi - 1 of the padded tile and its nine taps' weights into a
  // stage; thread tid takes the 16-byte chunks tid, tid + CONV_T, ... of every
  // row (chunk q of a row: voxel q / C8, channels 8 (q % C8) ..)
  const int nrow = p.by + 2, rsplit = max(1, min(nrow, CONV_T / (P * C8)));
  auto load = [&](int gi, int st) {
    const uint32_t As = sm0 + st * st_bytes, Bs = As + p.a_bytes;
    const int zz = z + gi - 1;
    const bool zok = zz >= 0 && zz < g.Z;
    const bf16 *plane = X + (long long)g.X * g.Y * ((long long)g.Z * b + (zok ? zz : z)) * Cin;
    for (int q = tid; q < P * C8 * rsplit; q += CONV_T) {
      const int qr = q / (P * C8), qc = q - qr * (P * C8);  // rows qr, qr + rsplit, ...
      const int xx = qc / C8, c8 = qc - xx * C8, gx = x0 + xx - 1;
      const bool xok = zok && gx >= 0 && gx < g.X;
      const bf16 *src = plane + ((long long)(xok ? gx : 0) * Cin + c8 * 8);
      uint32_t dst = As + (uint32_t)(c8 * PL + xx + qr * P) * 16u;
      for (int yy = qr; yy < nrow; yy += rsplit, dst += (uint32_t)(P * rsplit) * 16u) {
        const int gy = y0 + yy - 1;
        const bool ok = xok && gy >= 0 && gy < g.Y;
        umma::cp16z(dst, src + (long long)(ok ? gy : 0) * g.X * Cin, ok);
      }
    }
    const int nb = 9 * N * C8;
    const bf16 *wsrc = W + (long long)gi * nb * 8;
    for (int q = tid; q < nb; q += CONV_T) umma::cp16z(Bs + (uint32_t)q * 16u, wsrc + q * 8, true);
    umma::cp_commit();
  };
  const bool three = p.NST == 3;
  load(0, 0);
  load(1, 1);
  if (three) load(2, 2);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = umma::idesc_bf16_f32(CONV_M, N);
  // the nine taps of layer gi: per accumulator tap by tap, channels in order
  auto mmas = [&](int gi, int st) {
    umma::fence_after_sync();
    const uint32_t a0 = sm0 + st * st_bytes, b0 = a0 + p.a_bytes;
    for (int mt = warp; mt < p.MT; mt += NI) {
      const uint64_t ad0 = umma::smem_desc(a0, (uint32_t)PL * 16u, 128) + (uint64_t)(mt * CONV_M);
      uint64_t bd = umma::smem_desc(b0, (uint32_t)N * 16u, 128);
      const uint32_t d = tmem + mt * N;
#pragma unroll
      for (int t9 = 0; t9 < 9; ++t9) {
        uint64_t ad = ad0 + (uint64_t)((t9 / 3) * P + t9 % 3);  // rows from the tap's first voxel
        for (int kk = 0; kk < C8 / 2; ++kk) {
          umma::mma_bf16(d, ad, bd, idesc, (gi | t9 | kk) != 0);
          ad += (uint64_t)(2 * PL);
          bd += (uint64_t)(2 * N);
        }
      }
    }
  };
  bool ok = true;
  // layer 0, 1, 2 in turn; with two stages the third layer's copies wait
  // for the first layer's MMAs
  if (three) umma::cp_wait<2>(); else umma::cp_wait<1>();
  umma::fence_async_smem();
  __syncthreads();
  if (issuer) {
    mmas(0, 0);
    umma::mma_commit(&bar[0]);
  }
  __syncwarp();
  if (three) umma::cp_wait<1>(); else umma::cp_wait<0>();
  umma::fence_async_smem();
  __syncthreads();
  if (issuer) mmas(1, 1);
  __syncwarp();
  if (three) {
    umma::cp_wait<0>();
  } else {
    ok = cta_wait(&bar[0], 0);
    if (ok) load(2, 0);
    umma::cp_wait<0>();
  }
  umma::fence_async_smem();
  __syncthreads();
  if (issuer) {
    if (ok) mmas(2, three ? 2 : 0);
    umma::mma_commit(&bar[1]);
  }
  __syncwarp();
  // the last commit covers every MMA issued before it (after a timeout
  // this is the one more bounded wait before the TMEM is freed)
  if (!cta_wait(&bar[1], 0)) ok = false;
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);
  } else {
    umma::fence_after_sync();
    for (int mt = warp >> 2; mt < p.MT; mt += 2) {
      const int pos = mt * CONV_M + (tid & 127), yy = pos / P, xx = pos - yy * P, gx = x0 + xx, gy = y0 + yy;
      const bool live = xx < p.bx && yy < p.by && gx < g.X && gy < g.Y;
      const long long v = (long long)gx + (long long)g.X * (gy + (long long)g.Y * (z + (long long)g.Z * b));
      const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + mt * N;
      for (int c0 = 0; c0 < N; c0 += 8) {
        float a[8];
        umma::tmem_ld8(lane_base + c0, a);
        if (!live) continue;
        if (bias)
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] += bias[c0 + i];
        if (mode == CONV_RELU_BF16) {
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = fmaxf(a[i], 0.0f);
        } else if (mode == CONV_MASK_BF16) {
          // input gradient times the ReLU derivative of the layer below
          const uint4 mq = *reinterpret_cast<const uint4 *>(mask + v * Cout + c0);
          const bf16 *m = reinterpret_cast<const bf16 *>(&mq);
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = (__bfloat162float(m[i]) > 0.0f) ? a[i] : 0.0f;
        }
        if (mode == CONV_F32) {
          float *o = reinterpret_cast<float *>(Y) + v * Cout + c0;
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = a[i];
        } else {
          __align__(16) bf16 o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __float2bfloat16(a[i]);
          *reinterpret_cast<uint4 *>(reinterpret_cast<bf16 *>(Y) + v * Cout + c0) = *reinterpret_cast<uint4 *>(o);
        }
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_free(tmem, ncols);
}

// ------------------------------------------------------------ k_wgrad
// rows m = tap*Cin + cin (27*Cin of them, tiles of 128), N = Cout, K = the
// voxels of this CTA's slice in chunks of 64, WG_ST stages.  Tiles in
// shared memory: [8-channel block][voxel] of 16 bytes, so a thread copies
// 16 bytes of its voxel (or of its tap's neighbour) at a time.
constexpr int WG_K = 64;

template <int WG_ST>
__global__ void __launch_bounds__(128) k_wgrad(Vol g, const bf16 *__restrict__ X, int Cin,
                                               const bf16 *__restrict__ DY, int Cout, long long slice,
                                               float *__restrict__ part, int *err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int N = Cout, C8 = Cin >> 3, N8 = N >> 3;
  const uint32_t a_bytes = 128 * WG_K * 2, b_bytes = N * WG_K * 2, st_bytes = a_bytes + b_bytes;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + WG_ST * st_bytes);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + WG_ST);
  const int tid = threadIdx.x, warp = tid >> 5;
  const uint32_t ncols = umma::tmem_cols(N);
  if (warp == 0) umma::tmem_alloc(tslot, ncols);
  if (tid == 0) {
    for (int i = 0; i < WG_ST; ++i) umma::mbar_init(&bar[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot, sm0 = umma::smem_u32(smem);
  const uint32_t idesc = umma::idesc_bf16_f32_mn(128, N);
  const int M = 27 * Cin;
  const int m0 = blockIdx.x * 128;
  const long long V = g.n();
  const long long v0 = (long long)blockIdx.y * slice;
  const long long v1 = min(V, v0 + slice);
  const int nchunk = v1 > v0 ? (int)((v1 - v0 + WG_K - 1) / WG_K) : 0;
  // thread: voxel kq of each chunk; of the tile's 16 row blocks (8 channels
  // of one tap each) h, h+2, ..., of the N8 blocks of dY h, h+2, ...
  const int kq = tid & (WG_K - 1), h = tid >> 6;
  int off[8], tap[8];  // the neighbour's first value from the voxel's; tap (27: past the last row)
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gb = m0 / 8 + 2 * i + h, t = min(gb / C8, 27);
    off[i] = (((t / 9 - 1) * g.Y + (t / 3) % 3 - 1) * g.X + t % 3 - 1) * Cin + (gb - t * C8) * 8;
    tap[i] = t;
  }
  // position of the voxel to load next (chunks are loaded in order)
  long long v = v0 + kq;
  int x, y, z, b;
  decomp(g, min(v, V - 1), x, y, z, b);
  auto load = [&](int st) {
    const uint32_t As = sm0 + st * st_bytes, Bs = As + a_bytes;
    const bool live = v < v1;
    // taps inside the volume: a bit per (dz, dy, dx)
    const unsigned mx = 2u | (x > 0 ? 1u : 0u) | (x < g.X - 1 ? 4u : 0u);
    const unsigned m3 = (y > 0 ? mx : 0u) | mx << 3 | (y < g.Y - 1 ? mx << 6 : 0u);
    const unsigned in = live ? (z > 0 ? m3 : 0u) | m3 << 9 | (z < g.Z - 1 ? m3 << 18 : 0u) : 0u;
    const bf16 *xv = X + v * Cin;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool ok = in >> tap[i] & 1u;
      umma::cp16z(As + (uint32_t)((2 * i + h) * WG_K + kq) * 16u, ok ? xv + off[i] : X, ok);
    }
    for (int n = h; n < N8; n += 2)
      umma::cp16z(Bs + (uint32_t)(n * WG_K + kq) * 16u, live ? DY + v * Cout + n * 8 : DY, live);
    v += WG_K;
    x += WG_K;
    while (x >= g.X) {
      x -= g.X;
      if (++y == g.Y) { y = 0; if (++z == g.Z) { z = 0; ++b; } }
    }
  };
  bool ok = true;
  int committed = 0;
  for (int c = 0; c < WG_ST - 1; ++c) {
    if (c < nchunk) load(c);
    umma::cp_commit();
  }
  for (int ch = 0; ch < nchunk; ++ch) {
    const int s = ch % WG_ST, nx = ch + WG_ST - 1;  // (WG_ST is a constant)
    // chunk nx goes where chunk ch-1 lies: its MMAs must have read it
    if (ch >= 1 && !cta_wait(&bar[(ch - 1) % WG_ST], ((ch - 1) / WG_ST) & 1)) { ok = false; break; }
    if (nx < nchunk) load(nx % WG_ST);
    umma::cp_commit();
    umma::cp_wait<WG_ST - 1>();
    umma::fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      umma::fence_after_sync();
      const uint32_t a0 = sm0 + s * st_bytes, b0 = a0 + a_bytes;
      for (int kk = 0; kk < WG_K / 16; ++kk) {
        const uint64_t ad = umma::smem_desc(a0 + kk * 256, 128, WG_K * 16);
        const uint64_t bd = umma::smem_desc(b0 + kk * 256, 128, WG_K * 16);
        umma::mma_bf16(tmem, ad, bd, idesc, (ch | kk) != 0);
      }
      umma::mma_commit(&bar[s]);
    }
    ++committed;
  }
  umma::cp_wait<0>();
  if (committed > 0) {
    // on an earlier timeout this is the one more bounded wait for the MMAs
    // in flight before the TMEM is freed
    const int tl = committed - 1;
    if (!cta_wait(&bar[tl % WG_ST], (tl / WG_ST) & 1)) ok = false;
  }
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);
  } else {
    umma::fence_after_sync();
    const int m = m0 + warp * 32 + (tid & 31);
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    float *o = part + ((long long)blockIdx.y * M + m) * N;
    for (int c0 = 0; c0 < N; c0 += 8) {
      float a[8];
      umma::tmem_ld8(lane_base + c0, a);
      if (m < M && committed > 0)
#pragma unroll
        for (int i = 0; i < 8; ++i) o[c0 + i] = a[i];
      else if (m < M)
#pragma unroll
        for (int i = 0; i < 8; ++i) o[c0 + i] = 0.0f;
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_free(tmem, ncols);
}

// dW[cout][tap][cin] = sum over slices (in order) of part[s][tap*Cin+cin][cout]
__global__ void __launch_bounds__(64) k_wgrad_reduce(const float *part, int nslices, int Cin, int Cout, float *dW) {
  const int M = 27 * Cin;
  const int i = blockIdx.x * 64 + threadIdx.x;
  if (i >= M * Cout) return;
  float s = 0.0f;
  for (int q0 = 0; q0 < nslices; q0 += 16) {  // 16 loads in flight, added in order
    float r[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) r[j] = q0 + j < nslices ? part[(long long)(q0 + j) * M * Cout + i] : 0.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (q0 + j < nslices) s += r[j];
  }
  const int m = i / Cout, n = i % Cout, t = m / Cin, ci = m % Cin;
  dW[((long long)n * 27 + t) * Cin + ci] = s;
}

// Column sums in the order of the rows.  The rows come to shared memory by
// 16-byte asynchronous copies of all threads, then one thread per column
// adds them: the sequential order bounds the kernels (4 cycles per row), so
// the loads must not stand in its way.
// bias gradient: db[c] = sum over voxels of dY[v][c] (FP32 partials per
// block of 1024 voxels, then the same in order); C <= 64
__global__ void __launch_bounds__(256) k_bias_part(const bf16 *DY, long long V, int C, float *part) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const long long v0 = (long long)blockIdx.x * 1024;
  const int n = (int)min(1024LL, V - v0), nq = n * (C >> 3);
  const uint32_t sm0 = umma::smem_u32(smem);
  for (int q = threadIdx.x; q < nq; q += 256) umma::cp16z(sm0 + q * 16, DY + v0 * C + q * 8, true);
  umma::cp_commit();
  umma::cp_wait<0>();
  __syncthreads();
  if (threadIdx.x >= C) return;
  const bf16 *e = reinterpret_cast<const bf16 *>(smem) + threadIdx.x;
  float s = 0.0f;
  int r = 0;
  for (; r + 16 <= n; r += 16) {
    float f[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) f[j] = __bfloat162float(e[(r + j) * C]);
#pragma unroll
    for (int j = 0; j < 16; ++j) s += f[j];
  }
  for (; r < n; ++r) s += __bfloat162float(e[r * C]);
  part[(long long)blockIdx.x * C + threadIdx.x] = s;
}
// db[c] = sum of nb block partials in order; C <= 64
constexpr int SUM_ROWS = 64;
__global__ void __launch_bounds__(256) k_bias_reduce(const float *part, int nb, int C, float *db) {
  __shared__ float row[2][SUM_ROWS * 64];
  float s = 0.0f, reg[16];
  // rows q0 .. of the next stretch in registers while the last one is added
  auto fetch = [&](int q0) {
    const int n = min(SUM_ROWS, nb - q0) * C;
#pragma unroll
    for (int j = 0; j < 16; ++j) reg[j] = threadIdx.x + 256 * j < n ? part[(long long)q0 * C + threadIdx.x + 256 * j] : 0.0f;
  };
  auto put = [&](float *to) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (threadIdx.x + 256 * j < SUM_ROWS * C) to[threadIdx.x + 256 * j] = reg[j];
  };
  fetch(0);
  put(row[0]);
  int k = 0;
  for (int q = 0; q < nb; q += SUM_ROWS, k ^= 1) {
    __syncthreads();
    const bool more = q + SUM_ROWS < nb;
    if (more) fetch(q + SUM_ROWS);
    if (threadIdx.x < C) {
      const int n = min(SUM_ROWS, nb - q);
#pragma unroll 16
      for (int r = 0; r < n; ++r) s += row[k][r * C + threadIdx.x];
    }
    if (more) put(row[k ^ 1]);
  }
  if (threadIdx.x < C) db[threadIdx.x] = s;
}

// ------------------------------------------------ pooling and upsampling
// All of them move 8 channels (16 bytes) per thread: element i of the
// launch is channel block i % (C/8) of voxel i / (C/8).  They are bound by
// memory; one channel per thread took up to five times as long (upsampling
// and concatenation to 48 channels of 1.3 M voxels: 416 us).
struct alignas(16) B8 { bf16 v[8]; };
__device__ __forceinline__ B8 ld8(const bf16 *p) { return *reinterpret_cast<const B8 *>(p); }
__device__ __forceinline__ void st8(bf16 *p, const B8 &q) { *reinterpret_cast<B8 *>(p) = q; }
__device__ __forceinline__ bool split8(long long i, long long n, int C, long long &v, int &c) {
  const int C8 = C >> 3;
  if (i >= n * C8) return false;
  v = i / C8;
  c = (int)(i - v * C8) * 8;
  return true;
}
__device__ __forceinline__ long long coarse_of(const Vol &gc, int x, int y, int z, int b) {
  return (long long)(x >> 1) + (long long)gc.X * ((long long)(y >> 1) + (long long)gc.Y *
                                                    ((long long)(z >> 1) + (long long)gc.Z * b));
}
// sum of the 8 children of coarse voxel (x,y,z,b), channels c..c+7 of C
__device__ __forceinline__ void children8(const Vol &gf, int x, int y, int z, int b, const bf16 *F, int C, int c,
                                          float *s) {
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = 0.0f;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const B8 f = ld8(F + nbr(gf, 2 * x, 2 * y, 2 * z, b, q & 1, (q >> 1) & 1, q >> 2) * C + c);
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] += __bfloat162float(f.v[i]);
  }
}
// 2x2x2 average: coarse (X/2, Y/2, Z/2) from fine
__global__ void k_pool(Vol gc, const bf16 *F, int C, bf16 *Cc) {
  long long vc;
  int c, x, y, z, b;
  if (!split8(blockIdx.x * (long long)blockDim.x + threadIdx.x, gc.n(), C, vc, c)) return;
  decomp(gc, vc, x, y, z, b);
  const Vol gf{2 * gc.X, 2 * gc.Y, 2 * gc.Z, gc.B};
  float s[8];
  children8(gf, x, y, z, b, F, C, c, s);
  B8 o;
#pragma unroll
  for (int i = 0; i < 8; ++i) o.v[i] = __float2bfloat16(0.125f * s[i]);
  st8(Cc + vc * C + c, o);
}
// its backward, added to dF (fine), then masked by the ReLU of the fine
// activation: dF = bf16(dC/8 + dF) where act > 0, else 0
__global__ void k_pool_bwd(Vol gc, const bf16 *dC, int C, bf16 *dF, const bf16 *act) {
  const Vol gf{2 * gc.X, 2 * gc.Y, 2 * gc.Z, gc.B};
  long long vf;
  int c, x, y, z, b;
  if (!split8(blockIdx.x * (long long)blockDim.x + threadIdx.x, gf.n(), C, vf, c)) return;
  decomp(gf, vf, x, y, z, b);
  const B8 q = ld8(dC + coarse_of(gc, x, y, z, b) * C + c), a = ld8(act + vf * C + c);
  B8 o = ld8(dF + vf * C + c);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float e = 0.125f * __bfloat162float(q.v[i]);
    e += __bfloat162float(o.v[i]);
    o.v[i] = __bfloat162float(a.v[i]) > 0.0f ? __float2bfloat16(e) : __float2bfloat16(0.0f);
  }
  st8(dF + vf * C + c, o);
}
// out[vf] = (coarse[vf/2] (C1 channels), skip[vf] (C2 channels))
__global__ void k_upcat(Vol gf, const bf16 *Cc, int C1, const bf16 *S, int C2, bf16 *O) {
  const int C = C1 + C2;
  long long vf;
  int c, x, y, z, b;
  if (!split8(blockIdx.x * (long long)blockDim.x + threadIdx.x, gf.n(), C, vf, c)) return;
  const bf16 *src = S + vf * C2 + (c - C1);
  if (c < C1) {
    decomp(gf, vf, x, y, z, b);
    const Vol gc{gf.X / 2, gf.Y / 2, gf.Z / 2, gf.B};
    src = Cc + coarse_of(gc, x, y, z, b) * C1 + c;
  }
  st8(O + vf * C + c, ld8(src));
}
// backward: dCoarse = sum of the 8 children's first C1 channels; dSkip =
// the last C2 channels
__global__ void k_upcat_bwd_coarse(Vol gc, const bf16 *dO, int C1, int C2, bf16 *dC) {
  long long vc;
  int c, x, y, z, b;
  if (!split8(blockIdx.x * (long long)blockDim.x + threadIdx.x, gc.n(), C1, vc, c)) return;
  decomp(gc, vc, x, y, z, b);
  const Vol gf{2 * gc.X, 2 * gc.Y, 2 * gc.Z, gc.B};
  float s[8];
  children8(gf, x, y, z, b, dO, C1 + C2, c, s);
  B8 o;
#pragma unroll
  for (int i = 0; i < 8; ++i) o.v[i] = __float2bfloat16(s[i]);
  st8(dC + vc * C1 + c, o);
}
__global__ void k_upcat_bwd_skip(long long Vf, const bf16 *dO, int C1, int C2, bf16 *dS) {
  long long vf;
  int c;
  if (!split8(blockIdx.x * (long long)blockDim.x + threadIdx.x, Vf, C2, vf, c)) return;
  st8(dS + vf * C2 + c, ld8(dO + vf * (C1 + C2) + C1 + c));
}

// ------------------------------------------------------------- head
// y[v] = sum_c wh[c] a[v][c] + bh (FP32)
__global__ void k_head(long long V, const bf16 *A, int C, const float *wh, const float *bh, float *Yo) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  float s = bh[0];
  for (int c = 0; c < C; c += 8) {
    const B8 a = ld8(A + v * C + c);
#pragma unroll
    for (int i = 0; i < 8; ++i) s += wh[c + i] * __bfloat162float(a.v[i]);
  }
  Yo[v] = s;
}
// masked MSE: dy = 2 (y - t) m / sum(m); per-block partial loss sums
__global__ void k_mse(long long V, const float *Yo, const float *T, const float *Mk, float inv_n, float *dy,
                      float *lpart) {
  __shared__ float red[256];
  const long long v = (long long)blockIdx.x * 256 + threadIdx.x;
  float l = 0.0f;
  if (v < V) {
    const float e = (Yo[v] - T[v]) * Mk[v];
    dy[v] = 2.0f * e * inv_n;
    l = e * e;
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) lpart[blockIdx.x] = red[0];
}
// out[0] = sum of a (FP64; block partials in out[1..], added in order)
__global__ void __launch_bounds__(256) k_sum_part(long long n, const float *a, double *out) {
  __shared__ double red[8];
  double s = 0.0;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += 256LL * SUM_BLOCKS) s += (double)a[i];
  s = warp_tree(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int i = 1; i < 8; ++i) s += red[i];
  out[1 + blockIdx.x] = s;
}
__global__ void k_sum_fin(double *out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < SUM_BLOCKS; i += 32) s += out[1 + i];
  s = warp_tree(s);
  if (threadIdx.x == 0) out[0] = s;
}
// head backward: dA[v][c] = dy[v] wh[c] (BF16), masked by the ReLU of A
__global__ void k_head_bwd_act(long long V, const float *dy, const bf16 *A, int C, const float *wh, bf16 *dA) {
  long long v;
  int c;
  if (!split8(blockIdx.x * (long long)blockDim.x + threadIdx.x, V, C, v, c)) return;
  const B8 a = ld8(A + v * C + c);
  const float d = dy[v];
  B8 o;
#pragma unroll
  for (int i = 0; i < 8; ++i) o.v[i] = __float2bfloat16(__bfloat162float(a.v[i]) > 0.0f ? d * wh[c + i] : 0.0f);
  st8(dA + v * C + c, o);
}
// head parameter gradients: partials over blocks of 1024 voxels of
// (dy a[c], dy) in FP32, C = 16, added in the order of the voxels
__global__ void __launch_bounds__(256) k_head_bwd_par(long long V, const float *dy, const bf16 *A, int C, float *part) {
  __shared__ float row[2][SUM_ROWS * 17];
  const long long v0 = (long long)blockIdx.x * 1024, v1 = min(V, v0 + 1024);
  float s = 0.0f;
  auto fill = [&](long long v, float *to) {
    const int r = threadIdx.x >> 1, c = (threadIdx.x & 1) * 8;
    if (r >= SUM_ROWS || v + r >= v1) return;
    const float d = dy[v + r];
    const B8 a = ld8(A + (v + r) * C + c);
#pragma unroll
    for (int i = 0; i < 8; ++i) to[r * 17 + c + i] = d * __bfloat162float(a.v[i]);
    if (c == 0) to[r * 17 + 16] = d * 1.0f;
  };
  fill(v0, row[0]);
  int k = 0;
  for (long long v = v0; v < v1; v += SUM_ROWS, k ^= 1) {
    __syncthreads();
    if (v + SUM_ROWS < v1) fill(v + SUM_ROWS, row[k ^ 1]);
    if (threadIdx.x <= C) {
      const int n = (int)min((long long)SUM_ROWS, v1 - v);
#pragma unroll 8
      for (int r = 0; r < n; ++r) s += row[k][r * 17 + threadIdx.x];
    }
  }
  if (threadIdx.x <= C) part[(long long)blockIdx.x * (C + 1) + threadIdx.x] = s;
}

// ---------------------------------------------------- residual loss
// The pressure system of each sample in the network's volume: per voxel
// the 7 coefficients (AD, ALI, ALJ, ALK, AUI, AUJ, AUK, FP32) of VF_MZAX's
// row (vf_mzax.f:42-56), b = the input's channel 0 (BB/s).  With the output
// y, taken as 0 off the counted cells as the solver's guess is, and the
// fixed scale c: r = m (b - c A (m y)); loss |r|^2 / sum(m).
__device__ __forceinline__ float vget(const Vol &g, const float *a, const float *Mk, int x, int y, int z, int b,
                                      int dx, int dy, int dz) {
  const long long v = nbr(g, x, y, z, b, dx, dy, dz);
  return v >= 0 ? a[v] * Mk[v] : 0.0f;
}
__global__ void k_res_fwd(Vol g, const float *Yo, const float *A7, const float *X4, const float *Mk, float c,
                          float *R, float *lpart) {
  __shared__ float red[256];
  const long long v = (long long)blockIdx.x * 256 + threadIdx.x;
  float l = 0.0f;
  if (v < g.n()) {
    int x, y, z, b;
    decomp(g, v, x, y, z, b);
    const float *a = A7 + 7 * v;
    const float ay = a[0] * Yo[v] * Mk[v] + a[1] * vget(g, Yo, Mk, x, y, z, b, -1, 0, 0) +
                     a[2] * vget(g, Yo, Mk, x, y, z, b, 0, -1, 0) + a[3] * vget(g, Yo, Mk, x, y, z, b, 0, 0, -1) +
                     a[4] * vget(g, Yo, Mk, x, y, z, b, 1, 0, 0) + a[5] * vget(g, Yo, Mk, x, y, z, b, 0, 1, 0) +
                     a[6] * vget(g, Yo, Mk, x, y, z, b, 0, 0, 1);
    const float r = Mk[v] * (X4[4 * v] - c * ay);
    R[v] = r;
    l = r * r;
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) lpart[blockIdx.x] = red[0];
}
// dy += w * d(|r|^2 / n)/dy = -2 w c / n * m[v] (A^T r)[v]; (A^T r)[v] =
// AD[v] r[v] + the coefficients of the neighbours' rows that point at v
__global__ void k_res_bwd(Vol g, const float *A7, const float *R, const float *Mk, float scale, float *dy) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= g.n()) return;
  int x, y, z, b;
  decomp(g, v, x, y, z, b);
  auto term = [&](int dx, int dyy, int dz, int k) {
    const long long u = nbr(g, x, y, z, b, dx, dyy, dz);
    return u >= 0 ? A7[7 * u + k] * R[u] : 0.0f;
  };
  // row u = v+1 holds ALI (index 1) toward v, row v-1 holds AUI (4) ...
  const float atr = A7[7 * v] * R[v] + term(1, 0, 0, 1) + term(0, 1, 0, 2) + term(0, 0, 1, 3) + term(-1, 0, 0, 4) +
                    term(0, -1, 0, 5) + term(0, 0, -1, 6);
  dy[v] += scale * Mk[v] * atr;
}

// -------------------------------------------------------- Adam, casts
// FP32 master p, moments m, v; step t (1-based); then the BF16 copy
__global__ void k_adam(long long n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}
// weights [cout][27][cin] FP32 -> BF16 forward copy [tap][cin/8][cout][cin%8]
// and the input-gradient copy, cin and cout swapped and tap 26 - tap
__global__ void k_wcast(const float *w, int Cin, int Cout, bf16 *wf, bf16 *wt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Cout * 27 * Cin) return;
  const int ci = i % Cin, t = (i / Cin) % 27, co = i / (27 * Cin);
  const bf16 q = __float2bfloat16(w[i]);
  wf[((t * (Cin >> 3) + (ci >> 3)) * Cout + co) * 8 + (ci & 7)] = q;
  if (wt) wt[(((26 - t) * (Cout >> 3) + (co >> 3)) * Cin + ci) * 8 + (co & 7)] = q;
}
// network input: 4 FP32 channels per voxel -> 16 BF16 channels (12 zero)
__global__ void k_pack_in(long long V, const float *x4, bf16 *x16) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V * 2) return;
  B8 o;
#pragma unroll
  for (int c = 0; c < 8; ++c) o.v[c] = __float2bfloat16(0.0f);
  if ((i & 1) == 0) {
    const float4 f = *reinterpret_cast<const float4 *>(x4 + (i >> 1) * 4);
    o.v[0] = __float2bfloat16(f.x); o.v[1] = __float2bfloat16(f.y);
    o.v[2] = __float2bfloat16(f.z); o.v[3] = __float2bfloat16(f.w);
  }
  st8(x16 + i * 8, o);
}

// ------------------------------------------------------------ launchers
static inline unsigned nb(long long n, int t) { return (unsigned)((n + t - 1) / t); }

static size_t wgrad_smem_bytes(int Cout, int WG_ST) {
  return smem_floor((size_t)WG_ST * (128 + Cout) * WG_K * 2 + 64, umma::tmem_cols(Cout));
}

bool unet_kernels_configure() {
  static int done = 0;
  if (done) return done > 0;
  const int mx = 227 * 1024;
  bool ok = cudaFuncSetAttribute(k_conv, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) == cudaSuccess &&
            cudaFuncSetAttribute(k_wgrad<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) == cudaSuccess &&
            cudaFuncSetAttribute(k_wgrad<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) == cudaSuccess &&
            cudaFuncSetAttribute(k_bias_part, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) == cudaSuccess;
  done = ok ? 1 : -1;
  return ok;
}

void launch_conv(cudaStream_t s, const ConvPlan &p, int X, int Y, int Z, int B, const void *x, int Cin, const void *w,
                 const float *bias, int Cout, int mode, const void *mask, void *y, int *err) {
  const Vol g{X, Y, Z, B};
  k_conv<<<(unsigned)((long long)p.nxt * p.nyt * Z * B), CONV_T, p.smem, s>>>(
      g, (const bf16 *)x, Cin, (const bf16 *)w, bias, Cout, mode, (const bf16 *)mask, y, err, p);
  count_launch();
}
// Voxels per slice of a weight gradient.  The slices fix the order in which
// the tensor cores add (their FP32 accumulation depends on it at 1e-4 of a
// gradient), so they are the same at every size.
constexpr long long WGRAD_SLICE = 8192;
long long wgrad_slices(long long V) { return (V + WGRAD_SLICE - 1) / WGRAD_SLICE; }
void launch_wgrad(cudaStream_t s, int X, int Y, int Z, int B, const void *x, int Cin, const void *dy, int Cout,
                  float *part, float *dw, int *err) {
  const Vol g{X, Y, Z, B};
  const int ns = (int)wgrad_slices(g.n());
  dim3 grid((27 * Cin + 127) / 128, ns);
  // Where the CTAs leave the SMs half empty, eight stages (one CTA per SM)
  // hide the copies' latency; else three stages and up to four CTAs do.
  if ((long long)grid.x * grid.y <= 2 * sm_count())
    k_wgrad<8><<<grid, 128, wgrad_smem_bytes(Cout, 8), s>>>(g, (const bf16 *)x, Cin, (const bf16 *)dy, Cout, WGRAD_SLICE,
                                                            part, err);
  else
    k_wgrad<3><<<grid, 128, wgrad_smem_bytes(Cout, 3), s>>>(g, (const bf16 *)x, Cin, (const bf16 *)dy, Cout, WGRAD_SLICE,
                                                            part, err);
  k_wgrad_reduce<<<nb(27LL * Cin * Cout, 64), 64, 0, s>>>(part, ns, Cin, Cout, dw);
  count_launch(2);
}
void launch_bias_grad(cudaStream_t s, long long V, const void *dy, int C, float *part, float *db) {
  const int n = (int)nb(V, 1024);
  k_bias_part<<<n, 256, (size_t)1024 * C * 2, s>>>((const bf16 *)dy, V, C, part);
  k_bias_reduce<<<1, 256, 0, s>>>(part, n, C, db);
  count_launch(2);
}
void launch_pool(cudaStream_t s, int Xc, int Yc, int Zc, int B, const void *f, int C, void *c) {
  const Vol gc{Xc, Yc, Zc, B};
  k_pool<<<nb(gc.n() * (C / 8), 256), 256, 0, s>>>(gc, (const bf16 *)f, C, (bf16 *)c);
  count_launch();
}
void launch_pool_bwd(cudaStream_t s, int Xc, int Yc, int Zc, int B, const void *dc, int C, void *df, const void *act) {
  const Vol gc{Xc, Yc, Zc, B};
  k_pool_bwd<<<nb(gc.n() * C, 256), 256, 0, s>>>(gc, (const bf16 *)dc, C, (bf16 *)df, (const bf16 *)act);
  count_launch();
}
void launch_upcat(cudaStream_t s, int X, int Y, int Z, int B, const void *c, int C1, const void *sk, int C2, void *o) {
  const Vol gf{X, Y, Z, B};
  k_upcat<<<nb(gf.n() * ((C1 + C2) / 8), 256), 256, 0, s>>>(gf, (const bf16 *)c, C1, (const bf16 *)sk, C2, (bf16 *)o);
  count_launch();
}
void launch_upcat_bwd(cudaStream_t s, int X, int Y, int Z, int B, const void *d, int C1, int C2, void *dc, void *dsk) {
  const Vol gf{X, Y, Z, B};
  const Vol gc{X / 2, Y / 2, Z / 2, B};
  k_upcat_bwd_coarse<<<nb(gc.n() * (C1 / 8), 256), 256, 0, s>>>(gc, (const bf16 *)d, C1, C2, (bf16 *)dc);
  k_upcat_bwd_skip<<<nb(gf.n() * (C2 / 8), 256), 256, 0, s>>>(gf.n(), (const bf16 *)d, C1, C2, (bf16 *)dsk);
  count_launch(2);
}
void launch_head(cudaStream_t s, long long V, const void *a, int C, const float *wh, const float *bh, float *y) {
  k_head<<<nb(V, 256), 256, 0, s>>>(V, (const bf16 *)a, C, wh, bh, y);
  count_launch();
}
void launch_mse(cudaStream_t s, long long V, const float *y, const float *t, const float *m, float inv_n, float *dy,
                float *lpart) {
  k_mse<<<nb(V, 256), 256, 0, s>>>(V, y, t, m, inv_n, dy, lpart);
  count_launch();
}
void launch_sum(cudaStream_t s, long long n, const float *a, double *out) {
  k_sum_part<<<SUM_BLOCKS, 256, 0, s>>>(n, a, out);
  k_sum_fin<<<1, 32, 0, s>>>(out);
  count_launch(2);
}
void launch_head_bwd(cudaStream_t s, long long V, const float *dy, const void *a, int C, const float *wh, void *da,
                     float *part) {
  k_head_bwd_act<<<nb(V * (C / 8), 256), 256, 0, s>>>(V, dy, (const bf16 *)a, C, wh, (bf16 *)da);
  k_head_bwd_par<<<nb(V, 1024), 256, 0, s>>>(V, dy, (const bf16 *)a, C, part);
  count_launch(2);
}
void launch_res_fwd(cudaStream_t s, int X, int Y, int Z, int B, const float *y, const float *a7, const float *x4,
                    const float *m, float c, float *r, float *lpart) {
  const Vol g{X, Y, Z, B};
  k_res_fwd<<<nb(g.n(), 256), 256, 0, s>>>(g, y, a7, x4, m, c, r, lpart);
  count_launch();
}
void launch_res_bwd(cudaStream_t s, int X, int Y, int Z, int B, const float *a7, const float *r, const float *m,
                    float scale, float *dy) {
  const Vol g{X, Y, Z, B};
  k_res_bwd<<<nb(g.n(), 256), 256, 0, s>>>(g, a7, r, m, scale, dy);
  count_launch();
}
void launch_adam(cudaStream_t s, long long n, float *p, const float *g, float *m, float *v, float lr, float b1,
                 float b2, float eps, float c1, float c2) {
  k_adam<<<nb(n, 256), 256, 0, s>>>(n, p, g, m, v, lr, b1, b2, eps, c1, c2);
  count_launch();
}
void launch_wcast(cudaStream_t s, const float *w, int Cin, int Cout, void *wf, void *wt) {
  k_wcast<<<nb(27LL * Cin * Cout, 256), 256, 0, s>>>(w, Cin, Cout, (bf16 *)wf, (bf16 *)wt);
  count_launch();
}
void launch_pack_in(cudaStream_t s, long long V, const float *x4, void *x16) {
  k_pack_in<<<nb(V * 2, 256), 256, 0, s>>>(V, x4, (bf16 *)x16);
  count_launch();
}
void launch_bias_reduce(cudaStream_t s, const float *part, int n, int C, float *out) {
  k_bias_reduce<<<1, 256, 0, s>>>(part, n, C, out);
  count_launch();
}

}  // namespace cadmas
