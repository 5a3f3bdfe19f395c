// unet.cu -- the learned warm start's network on the host side: the layer
// table of the 3-level 3-D U-Net, its buffers, forward, backward (input and
// weight gradients of every layer), the masked MSE loss and Adam, behind the
// cadmas_unet_* entry points.
//
// Architecture (channels-last BF16 activations, FP32 master weights):
//   in 4 (+12 zero) -> c11 16 -> c12 16 (skip1) -> pool -> c21 32 ->
//   c22 32 (skip2) -> pool -> c31 64 -> c32 64 -> up + skip2 (96) ->
//   c41 32 -> c42 32 -> up + skip1 (48) -> c51 16 -> c52 16 -> head 1
// every cNN a 3x3x3 convolution with bias and ReLU, pooling 2x2x2 average,
// upsampling nearest, the head a 1x1x1 convolution with bias (FP32 out).
// Parameters (FP32, in this order): per convolution W[cout][27][cin] then
// b[cout]; then the head's 16 weights and its bias.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <thread>
#include <vector>
#include "../../include/cadmas_gpu.h"
#include "kernels.h"

using namespace cadmas;

namespace {

struct Layer {
  int cin, cout, res;
  size_t w, b;  // offsets of W and b in the parameter vector
};

constexpr int NL = 10;
const int LCH[NL][3] = {{16, 16, 0}, {16, 16, 0}, {16, 32, 1}, {32, 32, 1}, {32, 64, 2},
                        {64, 64, 2}, {96, 32, 1}, {32, 32, 1}, {48, 16, 0}, {16, 16, 0}};

struct Table {
  Layer L[NL];
  size_t head_w, head_b, n;
  Table() {
    size_t o = 0;
    for (int l = 0; l < NL; ++l) {
      L[l] = Layer{LCH[l][0], LCH[l][1], LCH[l][2], o, o + (size_t)27 * LCH[l][0] * LCH[l][1]};
      o = L[l].b + LCH[l][1];
    }
    head_w = o;
    head_b = o + 16;
    n = o + 17;
  }
};
const Table TAB;

template <class T>
int dmalloc(T **p, size_t n) {
  return cudaMalloc((void **)p, (n ? n : 1) * sizeof(T)) == cudaSuccess ? CADMAS_OK : CADMAS_ENOMEM;
}

// Upload threads, bytes per pinned chunk, and the pageable bytes from which
// they are used.  The driver's own staging of pageable memory is one
// thread's memcpy: the 67 MB of a training step on four 132x36x68 volumes
// took 6 ms of a step's 12.1, 6.6 with the threads; for the 5 MB of one
// volume's forward starting the threads costs more (1.14 against 0.97 ms).
constexpr int UP_T = 4;
constexpr size_t UP_CHUNK = 512 << 10, UP_MIN = 16 << 20;

}  // namespace

struct cadmas_unet {
  cudaStream_t s = nullptr;
  bool own_stream = true;
  int X = 0, Y = 0, Z = 0, B = 0;
  long long V[3] = {0, 0, 0};
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  long long step = 0;
  void *wf[NL] = {}, *wt[NL] = {};
  ConvPlan pf[NL] = {}, pt[NL] = {};  // tilings of layer l's convolution and of its input gradient
  // activations (BF16) and their gradients
  void *xin = nullptr, *a[NL] = {}, *p1 = nullptr, *p2 = nullptr, *u2 = nullptr, *u1 = nullptr;
  void *d[NL] = {}, *du2 = nullptr, *du1 = nullptr, *dp1 = nullptr, *dp2 = nullptr;
  float *x4 = nullptr, *y = nullptr, *t = nullptr, *mk = nullptr, *dy = nullptr;
  float *part = nullptr, *bpart = nullptr, *lpart = nullptr;
  float *a7 = nullptr, *r = nullptr;  // pressure systems and residual (residual loss)
  size_t part_n = 0;
  int *err = nullptr;
  std::vector<float> hl;
  // Host arrays come through pinned chunks on a stream of their own, filled
  // by a few threads; allocated by the first upload that is large enough.
  cudaStream_t sc = nullptr;
  cudaEvent_t up = nullptr;                  // the last upload has arrived
  unsigned char *pin = nullptr;              // UP_T x 2 chunks
  cudaEvent_t pin_ev[UP_T][2] = {};          // a chunk's last copy has been made
  double *cnt = nullptr, *cnt_h = nullptr;   // sum of the mask: partials and result, pinned copy
};

namespace {

void dims(const cadmas_unet *n, int res, int &X, int &Y, int &Z) {
  X = n->X >> res;
  Y = n->Y >> res;
  Z = n->Z >> res;
}

// convolution of layer l with ReLU
void conv(cadmas_unet *n, int l, const void *x) {
  const Layer &L = TAB.L[l];
  int X, Y, Z;
  dims(n, L.res, X, Y, Z);
  launch_conv(n->s, n->pf[l], X, Y, Z, n->B, x, L.cin, n->wf[l], n->p + L.b, L.cout, CONV_RELU_BF16, nullptr, n->a[l],
              n->err);
}
// its input gradient, times the ReLU derivative of the layer below where
// `mask` gives that layer's activations
void conv_t(cadmas_unet *n, int l, const void *mask, void *dx) {
  const Layer &L = TAB.L[l];
  int X, Y, Z;
  dims(n, L.res, X, Y, Z);
  launch_conv(n->s, n->pt[l], X, Y, Z, n->B, n->d[l], L.cout, n->wt[l], nullptr, L.cin, mask ? CONV_MASK_BF16 : CONV_BF16,
              mask, dx, n->err);
}

void cast_weights(cadmas_unet *n) {
  for (int l = 0; l < NL; ++l)
    launch_wcast(n->s, n->p + TAB.L[l].w, TAB.L[l].cin, TAB.L[l].cout, n->wf[l], l > 0 ? n->wt[l] : nullptr);
}

int check(cadmas_unet *n) {
  int e = 0;
  if (cudaMemcpyAsync(&e, n->err, sizeof(int), cudaMemcpyDeviceToHost, n->s) != cudaSuccess) return CADMAS_ECUDA;
  if (cudaStreamSynchronize(n->s) != cudaSuccess) return CADMAS_ECUDA;
  if (cudaGetLastError() != cudaSuccess) return CADMAS_ECUDA;
  return e ? CADMAS_ETIMEOUT : CADMAS_OK;
}

// The end of an entry point: after an error, waits for what is still queued,
// so that nothing reads or writes the caller's arrays any more.
int leave(cadmas_unet *n, int rc) {
  if (rc) {
    cudaStreamSynchronize(n->sc);
    cudaStreamSynchronize(n->s);
  }
  return rc;
}

// forward of the batch in n->x4 (FP32, 4 channels) to n->y
void forward(cadmas_unet *n) {
  launch_pack_in(n->s, n->V[0], n->x4, n->xin);
  conv(n, 0, n->xin);
  conv(n, 1, n->a[0]);
  launch_pool(n->s, n->X / 2, n->Y / 2, n->Z / 2, n->B, n->a[1], 16, n->p1);
  conv(n, 2, n->p1);
  conv(n, 3, n->a[2]);
  launch_pool(n->s, n->X / 4, n->Y / 4, n->Z / 4, n->B, n->a[3], 32, n->p2);
  conv(n, 4, n->p2);
  conv(n, 5, n->a[4]);
  launch_upcat(n->s, n->X / 2, n->Y / 2, n->Z / 2, n->B, n->a[5], 64, n->a[3], 32, n->u2);
  conv(n, 6, n->u2);
  conv(n, 7, n->a[6]);
  launch_upcat(n->s, n->X, n->Y, n->Z, n->B, n->a[7], 32, n->a[1], 16, n->u1);
  conv(n, 8, n->u1);
  conv(n, 9, n->a[8]);
  launch_head(n->s, n->V[0], n->a[9], 16, n->p + TAB.head_w, n->p + TAB.head_b, n->y);
}

// weight and bias gradients of layer l from its input x and output grad dyl
void layer_grads(cadmas_unet *n, int l, const void *x, const void *dyl) {
  const Layer &L = TAB.L[l];
  int X, Y, Z;
  dims(n, L.res, X, Y, Z);
  launch_wgrad(n->s, X, Y, Z, n->B, x, L.cin, dyl, L.cout, n->part, n->g + L.w, n->err);
  launch_bias_grad(n->s, n->V[L.res], dyl, L.cout, n->bpart, n->g + L.b);
}

// backward from n->dy (FP32 loss gradient of the output) into n->g
void backward(cadmas_unet *n) {
  const int nbh = (int)((n->V[0] + 1023) / 1024);
  launch_head_bwd(n->s, n->V[0], n->dy, n->a[9], 16, n->p + TAB.head_w, n->d[9], n->bpart);
  launch_bias_reduce(n->s, n->bpart, nbh, 17, n->g + TAB.head_w);
  // c52, c51
  layer_grads(n, 9, n->a[8], n->d[9]);
  conv_t(n, 9, n->a[8], n->d[8]);
  layer_grads(n, 8, n->u1, n->d[8]);
  conv_t(n, 8, n->u1, n->du1);
  // split: d of c42's output (coarse, 32) and of skip1 (16)
  launch_upcat_bwd(n->s, n->X, n->Y, n->Z, n->B, n->du1, 32, 16, n->d[7], n->d[1]);
  // c42, c41
  layer_grads(n, 7, n->a[6], n->d[7]);
  conv_t(n, 7, n->a[6], n->d[6]);
  layer_grads(n, 6, n->u2, n->d[6]);
  conv_t(n, 6, n->u2, n->du2);
  launch_upcat_bwd(n->s, n->X / 2, n->Y / 2, n->Z / 2, n->B, n->du2, 64, 32, n->d[5], n->d[3]);
  // c32, c31
  layer_grads(n, 5, n->a[4], n->d[5]);
  conv_t(n, 5, n->a[4], n->d[4]);
  layer_grads(n, 4, n->p2, n->d[4]);
  conv_t(n, 4, nullptr, n->dp2);
  // skip2 gets the pooled path too, then the ReLU of c22
  launch_pool_bwd(n->s, n->X / 4, n->Y / 4, n->Z / 4, n->B, n->dp2, 32, n->d[3], n->a[3]);
  // c22, c21
  layer_grads(n, 3, n->a[2], n->d[3]);
  conv_t(n, 3, n->a[2], n->d[2]);
  layer_grads(n, 2, n->p1, n->d[2]);
  conv_t(n, 2, nullptr, n->dp1);
  launch_pool_bwd(n->s, n->X / 2, n->Y / 2, n->Z / 2, n->B, n->dp1, 16, n->d[1], n->a[1]);
  // c12, c11
  layer_grads(n, 1, n->a[0], n->d[1]);
  conv_t(n, 1, n->a[0], n->d[0]);
  layer_grads(n, 0, n->xin, n->d[0]);
}

struct Piece {
  void *dst;
  const void *src;
  size_t bytes;
};

bool upload_setup(cadmas_unet *n) {
  if (!n->pin && cudaMallocHost((void **)&n->pin, UP_T * 2 * UP_CHUNK) != cudaSuccess) n->pin = nullptr;
  bool ok = n->pin != nullptr;
  for (auto &t : n->pin_ev)
    for (cudaEvent_t &e : t)
      if (ok && !e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        e = nullptr;
        ok = false;
      }
  if (!ok) cudaGetLastError();  // the caller copies without them
  return ok;
}

// Whether the launches since the last look went through: looked at before
// anything that may clear the runtime's last error.
int launched() { return cudaGetLastError() == cudaSuccess ? CADMAS_OK : CADMAS_ECUDA; }

// Host arrays to the device on the upload stream; n->s waits for them.  It
// may clear the runtime's last error.
// Small or pinned arrays go straight; pageable ones in chunks through the
// pinned buffers.  Returns when the arrays have been read or the copies of
// the pinned ones are queued (the entry points wait for them before they
// return to the arrays' owner: check(), and leave() after an error).
int upload(cadmas_unet *n, std::initializer_list<Piece> pieces) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return CADMAS_ECUDA;
  std::vector<Piece> chunks;
  size_t total = 0;
  for (const Piece &p : pieces) total += p.bytes;
  for (const Piece &p : pieces) {
    bool straight = total < UP_MIN;
    if (!straight) {
      cudaPointerAttributes at{};
      if (cudaPointerGetAttributes(&at, p.src) == cudaSuccess) straight = at.type != cudaMemoryTypeUnregistered;
      else cudaGetLastError();  // plain memory, to older drivers
    }
    if (straight) {
      if (cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyHostToDevice, n->sc) != cudaSuccess) return CADMAS_ECUDA;
      continue;
    }
    for (size_t o = 0; o < p.bytes; o += UP_CHUNK)
      chunks.push_back({(char *)p.dst + o, (const char *)p.src + o, std::min(UP_CHUNK, p.bytes - o)});
  }
  if (!chunks.empty() && !upload_setup(n)) {  // no pinned memory to be had: as the small arrays
    for (const Piece &c : chunks)
      if (cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyHostToDevice, n->sc) != cudaSuccess) return CADMAS_ECUDA;
    chunks.clear();
  }
  if (!chunks.empty()) {
    std::atomic<size_t> next{0};
    std::atomic<bool> bad{false};
    auto work = [&](int t) {
      if (t > 0 && cudaSetDevice(dev) != cudaSuccess) { bad = true; return; }
      for (int k = 0; !bad; k ^= 1) {
        const size_t c = next.fetch_add(1);
        if (c >= chunks.size()) return;
        unsigned char *buf = n->pin + (size_t)(2 * t + k) * UP_CHUNK;
        if (cudaEventSynchronize(n->pin_ev[t][k]) != cudaSuccess) { bad = true; return; }
        std::memcpy(buf, chunks[c].src, chunks[c].bytes);
        if (cudaMemcpyAsync(chunks[c].dst, buf, chunks[c].bytes, cudaMemcpyHostToDevice, n->sc) != cudaSuccess ||
            cudaEventRecord(n->pin_ev[t][k], n->sc) != cudaSuccess) { bad = true; return; }
      }
    };
    const int nt = (int)std::min<size_t>(UP_T, chunks.size());
    std::vector<std::thread> pool;
    int started = 1;
    try {
      for (; started < nt; ++started) pool.emplace_back(work, started);
    } catch (...) {}  // fewer threads do the same work
    work(0);
    for (std::thread &t : pool) t.join();
    if (bad) return CADMAS_ECUDA;
  }
  if (cudaEventRecord(n->up, n->sc) != cudaSuccess || cudaStreamWaitEvent(n->s, n->up, 0) != cudaSuccess)
    return CADMAS_ECUDA;
  return CADMAS_OK;
}

// 1 / (counted cells) of the mask just uploaded: summed on the upload
// stream, beside the forward that runs on n->s
int mask_inv(cadmas_unet *n, double &inv) {
  launch_sum(n->sc, n->V[0], n->mk, n->cnt);
  if (cudaMemcpyAsync(n->cnt_h, n->cnt, sizeof(double), cudaMemcpyDeviceToHost, n->sc) != cudaSuccess ||
      cudaStreamSynchronize(n->sc) != cudaSuccess)
    return CADMAS_ECUDA;
  inv = *n->cnt_h > 0.0 ? 1.0 / *n->cnt_h : 0.0;
  return CADMAS_OK;
}

// Sums of the per-block loss partials, k blocks of them, each in order.
int lsum(cadmas_unet *n, int k, double *out) {
  const int nbk = (int)((n->V[0] + 255) / 256);
  n->hl.resize((size_t)k * nbk);
  if (cudaMemcpyAsync(n->hl.data(), n->lpart, n->hl.size() * sizeof(float), cudaMemcpyDeviceToHost, n->s) != cudaSuccess)
    return CADMAS_ECUDA;
  if (cudaStreamSynchronize(n->s) != cudaSuccess) return CADMAS_ECUDA;
  for (int i = 0; i < k; ++i) {
    out[i] = 0.0;
    for (int j = 0; j < nbk; ++j) out[i] += n->hl[(size_t)i * nbk + j];
  }
  return CADMAS_OK;
}

}  // namespace

extern "C" {

size_t cadmas_unet_param_count(void) { return TAB.n; }

int cadmas_unet_destroy(cadmas_unet *n) {
  if (!n) return CADMAS_OK;
  for (float *q : {n->p, n->g, n->m, n->v, n->x4, n->y, n->t, n->mk, n->dy, n->part, n->bpart, n->lpart, n->a7, n->r})
    if (q) cudaFree(q);
  if (n->cnt) cudaFree(n->cnt);
  if (n->sc) cudaStreamSynchronize(n->sc);
  if (n->cnt_h) cudaFreeHost(n->cnt_h);
  if (n->pin) cudaFreeHost(n->pin);
  for (auto &t : n->pin_ev)
    for (cudaEvent_t e : t) if (e) cudaEventDestroy(e);
  if (n->up) cudaEventDestroy(n->up);
  if (n->sc) cudaStreamDestroy(n->sc);
  for (int l = 0; l < NL; ++l)
    for (void *q : {n->wf[l], n->wt[l], n->a[l], n->d[l]})
      if (q) cudaFree(q);
  for (void *q : {n->xin, n->p1, n->p2, n->u2, n->u1, n->du2, n->du1, n->dp1, n->dp2})
    if (q) cudaFree(q);
  if (n->err) cudaFree(n->err);
  if (n->s && n->own_stream) cudaStreamDestroy(n->s);
  delete n;
  return CADMAS_OK;
}

int cadmas_unet_create(int nx, int ny, int nz, int batch, cadmas_unet **out) {
  return cadmas::unet_new(nx, ny, nz, batch, nullptr, out);
}

}  // extern "C"

namespace cadmas {

// A network on the given stream (its own stream when null).
int unet_new(int nx, int ny, int nz, int batch, cudaStream_t stream, cadmas_unet **out) {
  if (!out || nx < 4 || ny < 4 || nz < 4 || batch < 1 || nx % 4 || ny % 4 || nz % 4) return CADMAS_EINVAL;
  if (!unet_kernels_configure()) return CADMAS_ECUDA;
  cadmas_unet *n = new cadmas_unet();
  n->X = nx; n->Y = ny; n->Z = nz; n->B = batch;
  for (int l = 0; l < NL; ++l) {
    const Layer &L = TAB.L[l];
    n->pf[l] = conv_plan(nx >> L.res, ny >> L.res, L.cin, L.cout);
    if (l > 0) n->pt[l] = conv_plan(nx >> L.res, ny >> L.res, L.cout, L.cin);
    if (n->pf[l].MT == 0 || (l > 0 && n->pt[l].MT == 0)) {
      delete n;
      return CADMAS_EUNSUPPORTED;
    }
  }
  for (int r = 0; r < 3; ++r) n->V[r] = (long long)(nx >> r) * (ny >> r) * (nz >> r) * batch;
  int rc = CADMAS_OK;
  if (stream) {
    n->s = stream;
    n->own_stream = false;
  } else if (cudaStreamCreateWithFlags(&n->s, cudaStreamNonBlocking) != cudaSuccess) {
    rc = CADMAS_ECUDA;
  }
  const size_t P = TAB.n;
#define AL(ptr, cnt) if (!rc) rc = dmalloc(&(ptr), (cnt))
  AL(n->p, P); AL(n->g, P); AL(n->m, P); AL(n->v, P);
  using u16 = unsigned short;
  for (int l = 0; l < NL; ++l) {
    const size_t w = (size_t)27 * TAB.L[l].cin * TAB.L[l].cout;
    AL(*(u16 **)&n->wf[l], w);
    if (l > 0) AL(*(u16 **)&n->wt[l], w);
    AL(*(u16 **)&n->a[l], (size_t)n->V[TAB.L[l].res] * TAB.L[l].cout);
    AL(*(u16 **)&n->d[l], (size_t)n->V[TAB.L[l].res] * TAB.L[l].cout);
  }
  AL(*(u16 **)&n->xin, (size_t)n->V[0] * 16);
  AL(*(u16 **)&n->p1, (size_t)n->V[1] * 16); AL(*(u16 **)&n->dp1, (size_t)n->V[1] * 16);
  AL(*(u16 **)&n->p2, (size_t)n->V[2] * 32); AL(*(u16 **)&n->dp2, (size_t)n->V[2] * 32);
  AL(*(u16 **)&n->u2, (size_t)n->V[1] * 96); AL(*(u16 **)&n->du2, (size_t)n->V[1] * 96);
  AL(*(u16 **)&n->u1, (size_t)n->V[0] * 48); AL(*(u16 **)&n->du1, (size_t)n->V[0] * 48);
  AL(n->x4, (size_t)n->V[0] * 4); AL(n->y, (size_t)n->V[0]); AL(n->t, (size_t)n->V[0]);
  AL(n->mk, (size_t)n->V[0]); AL(n->dy, (size_t)n->V[0]);
  // wgrad partial sums: the largest (slices x 27 Cin x Cout) of any layer
  for (int l = 0; l < NL; ++l) {
    const long long ns = wgrad_slices(n->V[TAB.L[l].res]);
    n->part_n = std::max(n->part_n, (size_t)ns * 27 * TAB.L[l].cin * TAB.L[l].cout);
  }
  AL(n->part, n->part_n);
  AL(n->bpart, (size_t)((n->V[0] + 1023) / 1024) * 128);
  AL(n->lpart, 2 * (size_t)((n->V[0] + 255) / 256));
  AL(n->cnt, (size_t)1 + SUM_BLOCKS);
  if (!rc && cudaMalloc((void **)&n->err, sizeof(int)) != cudaSuccess) rc = CADMAS_ENOMEM;
  if (!rc && cudaMallocHost((void **)&n->cnt_h, sizeof(double)) != cudaSuccess) rc = CADMAS_ENOMEM;
  if (!rc && cudaStreamCreateWithFlags(&n->sc, cudaStreamNonBlocking) != cudaSuccess) rc = CADMAS_ECUDA;
  if (!rc && cudaEventCreateWithFlags(&n->up, cudaEventDisableTiming) != cudaSuccess) rc = CADMAS_ECUDA;
#undef AL
  if (rc) { cadmas_unet_destroy(n); return rc; }
  cudaMemsetAsync(n->err, 0, sizeof(int), n->s);
  cudaMemsetAsync(n->p, 0, P * sizeof(float), n->s);
  cudaMemsetAsync(n->m, 0, P * sizeof(float), n->s);
  cudaMemsetAsync(n->v, 0, P * sizeof(float), n->s);
  cast_weights(n);
  if (cudaStreamSynchronize(n->s) != cudaSuccess) { cadmas_unet_destroy(n); return CADMAS_ECUDA; }
  *out = n;
  return CADMAS_OK;
}

void unet_dims(const cadmas_unet *n, int &X, int &Y, int &Z) { X = n->X; Y = n->Y; Z = n->Z; }
float *unet_input(cadmas_unet *n) { return n->x4; }
const float *unet_output(const cadmas_unet *n) { return n->y; }
const int *unet_error(const cadmas_unet *n) { return n->err; }
void unet_run_forward(cadmas_unet *n) { forward(n); }
int unet_error_host(cadmas_unet *n) { return check(n); }

}  // namespace cadmas

static int set_params(cadmas_unet *n, const float *p) {
  if (cudaMemcpyAsync(n->p, p, TAB.n * sizeof(float), cudaMemcpyHostToDevice, n->s) != cudaSuccess)
    return CADMAS_ECUDA;
  cudaMemsetAsync(n->m, 0, TAB.n * sizeof(float), n->s);
  cudaMemsetAsync(n->v, 0, TAB.n * sizeof(float), n->s);
  n->step = 0;
  cast_weights(n);
  return check(n);
}

static int get_params(cadmas_unet *n, float *p) {
  if (cudaMemcpyAsync(p, n->p, TAB.n * sizeof(float), cudaMemcpyDeviceToHost, n->s) != cudaSuccess)
    return CADMAS_ECUDA;
  return check(n);
}

static int forward_host(cadmas_unet *n, const float *x, float *y) {
  int rc = upload(n, {{n->x4, x, n->V[0] * 4 * sizeof(float)}});
  if (rc) return rc;
  forward(n);
  if (cudaMemcpyAsync(y, n->y, n->V[0] * sizeof(float), cudaMemcpyDeviceToHost, n->s) != cudaSuccess)
    return CADMAS_ECUDA;
  return check(n);
}

static int time_forward(cadmas_unet *n, int reps, float *ms) {
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return CADMAS_ECUDA;
  cudaEventRecord(e0, n->s);
  for (int r = 0; r < reps; ++r) forward(n);
  cudaEventRecord(e1, n->s);
  int rc = check(n);
  float t = 0.0f;
  if (!rc && cudaEventElapsedTime(&t, e0, e1) != cudaSuccess) rc = CADMAS_ECUDA;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms = t / reps;
  return rc;
}

static int grad_host(cadmas_unet *n, const float *x, const float *t, const float *m, float *loss, float *grad) {
  const long long V = n->V[0];
  int rc = upload(n, {{n->x4, x, V * 4 * sizeof(float)}});
  if (rc) return rc;
  forward(n);
  double cnt_inv = 0.0, l = 0.0;
  if ((rc = launched()) ||
      (rc = upload(n, {{n->t, t, V * sizeof(float)}, {n->mk, m, V * sizeof(float)}})) ||
      (rc = mask_inv(n, cnt_inv)))
    return rc;
  const float inv = (float)cnt_inv;
  launch_mse(n->s, V, n->y, n->t, n->mk, inv, n->dy, n->lpart);
  backward(n);
  if ((rc = lsum(n, 1, &l))) return rc;
  *loss = (float)(l * inv);
  if (grad && cudaMemcpyAsync(grad, n->g, TAB.n * sizeof(float), cudaMemcpyDeviceToHost, n->s) != cudaSuccess)
    return CADMAS_ECUDA;
  return check(n);
}

static int train_sys(cadmas_unet *n, const float *x, const float *t, const float *m, const float *a7, float c,
                     float w_mse, float w_res, float lr, int update, float *loss, float *grad) {
  const long long V = n->V[0];
  if (!n->a7 && (dmalloc(&n->a7, (size_t)V * 7) || dmalloc(&n->r, (size_t)V))) return CADMAS_ENOMEM;
  // the forward runs while the targets, masks and systems come
  int rc = upload(n, {{n->x4, x, V * 4 * sizeof(float)}});
  if (rc) return rc;
  forward(n);
  double inv = 0.0, l[2];
  if ((rc = launched()) ||
      (rc = upload(n, {{n->mk, m, V * sizeof(float)}, {n->t, t, V * sizeof(float)}, {n->a7, a7, V * 7 * sizeof(float)}})) ||
      (rc = mask_inv(n, inv)))
    return rc;
  // mean-square error of y against t, weighted by w_mse in the gradient;
  // residual |m (b - c A y)|^2 / n, weighted by w_res
  launch_mse(n->s, V, n->y, n->t, n->mk, (float)(inv * w_mse), n->dy, n->lpart);
  launch_res_fwd(n->s, n->X, n->Y, n->Z, n->B, n->y, n->a7, n->x4, n->mk, c, n->r, n->lpart + (V + 255) / 256);
  launch_res_bwd(n->s, n->X, n->Y, n->Z, n->B, n->a7, n->r, n->mk, (float)(-2.0 * c * w_res * inv), n->dy);
  backward(n);
  if ((rc = lsum(n, 2, l))) return rc;
  const double lm = l[0], lr2 = l[1];
  *loss = (float)(w_mse * lm * inv + w_res * lr2 * inv);
  if (grad && cudaMemcpyAsync(grad, n->g, TAB.n * sizeof(float), cudaMemcpyDeviceToHost, n->s) != cudaSuccess)
    return CADMAS_ECUDA;
  if (update) {
    n->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, (float)n->step), c2 = 1.0f - std::pow(b2, (float)n->step);
    launch_adam(n->s, (long long)TAB.n, n->p, n->g, n->m, n->v, lr, b1, b2, 1.0e-8f, c1, c2);
    cast_weights(n);
  }
  return check(n);
}

static int train_step(cadmas_unet *n, const float *x, const float *t, const float *m, float lr, float *loss) {
  int rc = grad_host(n, x, t, m, loss, nullptr);
  if (rc) return rc;
  n->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - std::pow(b1, (float)n->step), c2 = 1.0f - std::pow(b2, (float)n->step);
  launch_adam(n->s, (long long)TAB.n, n->p, n->g, n->m, n->v, lr, b1, b2, 1.0e-8f, c1, c2);
  cast_weights(n);
  return check(n);
}

extern "C" {

int cadmas_unet_set_params(cadmas_unet *n, const float *p) {
  return n && p ? leave(n, set_params(n, p)) : CADMAS_EINVAL;
}

int cadmas_unet_get_params(cadmas_unet *n, float *p) { return n && p ? leave(n, get_params(n, p)) : CADMAS_EINVAL; }

int cadmas_unet_forward(cadmas_unet *n, const float *x, float *y) {
  return n && x && y ? leave(n, forward_host(n, x, y)) : CADMAS_EINVAL;
}

int cadmas_unet_time_forward(cadmas_unet *n, int reps, float *ms) {
  return n && reps >= 1 && ms ? leave(n, time_forward(n, reps, ms)) : CADMAS_EINVAL;
}

int cadmas_unet_grad(cadmas_unet *n, const float *x, const float *t, const float *m, float *loss, float *grad) {
  return n && x && t && m && loss ? leave(n, grad_host(n, x, t, m, loss, grad)) : CADMAS_EINVAL;
}

int cadmas_unet_train_sys(cadmas_unet *n, const float *x, const float *t, const float *m, const float *a7, float c,
                          float w_mse, float w_res, float lr, int update, float *loss, float *grad) {
  if (!n || !x || !t || !m || !a7 || !loss || !(c > 0.0f)) return CADMAS_EINVAL;
  return leave(n, train_sys(n, x, t, m, a7, c, w_mse, w_res, lr, update, loss, grad));
}

int cadmas_unet_train_step(cadmas_unet *n, const float *x, const float *t, const float *m, float lr, float *loss) {
  return n && x && t && m && loss ? leave(n, train_step(n, x, t, m, lr, loss)) : CADMAS_EINVAL;
}

}  // extern "C"
