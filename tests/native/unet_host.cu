// Host check of the network's entry points (unet.cu) against a stand-in for
// the CUDA runtime: streams count the work queued on them, copies are made at
// once, kernels do nothing, and one call after another is made to fail.
//   launch   a launch that fails, in the forward or in the backward, is reported
//   runtime  so is a runtime call that fails; and when an entry point returns,
//            with an error or not, none of the caller's arrays is in use any
//            more: nothing is queued on either stream
// Prints the number of failures.
#include "kernels.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

namespace fake {
struct Stream { long long last = 0, done = 0, waits = 0; };  // waits: what this stream waits for on the other one
Stream st[3];                                                // by handle 1, 2
int nstream = 0;
std::mutex mu;
cudaError_t last_error = cudaSuccess;
long long calls = 0, fail_at = -1, launches = 0, fail_launch = -1;
bool failed = false, attr_error = false, ignorable = false;
Stream &of(cudaStream_t s) { return st[(size_t)s]; }
struct Event { Stream *s; long long seq; };
// every call that may fail; `harmless`: the code goes on without it
bool bad(bool harmless = false) {
  std::lock_guard<std::mutex> l(mu);
  if (calls++ != fail_at) return false;
  failed = true;
  ignorable = harmless;
  last_error = cudaErrorUnknown;
  return true;
}
cudaError_t queue(cudaStream_t s, bool harmless = false) {
  if (bad(harmless)) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(mu);
  ++of(s).last;
  return cudaSuccess;
}
void launch(cudaStream_t s) {
  std::lock_guard<std::mutex> l(mu);
  if (launches++ == fail_launch) { failed = true; last_error = cudaErrorInvalidConfiguration; return; }
  ++of(s).last;
}
cudaError_t Malloc(void **p, size_t n) { *p = calloc(1, n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t MallocHost(void **p, size_t n, bool harmless = true) {
  if (bad(harmless)) return cudaErrorMemoryAllocation;
  return Malloc(p, n);
}
cudaError_t Free(void *p) { free(p); return cudaSuccess; }
cudaError_t MemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t q) {
  const cudaError_t e = queue(q);
  if (e == cudaSuccess) memcpy(d, s, n);
  return e;
}
cudaError_t MemsetAsync(void *d, int v, size_t n, cudaStream_t q) {
  const cudaError_t e = queue(q);
  if (e == cudaSuccess) memset(d, v, n);
  return e;
}
cudaError_t StreamCreate(cudaStream_t *s, unsigned) { *s = (cudaStream_t)(size_t)++nstream; of(*s) = Stream{}; return cudaSuccess; }
cudaError_t StreamSync(cudaStream_t s) {
  if (bad()) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(mu);
  Stream &a = of(s), &b = st[3 - (size_t)s];
  a.done = a.last;
  if (a.waits > b.done) b.done = a.waits;
  return cudaSuccess;
}
cudaError_t StreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t EventCreate(cudaEvent_t *e, unsigned = 0) {
  if (bad(true)) return cudaErrorUnknown;
  *e = (cudaEvent_t) new Event{nullptr, 0};
  return cudaSuccess;
}
cudaError_t EventDestroy(cudaEvent_t e) { delete (Event *)e; return cudaSuccess; }
cudaError_t EventRecord(cudaEvent_t e, cudaStream_t s) {
  if (bad()) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(mu);
  *(Event *)e = Event{&of(s), of(s).last};
  return cudaSuccess;
}
cudaError_t EventSync(cudaEvent_t e) {
  if (bad()) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(mu);
  Event &v = *(Event *)e;
  if (v.s && v.s->done < v.seq) v.s->done = v.seq;
  return cudaSuccess;
}
cudaError_t EventElapsed(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return bad() ? cudaErrorUnknown : cudaSuccess; }
cudaError_t StreamWait(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (bad()) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(mu);
  of(s).waits = ((Event *)e)->seq;
  return cudaSuccess;
}
cudaError_t GetLast() {
  std::lock_guard<std::mutex> l(mu);
  const cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}
cudaError_t PtrAttr(cudaPointerAttributes *a, const void *) {
  *a = cudaPointerAttributes{};
  a->type = cudaMemoryTypeUnregistered;
  if (attr_error) {
    std::lock_guard<std::mutex> l(mu);
    last_error = cudaErrorInvalidValue;
    return cudaErrorInvalidValue;
  }
  return bad(true) ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t GetDevice(int *d) { *d = 0; return bad() ? cudaErrorUnknown : cudaSuccess; }
cudaError_t SetDevice(int) { return bad() ? cudaErrorUnknown : cudaSuccess; }
bool idle() { return st[1].last == st[1].done && st[2].last == st[2].done; }
}  // namespace fake

namespace cadmas {
std::atomic<long long> g_kernel_launches{0};
#define L(name, ...) void name(cudaStream_t s, __VA_ARGS__) { fake::launch(s); }
using ll = long long;
using cp = const void *;
using cf = const float *;
L(launch_conv, const ConvPlan &, int, int, int, int, cp, int, cp, cf, int, int, cp, void *, int *)
L(launch_wgrad, int, int, int, int, cp, int, cp, int, float *, float *, int *)
L(launch_bias_grad, ll, cp, int, float *, float *)
L(launch_pool, int, int, int, int, cp, int, void *)
L(launch_pool_bwd, int, int, int, int, cp, int, void *, cp)
L(launch_upcat, int, int, int, int, cp, int, cp, int, void *)
L(launch_upcat_bwd, int, int, int, int, cp, int, int, void *, void *)
L(launch_head, ll, cp, int, cf, cf, float *)
L(launch_mse, ll, cf, cf, cf, float, float *, float *)
L(launch_sum, ll, cf, double *)
L(launch_head_bwd, ll, cf, cp, int, cf, void *, float *)
L(launch_adam, ll, float *, cf, float *, float *, float, float, float, float, float, float)
L(launch_wcast, cf, int, int, void *, void *)
L(launch_pack_in, ll, cf, void *)
L(launch_res_fwd, int, int, int, int, cf, cf, cf, cf, float, float *, float *)
L(launch_res_bwd, int, int, int, int, cf, cf, cf, float, float *)
L(launch_bias_reduce, cf, int, int, float *)
#undef L
bool unet_kernels_configure() { return true; }
long long wgrad_slices(long long V) { return (V + 8191) / 8192; }
}  // namespace cadmas

#define cudaMalloc fake::Malloc
#define cudaMallocHost fake::MallocHost
#define cudaFree fake::Free
#define cudaFreeHost fake::Free
#define cudaMemcpyAsync fake::MemcpyAsync
#define cudaMemsetAsync fake::MemsetAsync
#define cudaStreamCreateWithFlags fake::StreamCreate
#define cudaStreamSynchronize fake::StreamSync
#define cudaStreamDestroy fake::StreamDestroy
#define cudaStreamWaitEvent fake::StreamWait
#define cudaEventCreate fake::EventCreate
#define cudaEventCreateWithFlags fake::EventCreate
#define cudaEventDestroy fake::EventDestroy
#define cudaEventRecord fake::EventRecord
#define cudaEventSynchronize fake::EventSync
#define cudaEventElapsedTime fake::EventElapsed
#define cudaGetLastError fake::GetLast
#define cudaGetDevice fake::GetDevice
#define cudaSetDevice fake::SetDevice
#define cudaPointerGetAttributes fake::PtrAttr
#include "unet.cu"

static long long fails = 0, checks = 0;
static const char *names[] = {"forward", "grad", "train_step", "train_sys", "set_params", "time_forward"};
static void check(bool c, const char *what, int entry, long long at) {
  ++checks;
  if (!c && fails++ < 20) printf("%s: %s, %lld\n", what, names[entry], at);
}
static std::vector<float> hx, ht, hm, ha, hy, hg, hp;

// one call of an entry point on a network of its own, the fail-th runtime call
// or launch from there failing; true if that many were reached
static bool one(int X, int Y, int Z, int entry, long long fail, bool launch) {
  using namespace fake;
  nstream = 0;
  fail_at = fail_launch = -1;
  cadmas_unet *n = nullptr;
  if (cadmas_unet_create(X, Y, Z, 1, &n) != CADMAS_OK) { check(false, "create", entry, fail); return false; }
  calls = launches = 0;
  failed = ignorable = false;
  last_error = cudaSuccess;
  (launch ? fail_launch : fail_at) = fail;
  float loss = 0.0f;
  int rc = -1;
  switch (entry) {
    case 0: rc = cadmas_unet_forward(n, hx.data(), hy.data()); break;
    case 1: rc = cadmas_unet_grad(n, hx.data(), ht.data(), hm.data(), &loss, hg.data()); break;
    case 2: rc = cadmas_unet_train_step(n, hx.data(), ht.data(), hm.data(), 1e-3f, &loss); break;
    case 3: rc = cadmas_unet_train_sys(n, hx.data(), ht.data(), hm.data(), ha.data(), 1.0f, 0.1f, 1.0f, 1e-3f, 1, &loss, hg.data()); break;
    case 4: rc = cadmas_unet_set_params(n, hp.data()); break;
    case 5: rc = cadmas_unet_time_forward(n, 2, &loss); break;
  }
  const bool reached = failed;
  if (reached && !ignorable) check(rc != CADMAS_OK, launch ? "launch error lost" : "runtime error lost", entry, fail);
  if (!reached) check(rc == CADMAS_OK, "error without a cause", entry, fail);
  if (!launch) check(idle(), "work still queued on return", entry, fail);
  fail_at = fail_launch = -1;
  cadmas_unet_destroy(n);
  return reached;
}

int main(int argc, char **argv) {
  const bool launch = argc > 1 && !strcmp(argv[1], "launch");
  // small arrays (copied directly) and arrays that come through the pinned chunks
  const int dims[][3] = {{8, 8, 8}, {128, 64, 64}};
  for (auto &d : dims) {
    const size_t V = (size_t)d[0] * d[1] * d[2];
    hx.assign(V * 4, 1.0f); ht.assign(V, 1.0f); hm.assign(V, 1.0f); ha.assign(V * 7, 1.0f); hy.assign(V, 0.0f);
    hg.assign(cadmas_unet_param_count(), 0.0f); hp = hg;
    const bool small = V < 10000;
    for (int entry = 0; entry < 6; ++entry)
      for (bool ae : {false, true}) {
        fake::attr_error = ae;
        // (the chunks' calls are alike: a few of them, and every call of the small arrays)
        for (long long k = 0; one(d[0], d[1], d[2], entry, k, launch); k += small || launch || k < 30 ? 1 : 29) {}
      }
  }
  printf("%lld checks, %lld failures\n", checks, fails);
  return fails != 0;
}
