// The library's launchers over a stand-in CUDA runtime of two devices, which
// keeps kernel attributes by device and refuses a launch beyond them as the
// real one does.  Device memory is host memory, kernels compute nothing: a
// launched pair's maxima stay 0, which meets any tolerance, and a resident
// loop runs the pairs it was given without meeting it.  Prints one line per
// check; the first word says what it is, the rest what happened.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "ig_internal.h"
#include "../include/igsolve.h"

namespace {
struct Attr {
  size_t smem = 48 * 1024;
  int cluster = 8, lowered = 0;
};
struct Config {
  dim3 grid, block;
  size_t smem = 0;
  cudaStream_t s = nullptr;
};
int device = 0, launched = 0, refuse = 0, loops = 0, loops_left = 1 << 30;
size_t most_memory = size_t(-1);
// an allocation of device 0 that is never touched
constexpr uintptr_t kRange = 0x7000000000ULL;
constexpr size_t kRangeSize = 4096;
cudaError_t last = cudaSuccess;
std::map<std::pair<int, const void*>, Attr> attrs;
Config config;

cudaError_t note(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t launch(const void* fn, size_t smem, int cluster) {
  const Attr& a = attrs[{device, fn}];
  if (refuse || smem > a.smem || cluster > a.cluster) return note(cudaErrorInvalidValue);
  launched++;
  return cudaSuccess;
}
int cluster_of(const cudaLaunchConfig_t* c) {
  int n = 1;
  for (unsigned q = 0; q < c->numAttrs; q++)
    if (c->attrs[q].id == cudaLaunchAttributeClusterDimension)
      n = (int)c->attrs[q].val.clusterDim.x;
  return n;
}
}  // namespace

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  config.grid = g;
  config.block = b;
  config.smem = smem;
  config.s = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = config.grid;
  *b = config.block;
  *smem = config.smem;
  *static_cast<cudaStream_t*>(s) = config.s;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(fn));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t smem, cudaStream_t) {
  return launch(reinterpret_cast<const void*>(k), smem, 1);
}
cudaError_t cudaLaunchKernel(const void* fn, dim3, dim3, void**, size_t smem, cudaStream_t) {
  return launch(fn, smem, 1);
}
cudaError_t cudaLaunchCooperativeKernel(const void* fn, dim3, dim3, void** args, size_t smem,
                                        cudaStream_t) {
  if (loops == loops_left) return note(cudaErrorInvalidValue);
  const cudaError_t e = launch(fn, smem, 1);
  if (e == cudaSuccess) {
    loops++;
    ig::CoopCtl* ctl = *static_cast<ig::CoopCtl**>(args[7]);
    ctl->pairs = *static_cast<int*>(args[6]);
    ctl->key = 0x7ff0000000000000ULL;
  }
  return e;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
  return launch(fn, c->dynamicSmemBytes, cluster_of(c));
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* fn, const cudaLaunchConfig_t* c) {
  const Attr& a = attrs[{device, fn}];
  if (c->dynamicSmemBytes > a.smem || cluster_of(c) > a.cluster)
    return note(cudaErrorInvalidValue);
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute what, int v) {
  Attr& a = attrs[{device, fn}];
  if (what == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if ((size_t)v < a.smem) a.lowered++;
    a.smem = (size_t)v;
  }
  if (what == cudaFuncAttributeNonPortableClusterSizeAllowed) a.cluster = v ? 16 : 8;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr what, int) {
  *v = what == cudaDevAttrMultiProcessorCount ? 152 : 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = n > most_memory ? nullptr : std::calloc(1, n);
  return *p ? cudaSuccess : note(cudaErrorMemoryAllocation);
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 2;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaMemGetInfo(size_t*, size_t*) { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return note(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  *a = cudaPointerAttributes();
  const auto at = reinterpret_cast<uintptr_t>(p);
  if (at >= kRange && at < kRange + kRangeSize) {
    a->type = cudaMemoryTypeDevice;
    a->device = 0;
  }
  return cudaSuccess;
}
int range_of(unsigned long long* base, size_t* size, unsigned long long) {
  *base = kRange;
  *size = kRangeSize;
  return 0;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* found) {
  *fn = reinterpret_cast<void*>(range_of);
  *found = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}

using namespace ig;

static bool sor(long side) {
  char scratch[64];
  static CoopCtl ctl;
  return launch_sor_coop(nullptr, reinterpret_cast<double*>(scratch),
                         reinterpret_cast<uint8_t*>(scratch), nullptr, kPlain,
                         Dims{side, side, side}, 1.5, 1e-3, 8, &ctl, scratch,
                         reinterpret_cast<double*>(scratch));
}

static bool tail() {
  TailArgs a{};
  for (long n : {33L, 17L, 9L})
    a.lv[a.nlev++] = tail_level(Dims{n, n, n}, nullptr, nullptr, nullptr, nullptr);
  a.nu1 = a.nu2 = 2;
  return launch_err_tail(nullptr, a);
}

static bool bottom(long n) {
  return launch_bottom_err(nullptr, nullptr, nullptr, nullptr, Dims{n, n, n}, 1e-3, 1.5, 10);
}

static void say(const char* what, bool took) {
  std::printf("%s took=%d launched=%d error=%d\n", what, took, launched, (int)cudaGetLastError());
  launched = 0;
}

// A solve of `pairs` pairs at most: which loop it took, and how often.
static void solve(const char* what, long side, long pairs) {
  const size_t n = (size_t)side * side * side;
  std::vector<uint8_t> fixed(n, 0);
  std::vector<double> val(n, 0.0), phi(n);
  loops = launched = 0;
  long sweeps = -1;
  double delta = 0.0;
  const int st = ig_solve3d(fixed.data(), val.data(), nullptr, side, side, side, 1e-3, pairs, 1.5,
                            nullptr, 0, phi.data(), &sweeps, &delta);
  // one launch sets the Dirichlet values
  std::printf("%s status=%d loops=%d launched=%d sweeps=%ld\n", what, st, loops,
              launched - loops - 1 > 0 ? 1 : 0, sweeps);
  loops = launched = 0;
  loops_left = 1 << 30;
  most_memory = size_t(-1);
}

static void routes() {
  solve("alone", 65, 100);
  solve("alone-turns", 65, 600);
  solve("no-pairs", 65, 0);
  {
    const CallInFlight session(kOtherCall);
    solve("beside-a-session", 65, 100);
    solve("small-beside-a-session", 33, 100);
    device = 1;
    solve("session-on-the-other-device", 65, 100);
    device = 0;
  }
  {
    const CallInFlight a(kSorCall), b(kSorCall), c(kSorCall);
    solve("beside-three-solves", 65, 100);
    const CallInFlight d(kSorCall);
    solve("beside-four-solves", 65, 100);
    solve("small-beside-four-solves", 33, 100);
  }
  solve("alone-again", 65, 100);
  loops_left = 0;
  solve("refused", 65, 100);
  loops_left = 1;
  solve("refused-later", 65, 600);
  most_memory = 3u << 20;  // the potential and the mask, not the loop's words
  solve("no-memory", 65, 100);
}

// offset and bytes of a result in the allocation: may a kernel write it?
static void ranges() {
  const struct {
    const char* what;
    size_t at, bytes, align;
  } q[] = {{"range-whole", 0, 4096, 8},  {"range-inside", 24, 800, 8}, {"range-past", 8, 4096, 8},
           {"range-odd", 4, 800, 8},     {"range-float", 4, 800, 4},   {"range-odd-float", 2, 8, 4},
           {"range-host", 1u << 20, 8, 8}};
  for (const auto& r : q)
    std::printf("%s %d\n", r.what,
                (int)device_range(reinterpret_cast<void*>(kRange + r.at), r.bytes, r.align));
  device = 1;
  std::printf("range-other-device %d\n",
              (int)device_range(reinterpret_cast<void*>(kRange), 8, 8));
  device = 0;
}

int main() {
  ranges();
  say("sor-large", sor(129));
  say("sor-small", sor(40));
  int lowered = 0;
  for (auto& a : attrs) lowered += a.second.lowered;
  std::printf("sor-attribute lowered=%d\n", lowered);
  device = 1;
  say("sor-second-device", sor(129));
  refuse = 1;
  say("sor-refused", sor(65));
  refuse = 0;
  for (device = 0; device < 2; device++) {
    const std::string d = std::to_string(device);
    say(("tail-device" + d).c_str(), tail());
    say(("bottom-device" + d).c_str(), bottom(21));  // 167 KB of shared memory
  }
  refuse = 1;
  say("tail-refused", tail());
  say("bottom-refused", bottom(21));
  refuse = device = 0;
  routes();
  return 0;
}
