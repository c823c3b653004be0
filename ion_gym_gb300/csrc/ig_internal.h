// ig_internal.h -- declarations shared by the CUDA translation units of
// libigsolve.so (kernel launchers, control blocks).  Not part of the C-ABI;
// the public entry points are in include/igsolve.h.
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <string>
#include <cuda_runtime.h>

namespace ig {

struct Dims {
  long nx, ny, nz;
  size_t n() const { return (size_t)nx * (size_t)ny * (size_t)nz; }
};

inline Dims coarse_of(const Dims& d) {
  return Dims{(d.nx + 1) / 2, (d.ny + 1) / 2, (d.nz + 1) / 2};
}

// Unsigned 31-bit division by a run-time constant (Granlund & Montgomery,
// "Division by invariant integers using multiplication", PLDI 1994):
// q = (umulhi(n, m) + n) >> s with s = ceil(log2 d) and
// m = floor(2^32 (2^s - d) / d) + 1, exact for every n < 2^31.
struct FastDiv {
  uint32_t d, m, s;
  __host__ __device__ FastDiv() : d(1), m(1), s(0) {}
  explicit FastDiv(uint32_t div) : d(div) {
    s = 0;
    while ((1ull << s) < div) ++s;
    m = (uint32_t)(((1ull << 32) * ((1ull << s) - div)) / div + 1);
  }
};

// Per-batch control block of the exact SOR loop.  A batch is up to
// kMaxBatch red-black pairs launched back to back; slot[2p + c] receives the
// max |update| of colour c of pair p (as order-preserving bits).  The colour-0
// launch of pair p first looks at pair p-1 (or at `prev`, the last pair of
// the previous batch) and, when it met `tol`, marks the batch done so every
// later launch returns at once.  The host then reads the slots and finds the
// pair that converged, exactly as the reference's per-pair test does.
constexpr int kMaxBatch = 256;
struct PairCtl {
  unsigned long long slot[2 * kMaxBatch];
  unsigned long long prev[2];
  double tol;
  int has_prev;
  int limit;
  int done;
  int pad_;
};

// Stencil selector for the fine sweeps.
enum StencilKind : int {
  kPlain = 0,        // theta is all ones: every stencil reduces to sum/6
  kThetaGhost = 1,   // theta given, ghost_linear weights
  kThetaSW = 2,      // theta given, Shortley-Weller weights
  kPlainSW = 3,      // theta all ones, Shortley-Weller residual (sum/2 - 3 phi);
                     // its sweeps equal kPlain's
};

// The theta of a solve sorted by what its nodes need (ig_f64.cu,
// k_theta_class / k_theta_fill): cls per node (0 free with six unit legs,
// 1 fixed, 2 free with a cut leg) and the cut nodes of each colour with
// their stencil weights -- ghost_linear: the six 1/theta and their sum; sw:
// the six leg products v is divided by, and den -- as `total`-long arrays,
// w[q * total + e].  Device memory, built once per solve.
struct ThetaPlan {
  const uint8_t* cls = nullptr;
  const uint32_t* idx = nullptr;  // colour 0's cut nodes, then colour 1's
  const double* w = nullptr;      // 7 * total
  uint32_t count[2] = {0, 0};
  __host__ __device__ uint32_t total() const { return count[0] + count[1]; }
};
constexpr int kThetaWeights = 7;

// ---- exact FP64 kernels (ig_f64.cu) ----
// cls, and the cut nodes of each colour counted into counts[2] (zeroed here)
void launch_theta_class(cudaStream_t s, const uint8_t* fixed, const float* th, Dims d,
                        uint8_t* cls, uint32_t* counts);
// idx and w of the plan; cursor[2] is scratch (zeroed here)
void launch_theta_fill(cudaStream_t s, const uint8_t* cls, const float* th, int kind, Dims d,
                       const uint32_t count[2], uint32_t* cursor, uint32_t* idx, double* w);
// launch_sweep / launch_residual of a solve whose theta is in a plan (kind
// kThetaGhost or kThetaSW): the same bits.
void launch_sweep_plan(cudaStream_t s, double* phi, const ThetaPlan& plan, int kind, Dims d,
                       double omega, int colour, PairCtl* ctl, int lp);
void launch_residual_plan(cudaStream_t s, const double* phi, const ThetaPlan& plan, int kind,
                          Dims d, double* out);
// One colour of the reference SOR sweep.  dslot: where the max |update| goes
// when ctl == nullptr (nullptr: not formed); with ctl the slot is
// ctl->slot[2*lp + colour].
void launch_sweep(cudaStream_t s, double* phi, const uint8_t* fixed,
                  const float* th, int kind, Dims d, double omega, int colour,
                  unsigned long long* dslot, PairCtl* ctl, int lp);
void launch_residual(cudaStream_t s, const double* phi, const uint8_t* fixed,
                     const float* th, int kind, Dims d, double* out,
                     unsigned long long* absmax /* nullable */);
// The whole bottom solve of multigrid3d._solve_err (e = 0, tol from
// max|f|, SOR pairs to 0.02 tol, at most max_pairs) in one CTA with the
// level in shared memory (18 bytes a node); false (nothing launched, no error
// left behind) when the level has more than kBottomSmemMax / 17 nodes or the
// launch was refused.
constexpr size_t kBottomSmemMax = 200 * 1024;
bool launch_bottom_err(cudaStream_t s, double* e, const uint8_t* fixed, const double* f,
                       Dims d, double rel_tol, double omega, long max_pairs);
// SOR pairs until one meets tol, at most `pairs`, in one cooperative launch
// (k_sor_flow): cls holds 0 at the nodes the plain update owns, plan the cut
// nodes of a theta solve (kind kThetaGhost / kThetaSW) or null.  ctl gets
// the pairs run, whether the last met tol and its max |update| key; status 1
// means a wait gave up.  word (32 bytes a slot of one colour) and prev (16)
// are scratch.  false: nothing was launched, since the device takes no such
// launch or refused this one (no error is left behind).
constexpr int kCoopThreads = 1024, kCoopCtas = 512;
struct CoopCtl {
  unsigned arrived;
  int status, pairs, hit;
  unsigned long long key;
  alignas(16) unsigned long long word[4][2 * kCoopCtas];  // a CTA's maximum, pair + 1
};
bool launch_sor_coop(cudaStream_t s, double* phi, const uint8_t* cls, const ThetaPlan* plan,
                     int kind, Dims d, double omega, double tol, int pairs, CoopCtl* ctl,
                     void* word, double* prev);
// multigrid3d._solve_err from level lv[0] (its right-hand side in f) down to
// the bottom lv[nlev - 1] (nlev >= 2) in one launch (k_err_tail); false
// (nothing launched, no error left behind) when the bottom does not fit in
// shared memory or the device takes no such cluster or refused this one.
constexpr int kTailLevels = 12, kTailCtas = 16, kTailThreads = 512;
struct TailLevel {
  double *e, *f, *r;
  const uint8_t* fixed;
  int nx, ny, nz;
  FastDiv dkk, dny, dnz;
  // set by the launch: rows a CTA, and the byte offsets of its part in
  // shared memory (values, right-hand side, mask)
  FastDiv drow;
  uint32_t oe, of, om;
};
struct TailArgs {
  TailLevel lv[kTailLevels];
  int nlev, nu1, nu2, max_cycles;
  double rel_tol, bottom_omega;
  long bottom_pairs;
  uint32_t orr, ob;  // the residual's and the bottom's scratch
};
TailLevel tail_level(Dims d, double* e, double* f, double* r, const uint8_t* fixed);
bool launch_err_tail(cudaStream_t s, TailArgs a);
void launch_sweep_rhs(cudaStream_t s, double* e, const uint8_t* fixed,
                      const double* f, Dims d, double omega, int colour,
                      unsigned long long* dslot, PairCtl* ctl, int lp);
void launch_residual_rhs(cudaStream_t s, const double* e, const uint8_t* fixed,
                         const double* f, Dims d, double* out);
// out = acc/8 (mode 0) or -((acc/8)*4) (mode 1, the coarse right-hand side)
void launch_restrict(cudaStream_t s, const double* fine, Dims d, double* out,
                     Dims c, int neg4);
void launch_prolong_add(cudaStream_t s, const double* coarse, Dims c,
                        double* out, const uint8_t* fixed, Dims d);
void launch_prolongate(cudaStream_t s, const double* coarse, Dims c,
                       double* out, Dims d);
void launch_coarsen_any(cudaStream_t s, const uint8_t* fixed, Dims d,
                        uint8_t* out, Dims c);
void launch_coarsen_mask(cudaStream_t s, const uint8_t* fixed,
                         const double* val, Dims d, uint8_t* fc, double* vc,
                         Dims c);
void launch_set_fixed(cudaStream_t s, double* phi, const uint8_t* fixed,
                      const double* val, size_t n);
// phi[fixed] = v_basis on mask, 0 on the rest of fixed (a basis's Dirichlet
// values without an array of them)
void launch_set_basis(cudaStream_t s, double* phi, const uint8_t* fixed, const uint8_t* mask,
                      double v, size_t n);
// flags[a] = 1 where fixed or the Dirichlet values -- val, or (val null) v on
// mask and 0 elsewhere -- are not invariant under the flip of axis a
// (multigrid3d.py:643-650); flags is zeroed here
void launch_sym_check(cudaStream_t s, const uint8_t* fixed, const double* val,
                      const uint8_t* mask, double v, Dims d, int* flags);
// max |a - b| (b nullable: max |a|) into *bits, NaN noted in *nan_flag
void launch_absdiff_max(cudaStream_t s, const double* a, const double* b,
                        size_t n, unsigned long long* bits, int* nan_flag);
// Two words of the device to mapped host memory.
void launch_report(cudaStream_t s, const unsigned long long* d, unsigned long long* host);
void launch_sym_project(cudaStream_t s, double* phi, Dims d, int axis);
void launch_residual_audit(cudaStream_t s, const double* u,
                           const uint8_t* fixed, const float* th, Dims d,
                           double* out);
void launch_err_sweep(cudaStream_t s, double* e, const uint8_t* fixed,
                      const float* th, const double* rhs, Dims d, double omega,
                      int colour, unsigned long long* dslot);
void launch_fill_ones_f32(cudaStream_t s, float* a, size_t n);

// Number of kernel launches this library has issued since it was loaded.
long launch_total();
// Adds n launches issued by another translation unit to that count.
void note_launches(long n);
// Launches this thread counted, recordings included.
long launch_total_thread();

// Sets the calling thread's ig_last_error() message.
void set_last_error(const std::string& m);

// The calling thread's stream on its current device (created on first use);
// a status, with the message set, when there is none.
int call_stream(cudaStream_t* s);

// A call that keeps the current device busy, for as long as the object lives.
// The resident SOR loop fills the device, so it asks who else is there.
enum CallKind { kSorCall, kOtherCall };
class CallInFlight {
 public:
  explicit CallInFlight(CallKind kind);
  ~CallInFlight();
  CallInFlight(const CallInFlight&) = delete;
  CallInFlight& operator=(const CallInFlight&) = delete;

 private:
  std::atomic<int>* n_;
};

// Whether a kernel may write [p, p + bytes) as elements of `align` bytes: memory
// of the current device, aligned, within one allocation.  Elsewhere a result is
// copied, which takes any address and reports a range past its allocation.
bool device_range(const void* p, size_t bytes, size_t align);

// Waits for the stream when a call leaves, early returns included: copies
// from pageable memory may still be reading the caller's (or the call's own)
// arrays.  Declared after them and after the call's CallBufs.
struct CallSync {
  cudaStream_t s;
  ~CallSync() { cudaStreamSynchronize(s); }
};

// A device buffer of one synchronous call on host arrays.  Small ones come
// from the device's stream-ordered pool, which keeps them for the next call
// (cudaMalloc and cudaFree cost more than the work of a small grid: three
// buffers 200 us); above kPoolBytes, where that no longer shows, the memory
// goes back to the device at once.
constexpr size_t kPoolBytes = size_t(64) << 20;
struct CallBuf {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  bool pooled = false;
  cudaError_t alloc(size_t bytes, cudaStream_t st) {
    s = st;
    pooled = bytes <= kPoolBytes;
    return pooled ? cudaMallocAsync(&p, bytes ? bytes : 16, st) : cudaMalloc(&p, bytes);
  }
  CallBuf() = default;
  CallBuf(const CallBuf&) = delete;
  CallBuf& operator=(const CallBuf&) = delete;
  ~CallBuf() {
    if (!p) return;
    if (pooled) {
      cudaFreeAsync(p, s);
    } else {
      cudaFree(p);
    }
  }
};

}  // namespace ig
