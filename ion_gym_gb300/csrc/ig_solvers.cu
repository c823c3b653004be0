// ig_solvers.cu -- host drivers of the FP64 solve paths and the C-ABI of
// libigsolve.so (declared in include/igsolve.h).
//
// The drivers restate the reference's Python drivers (solve3d, solve3d_mg,
// solve3d_vmg, _solve_err, the basis loops) with the arrays resident in HBM:
// the host only launches kernels and reads back the few scalars the
// reference branches on (a sweep pair's max |update|, a cycle's max change,
// max |f| of an error level).  Sweep pairs run in batches whose launches
// stop themselves on the device once a pair met the tolerance (PairCtl), so
// the host synchronizes once per batch, not once per pair, and the result is
// still the reference's pair-exact stop.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <limits>
#include <mutex>
#include <stdexcept>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "ig_common.cuh"
#include "ig_internal.h"
#include "../../include/igsolve.h"

namespace ig {
namespace {

thread_local std::string t_err;
std::atomic<int> g_stop{0};

struct Prof {
  std::atomic<int> on{0};
  double ms = 0.0;
  long launches = 0;
  long nodes = 0;
} g_prof;

struct Status : std::runtime_error {
  int code;
  Status(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define CK(x)                                                                  \
  do {                                                                         \
    cudaError_t e_ = (x);                                                      \
    if (e_ != cudaSuccess)                                                     \
      throw Status(IG_CUDA_ERROR, std::string(#x) + ": " +                     \
                                      cudaGetErrorString(e_) + " (line " +    \
                                      std::to_string(__LINE__) + ")");         \
  } while (0)

// A calling thread's stream and pinned control block.  Taken on the thread's
// first call and handed on when it ends, so a program has as many as it had
// threads at once: the basis door starts its workers anew on every call, and
// a stream, two events and a pinned allocation for each (which wait for the
// device) were made, and lost, every time.
struct ThreadCtx {
  int dev = -1;
  cudaStream_t s = nullptr;
  PairCtl* ctl_h = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

// The idle ones (never destroyed: the driver reclaims them at process exit).
struct CtxPool {
  std::mutex mu;
  std::vector<ThreadCtx> idle;
};
CtxPool& ctx_pool() {
  static CtxPool* p = new CtxPool;
  return *p;
}

// The calls in flight on a device, counted by CallInFlight.
struct DeviceCalls {
  std::atomic<int> sor{0}, other{0};
};
DeviceCalls& device_calls() {
  constexpr int kMost = 64;
  static DeviceCalls k[kMost + 1];  // the last: devices past the rest
  int dev = kMost;
  if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
  return k[dev < 0 || dev > kMost ? kMost : dev];
}

struct CtxHolder {
  ThreadCtx c;
  void hand_on() {
    if (c.dev < 0) return;
    CtxPool& p = ctx_pool();
    std::lock_guard<std::mutex> lk(p.mu);
    p.idle.push_back(c);
    c = ThreadCtx();
  }
  ~CtxHolder() { hand_on(); }
};
thread_local CtxHolder t_ctx;

ThreadCtx& ctx() {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
    throw Status(IG_NO_DEVICE, "no CUDA device is visible");
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (t_ctx.c.dev != dev) {
    t_ctx.hand_on();
    CtxPool& p = ctx_pool();
    {
      std::lock_guard<std::mutex> lk(p.mu);
      for (size_t q = p.idle.size(); q-- > 0;)
        if (p.idle[q].dev == dev) {
          t_ctx.c = p.idle[q];
          p.idle.erase(p.idle.begin() + (long)q);
          return t_ctx.c;
        }
    }
    ThreadCtx c;
    CK(cudaStreamCreateWithFlags(&c.s, cudaStreamNonBlocking));
    CK(cudaMallocHost(&c.ctl_h, sizeof(PairCtl)));
    CK(cudaEventCreate(&c.ev0));
    CK(cudaEventCreate(&c.ev1));
    // keep freed stream-ordered allocations cached between solves
    cudaMemPool_t pool;
    CK(cudaDeviceGetDefaultMemPool(&pool, dev));
    uint64_t thr = std::numeric_limits<uint64_t>::max();
    CK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr));
    c.dev = dev;
    t_ctx.c = c;
  }
  return t_ctx.c;
}

// Stream-ordered device buffer.
template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  cudaStream_t s = nullptr;
  DBuf() = default;
  DBuf(size_t count, cudaStream_t st) { alloc(count, st); }
  void alloc(size_t count, cudaStream_t st) {
    release();
    s = st;
    n = count;
    if (count) CK(cudaMallocAsync((void**)&p, std::max<size_t>(count * sizeof(T), 16), st));
  }
  void release() {
    if (p) cudaFreeAsync(p, s);
    p = nullptr;
    n = 0;
  }
  ~DBuf() { release(); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n), s(o.s) { o.p = nullptr; o.n = 0; }
  DBuf& operator=(DBuf&& o) noexcept {
    release();
    p = o.p; n = o.n; s = o.s;
    o.p = nullptr; o.n = 0;
    return *this;
  }
};

void check_dims(long nx, long ny, long nz) {
  if (nx < 1 || ny < 1 || nz < 1)
    throw Status(IG_BAD_ARG, "every axis of the grid must be >= 1");
  const double n = (double)nx * (double)ny * (double)nz;
  if (n >= 2147483648.0)
    throw Status(IG_BAD_ARG, "grids of 2^31 nodes or more are not supported");
}

int stencil_check(int stencil) {
  if (stencil != 0 && stencil != 1)
    throw Status(IG_BAD_ARG, "unknown stencil code (0 = ghost_linear, 1 = sw)");
  return stencil;
}

// Sweep kernel kind for a fine grid: theta None reduces both stencils to
// sum/6 (Shortley-Weller with unit legs halves num and den alike).
int sweep_kind(bool theta, int stencil) {
  if (!theta) return kPlain;
  return stencil == 0 ? kThetaGhost : kThetaSW;
}

// Residual kind: with theta None the two stencils differ by a factor of 2
// (ghost_linear: sum - 6 phi; Shortley-Weller: sum/2 - 3 phi).
constexpr int kPlainSWResid = kPlainSW;

double optimal_omega_libm(const Dims& d) {
  // solver3d.optimal_omega (solver3d.py:201-230) for unit spacing
  double num = 0.0, wsum = 0.0;
  const long ns[3] = {d.nx, d.ny, d.nz};
  bool any = false;
  for (long n : ns)
    if (n >= 2) {
      num += std::cos(M_PI / (double)(n + 1));
      wsum += 1.0;
      any = true;
    }
  if (!any) return 1.0;
  double rho = num / wsum;
  rho = std::min(rho, 1.0 - 1e-15);
  return 2.0 / (1.0 + std::sqrt(1.0 - rho * rho));
}

inline double umax(unsigned long long a, unsigned long long b) {
  return bits_to_double(a > b ? a : b);
}

struct PairsResult {
  long pairs;
  double delta;
  bool converged;
};

// The reference's "for s in range(max): d = max(d1, d2); if d < tol: stop"
// loop, in device-terminated batches.  launch_pair(lp, ctl) enqueues the
// colour-0 and colour-1 launches of local pair lp.
template <class F>
PairsResult run_pairs(ThreadCtx& c, PairCtl* ctl_d, double tol, long max_pairs,
                      size_t nodes, F&& launch_pair) {
  PairCtl* h = c.ctl_h;
  long base = 0;
  int has_prev = 0;
  unsigned long long prev[2] = {0, 0};
  double last = std::numeric_limits<double>::quiet_NaN();
  int B = 8;
  const bool prof = g_prof.on.load() != 0;
  while (base < max_pairs) {
    const int lim = (int)std::min<long>(B, max_pairs - base);
    std::memset(h, 0, sizeof(PairCtl));
    h->prev[0] = prev[0];
    h->prev[1] = prev[1];
    h->has_prev = has_prev;
    h->limit = lim;
    h->tol = tol;
    CK(cudaMemcpyAsync(ctl_d, h, sizeof(PairCtl), cudaMemcpyHostToDevice, c.s));
    if (prof) CK(cudaEventRecord(c.ev0, c.s));
    for (int lp = 0; lp < lim; lp++) launch_pair(lp, ctl_d);
    CK(cudaGetLastError());
    if (prof) CK(cudaEventRecord(c.ev1, c.s));
    CK(cudaMemcpyAsync(h, ctl_d, sizeof(PairCtl), cudaMemcpyDeviceToHost, c.s));
    CK(cudaStreamSynchronize(c.s));
    int ran = lim;
    PairsResult res{0, 0.0, false};
    for (int lp = 0; lp < lim; lp++) {
      const double d = umax(h->slot[2 * lp], h->slot[2 * lp + 1]);
      if (d < tol) {
        res = {base + lp + 1, d, true};
        ran = lp + 1;
        break;
      }
      last = d;
    }
    if (prof) {
      float ms = 0.f;
      CK(cudaEventElapsedTime(&ms, c.ev0, c.ev1));
      g_prof.ms += ms;
      g_prof.launches += 2L * ran;
      g_prof.nodes += (long)nodes * ran;
    }
    if (res.converged) return res;
    prev[0] = h->slot[2 * lim - 2];
    prev[1] = h->slot[2 * lim - 1];
    has_prev = 1;
    base += lim;
    B = std::min(kMaxBatch, 2 * B);
  }
  return {max_pairs, last, false};
}

// Two 64-bit words of the device, written by a kernel to the context's
// pinned memory: the copy engine takes the copies of all streams in turn, so
// a few bytes behind a copy that waits for another solve's kernels wait for
// them too (eight bases at once: one read in ten 400 to 880 us).
// As a 64-bit max key (sync) and, with `nan`, an int in the second word's low
// half that flags NaN.
double read_absmax(ThreadCtx& c, const unsigned long long* words_d, bool nan) {
  launch_report(c.s, words_d, c.ctl_h->slot);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c.s));
  const unsigned long long* w = c.ctl_h->slot;
  if (nan && (int)w[1]) return std::numeric_limits<double>::quiet_NaN();
  return bits_to_double(w[0]);
}

double device_absmax(ThreadCtx& c, const double* a, const double* b, size_t n,
                     DBuf<unsigned long long>& scratch) {
  // scratch: [0] = max bits, [1] = NaN flag (as int in the low word)
  CK(cudaMemsetAsync(scratch.p, 0, 16, c.s));
  launch_absdiff_max(c.s, a, b, n, scratch.p, (int*)(scratch.p + 1));
  return read_absmax(c, scratch.p, true);
}

// ---------------------------------------------------------------- SOR
// A solve's theta in plan form (empty: no theta, or the general kernels).
struct Theta {
  DBuf<uint8_t> cls;
  DBuf<uint32_t> idx;
  DBuf<double> w;
  ThetaPlan plan;
  bool on() const { return plan.cls != nullptr; }
};

struct FineGrid {
  Dims d;
  DBuf<uint8_t> fixed;
  DBuf<double> phi;
  DBuf<float> th;  // empty when theta is None, or once the plan holds it
  int stencil = 0;
  bool theta = false;
  Theta plan;
};

// The theta of one solve as a plan, where that pays: few cut nodes (at most
// a tenth of the grid; every geometry's surface nodes are far fewer), so
// that the lists (60 bytes a cut node) and cls stay below the theta array
// they replace and no solve needs more memory than with that array.
// theta arrays with more cut nodes keep the general kernels.  `th` is freed
// when the plan took it over.
void plan_theta(ThreadCtx& c, Theta& t, DBuf<float>& th, const uint8_t* fixed, Dims d,
                int stencil) {
  if (!th.p) return;
  const size_t n = d.n();
  t.cls.alloc(n, c.s);
  DBuf<uint32_t> cnt(2, c.s);
  launch_theta_class(c.s, fixed, th.p, d, t.cls.p, cnt.p);
  CK(cudaGetLastError());
  uint32_t count[2] = {0, 0};
  CK(cudaMemcpyAsync(count, cnt.p, sizeof(count), cudaMemcpyDeviceToHost, c.s));
  CK(cudaStreamSynchronize(c.s));
  const size_t total = (size_t)count[0] + count[1];
  if (total > n / 10) {
    t.cls.release();
    return;
  }
  t.idx.alloc(total, c.s);
  t.w.alloc(kThetaWeights * total, c.s);
  launch_theta_fill(c.s, t.cls.p, th.p, stencil == 0 ? kThetaGhost : kThetaSW, d, count, cnt.p,
                    t.idx.p, t.w.p);
  CK(cudaGetLastError());
  t.plan.cls = t.cls.p;
  t.plan.idx = t.idx.p;
  t.plan.w = t.w.p;
  t.plan.count[0] = count[0];
  t.plan.count[1] = count[1];
  th.release();
}

// A call's Dirichlet values: val (n), or v on the nodes of mask and 0 on the
// rest of the metal (a basis).  Caller's memory.
struct Dirichlet {
  const double* val = nullptr;
  const uint8_t* mask = nullptr;
  double v = 0.0;
};

// ... and on the device.
struct DirichletDev {
  DBuf<double> val;
  DBuf<uint8_t> mask;
  void load(ThreadCtx& c, const Dirichlet& b, size_t n) {
    if (b.val) {
      val.alloc(n, c.s);
      CK(cudaMemcpyAsync(val.p, b.val, n * 8, cudaMemcpyDefault, c.s));
    } else {
      mask.alloc(n, c.s);
      CK(cudaMemcpyAsync(mask.p, b.mask, n, cudaMemcpyDefault, c.s));
    }
  }
};

// phi = phi0 (or 0); phi[fixed] = val[fixed]  (solver3d.py:263-265)
void init_phi(ThreadCtx& c, FineGrid& g, const Dirichlet& b, const double* phi0_h,
              DirichletDev& d) {
  const size_t n = g.d.n();
  if (phi0_h)
    CK(cudaMemcpyAsync(g.phi.p, phi0_h, n * 8, cudaMemcpyDefault, c.s));
  else
    CK(cudaMemsetAsync(g.phi.p, 0, n * 8, c.s));
  d.load(c, b, n);
  if (b.val)
    launch_set_fixed(c.s, g.phi.p, g.fixed.p, d.val.p, n);
  else
    launch_set_basis(c.s, g.phi.p, g.fixed.p, d.mask.p, b.v, n);
}

// One colour of a fine grid's sweep by the plan or the general kernels.
void fine_sweep(cudaStream_t s, double* phi, const uint8_t* fx, const float* th, const Theta& t,
                int kind, Dims d, double omega, int colour, PairCtl* ctl, int lp) {
  if (t.on())
    launch_sweep_plan(s, phi, t.plan, kind, d, omega, colour, ctl, lp);
  else
    launch_sweep(s, phi, fx, th, kind, d, omega, colour, nullptr, ctl, lp);
}

// Slots of one colour up to which the SOR loop is one launch (k_sor_flow):
// eight nodes a thread.  A half-sweep of solve3d, launched against resident
// (us, host copies of the call included): 33^3 7.1 / 2.1, 65^3 11.1 / 3.8,
// 97^3 22.9 / 8.6, 129^3 31.3 / 19.9; with theta (sw) 33^3 9.6 / 2.7, 65^3
// 14.6 / 3.9, 129^3 44.6 / 20.6.  Past that the sweep itself fills the GPU,
// one call would hold every SM for long, and a thread's neighbour slots fill
// its SM's shared memory.
constexpr long kCoopSlots = 8L * 152 * kCoopThreads;

// A resident loop has a CTA on every SM until it ends, and other streams'
// kernels come in where it leaves room, or between two launches.  So it runs
// in turns, after each of which the host looks who else is there:
//  * Calls of another kind in this process (sessions, V-cycles, geometry, host
//    fields) are many short launches, each of which would wait for a turn:
//    while there is one, the sweeps are launched.  Beside three solves in a
//    loop a batch of eight 65^3 decks took 160 ms (solves of 65^3) and 1.8 s
//    (129^3) without this, 6.6 and 36 ms beside launched sweeps.
//  * Up to kCoopCalls solves keep their loops, which then take turns; with
//    more, launched sweeps overlap better, unless two loops fit on an SM.
//    Solves a second, launched / resident: 65^3 two calls 378 / 638, four
//    594 / 658, six 749 / 660, eight 807 / 663; 49^3 eight 1372 / 2064; 33^3
//    eight 2875 / 8368.
// A turn is about 2 ms (kernels of other libraries and processes wait for no
// more than that), a pair some 3 us and 34 ps a slot; a turn costs some 25 us
// besides.
constexpr int kCoopCalls = 4;
constexpr long kCoopShared = 512L * 152;  // slots: half an SM's registers
inline int coop_turn(long slots) { return (int)(2e9 / (3e6 + 34.0 * (double)slots)); }
// Launched pairs before the host looks again.
constexpr long kLaunchedTurn = 2 * kMaxBatch;

bool may_stay(long slots) {
  const DeviceCalls& k = device_calls();
  return k.other.load() == 0 && (slots <= kCoopShared || k.sor.load() <= kCoopCalls);
}

// What a solve's resident loop needs; `on` while it may still be had.
struct Resident {
  bool on = false;
  DBuf<CoopCtl> ctl;
  DBuf<ulonglong2> word;
  DBuf<double> before;
};

// Up to `pairs` pairs by k_sor_flow; false: nothing was run (no memory for it,
// or the device refused the launch).
bool resident_pairs(ThreadCtx& c, Resident& R, double* phi, const uint8_t* fx, const Theta& t,
                    int kind, Dims d, double omega, double tol, int pairs, PairsResult* out) {
  if (!R.before.p) {
    const size_t slots = (size_t)(d.nx * d.ny * ((d.nz + 1) / 2));
    try {
      R.ctl.alloc(1, c.s);
      R.word.alloc(2 * slots, c.s);
      R.before.alloc(2 * slots, c.s);
    } catch (const Status&) {
      cudaGetLastError();
      R.ctl.release();
      R.word.release();
      return false;
    }
  }
  const bool prof = g_prof.on.load() != 0;
  if (prof) CK(cudaEventRecord(c.ev0, c.s));
  if (!launch_sor_coop(c.s, phi, t.on() ? t.plan.cls : fx, t.on() ? &t.plan : nullptr, kind, d,
                       omega, tol, pairs, R.ctl.p, R.word.p, R.before.p))
    return false;
  if (prof) CK(cudaEventRecord(c.ev1, c.s));
  CoopCtl h;
  CK(cudaMemcpyAsync(&h, R.ctl.p, offsetof(CoopCtl, word), cudaMemcpyDeviceToHost, c.s));
  CK(cudaStreamSynchronize(c.s));
  if (h.status) throw Status(IG_CUDA_ERROR, "SOR loop: a wait ran out of time");
  if (prof) {
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, c.ev0, c.ev1));
    g_prof.ms += ms;
    g_prof.launches += 1;
    g_prof.nodes += (long)d.n() * h.pairs;
  }
  *out = {h.pairs, bits_to_double(h.key), h.hit != 0};
  return true;
}

PairsResult sor_loop(ThreadCtx& c, double* phi, const uint8_t* fx,
                     const float* th, const Theta& t, int stencil, Dims d, double omega,
                     double tol, long max_pairs, PairCtl* ctl_d) {
  const int kind = sweep_kind(th || t.on(), stencil);
  cudaStream_t s = c.s;
  auto launched = [&](long pairs) {
    return run_pairs(c, ctl_d, tol, pairs, d.n(), [&](int lp, PairCtl* ctl) {
      for (int colour = 0; colour < 2; colour++)
        fine_sweep(s, phi, fx, th, t, kind, d, omega, colour, ctl, lp);
    });
  };
  const long slots = d.nx * d.ny * ((d.nz + 1) / 2);
  Resident R;
  R.on = !(th && !t.on()) && slots <= kCoopSlots;
  long base = 0;
  PairsResult r{0, std::numeric_limits<double>::quiet_NaN(), false};
  while (R.on && base < max_pairs && !r.converged) {
    const long left = max_pairs - base;
    if (may_stay(slots))
      R.on = resident_pairs(c, R, phi, fx, t, kind, d, omega, tol,
                            (int)std::min<long>(coop_turn(slots), left), &r);
    else
      r = launched(std::min(kLaunchedTurn, left));
    if (R.on) base += r.pairs;
  }
  if ((!R.on && base < max_pairs) || max_pairs < 1) {
    r = launched(max_pairs - base);
    base += r.pairs;
  }
  return {base, r.delta, r.converged};
}

// ---------------------------------------------------------------- V-cycle
//
// The launches between two decisions of a cycle, the same ones each time (the
// solve's buffers, grid and options): enqueued one by one the first kDirect
// times and run as a graph from then on.  With eight bases at once each
// launch waits its turn in the driver and a graph of twenty is one turn (2 us
// of the host against 30): 4.1 -> 0.7 us between two sweeps of a stream
// (median), 8 bases of a 97 x 97 x 193 ring deck 78 -> 75 ms, 4 with theta at
// 65 x 65 x 129 24.8 -> 23.1 ms.  Making one takes 30 to 60 us, two runs'
// launches.  Where nothing can be captured it keeps enqueuing.
struct Replay {
  static constexpr int kDirect = 3;
  cudaGraphExec_t x = nullptr;
  int runs = 0;
  long kernels = 0;
  Replay() = default;
  Replay(Replay&& o) noexcept : x(o.x), runs(o.runs), kernels(o.kernels) { o.x = nullptr; }
  Replay& operator=(Replay&&) = delete;
  ~Replay() {
    if (x) cudaGraphExecDestroy(x);
  }
  // Runs what `enqueue` enqueues.  false: nothing was run (not yet a graph, or
  // none to be had).
  template <class F>
  bool operator()(ThreadCtx& c, F&& enqueue) {
    if (!x && runs++ == kDirect) capture(c, enqueue);
    if (!x) return false;
    CK(cudaGraphLaunch(x, c.s));
    note_launches(kernels);
    return true;
  }

 private:
  template <class F>
  void capture(ThreadCtx& c, F&& enqueue) {
    if (cudaStreamBeginCapture(c.s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    cudaGraph_t g = nullptr;
    bool ok = false;
    const long before = launch_total_thread();
    try {
      ok = enqueue();
    } catch (...) {
    }
    kernels = launch_total_thread() - before;
    note_launches(-kernels);  // recorded, not run
    ok = cudaStreamEndCapture(c.s, &g) == cudaSuccess && ok;
    if (!ok || cudaGraphInstantiate(&x, g, 0) != cudaSuccess) x = nullptr;
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
  }
};

struct ErrLevel {
  Dims d;
  DBuf<uint8_t> fixed;
  DBuf<double> e, f, r;
  bool bottom = false;
  Replay cycle;  // of a level above one that runs in one launch
};

struct VCycle {
  std::vector<ErrLevel> lv;  // lv[0]: the first coarse (error) level
  DBuf<unsigned long long> slots;  // the max keys of a cycle's last sweep pair
  DBuf<unsigned long long> red;    // absmax scratch
  DBuf<PairCtl> ctl;
  double bottom_omega = 1.0;
  int nu1 = 3, nu2 = 3;
  double rel_tol = 0.05;
  int max_cycles_err = 30;
  int min_coarse = 9;
};

// Builds the error hierarchy below a fine grid: block-ANY masks
// (multigrid3d.py:675 on the fine grid, :578 on every error level).
void build_err_levels(ThreadCtx& c, VCycle& v, const uint8_t* fine_fixed,
                      Dims fine) {
  Dims d = coarse_of(fine);
  const uint8_t* src = fine_fixed;
  Dims sd = fine;
  while (true) {
    ErrLevel L;
    L.d = d;
    L.fixed.alloc(d.n(), c.s);
    launch_coarsen_any(c.s, src, sd, L.fixed.p, d);
    L.e.alloc(d.n(), c.s);
    L.f.alloc(d.n(), c.s);
    L.bottom = std::min({d.nx, d.ny, d.nz}) <= v.min_coarse;
    if (!L.bottom) L.r.alloc(d.n(), c.s);
    v.lv.push_back(std::move(L));
    if (v.lv.back().bottom) break;
    src = v.lv.back().fixed.p;
    sd = d;
    d = coarse_of(d);
  }
  CK(cudaGetLastError());
}

// Nodes up to which a level and everything below it run in one launch
// (k_err_tail, 16 SMs): above, the launched kernels' 152 SMs win.
constexpr size_t kTailNodes = 65536;
// max|f| up to which a level's error solve cannot overflow.  Beyond it (NaN
// and infinities included) the cycles may run to their caps, which the host
// should be driving.
constexpr double kTailMaxF = 1e200;

// Level L's error solve as one launch: its arguments; false: not possible.
bool err_tail_args(VCycle& v, size_t L, double fmax, TailArgs* t) {
  if (v.lv[L].bottom || v.lv[L].d.n() > kTailNodes || v.lv.size() - L > (size_t)kTailLevels ||
      v.nu2 < 1 || !(fmax < kTailMaxF))
    return false;
  t->nlev = (int)(v.lv.size() - L);
  for (size_t q = L; q < v.lv.size(); q++)
    t->lv[q - L] = tail_level(v.lv[q].d, v.lv[q].e.p, v.lv[q].f.p, v.lv[q].r.p, v.lv[q].fixed.p);
  t->nu1 = v.nu1;
  t->nu2 = v.nu2;
  t->max_cycles = v.max_cycles_err;
  t->rel_tol = v.rel_tol;
  t->bottom_omega = v.bottom_omega;
  t->bottom_pairs = 20000;
  return true;
}

// Runs it; false: not done.
bool solve_err_tail(ThreadCtx& c, VCycle& v, size_t L, double fmax) {
  TailArgs t;
  if (!err_tail_args(v, L, fmax, &t) || !launch_err_tail(c.s, t)) return false;
  CK(cudaGetLastError());
  return true;
}

// multigrid3d._solve_err (multigrid3d.py:553-599) on level L; the level's
// right-hand side is already in lv[L].f, the solution lands in lv[L].e.
// above: max|f| of the level above (its corrections' right-hand sides stay
// within a few powers of ten of it).
void solve_err(ThreadCtx& c, VCycle& v, size_t L, double above) {
  ErrLevel& a = v.lv[L];
  const size_t n = a.d.n();
  if (solve_err_tail(c, v, L, above)) return;
  if (a.bottom && launch_bottom_err(c.s, a.e.p, a.fixed.p, a.f.p, a.d, v.rel_tol,
                                    v.bottom_omega, 20000)) {
    CK(cudaGetLastError());
    return;
  }
  CK(cudaMemsetAsync(a.e.p, 0, n * 8, c.s));
  const double fmax = device_absmax(c, a.f.p, nullptr, n, v.red);
  const double scale = (1e-300 > fmax) ? 1e-300 : fmax;  // max(|f|.max(), 1e-300)
  const double tol = v.rel_tol * scale / 6.0;
  if (a.bottom) {
    const double om = v.bottom_omega;
    double* e = a.e.p;
    const uint8_t* fx = a.fixed.p;
    const double* f = a.f.p;
    const Dims d = a.d;
    cudaStream_t s = c.s;
    run_pairs(c, v.ctl.p, 0.02 * tol, 20000, 0, [&](int lp, PairCtl* ctl) {
      launch_sweep_rhs(s, e, fx, f, d, om, 0, nullptr, ctl, lp);
      launch_sweep_rhs(s, e, fx, f, d, om, 1, nullptr, ctl, lp);
    });
    return;
  }
  ErrLevel& b = v.lv[L + 1];
  unsigned long long* sl = v.slots.p;
  const auto down = [&] {
    for (int q = 0; q < 2 * v.nu1; q++)
      launch_sweep_rhs(c.s, a.e.p, a.fixed.p, a.f.p, a.d, 1.0, q & 1, nullptr, nullptr, 0);
    launch_residual_rhs(c.s, a.e.p, a.fixed.p, a.f.p, a.d, a.r.p);
    launch_restrict(c.s, a.r.p, a.d, b.f.p, b.d, 1);
  };
  const auto up = [&] {
    launch_prolong_add(c.s, b.e.p, b.d, a.e.p, a.fixed.p, a.d);
    if (v.nu2 <= 0) return;
    // the last pair's max |update| decides; the others' are not formed
    CK(cudaMemsetAsync(sl, 0, 16, c.s));
    for (int q = 0; q < 2 * v.nu2; q++)
      launch_sweep_rhs(c.s, a.e.p, a.fixed.p, a.f.p, a.d, 1.0, q & 1,
                       q / 2 + 1 == v.nu2 ? sl + (q & 1) : nullptr, nullptr, 0);
    launch_report(c.s, sl, c.ctl_h->slot);
  };
  TailArgs tail;
  const bool one = err_tail_args(v, L + 1, fmax, &tail);
  for (int cyc = 0; cyc < v.max_cycles_err; cyc++) {
    const bool replayed = one && a.cycle(c, [&] {
      down();
      if (!launch_err_tail(c.s, tail)) return false;
      up();
      return true;
    });
    if (!replayed) {
      down();
      solve_err(c, v, L + 1, fmax);
      up();
    }
    CK(cudaGetLastError());
    if (v.nu2 > 0) {
      CK(cudaStreamSynchronize(c.s));
      if (umax(c.ctl_h->slot[0], c.ctl_h->slot[1]) < tol) break;
    } else {
      if (0.0 < tol) break;
    }
  }
}

// Axes along which fixed and the values are exactly flip-invariant
// (multigrid3d.py:643-650).
std::vector<int> sym_axes(ThreadCtx& c, const FineGrid& g, const Dirichlet& b,
                          const DirichletDev& d) {
  DBuf<int> flags(3, c.s);
  launch_sym_check(c.s, g.fixed.p, d.val.p, d.mask.p, b.v, g.d, flags.p);
  CK(cudaGetLastError());
  int h[3] = {1, 1, 1};
  CK(cudaMemcpyAsync(h, flags.p, sizeof(h), cudaMemcpyDeviceToHost, c.s));
  CK(cudaStreamSynchronize(c.s));
  const long n[3] = {g.d.nx, g.d.ny, g.d.nz};
  std::vector<int> axes;
  for (int a = 0; a < 3; a++)
    if (n[a] >= 3 && !h[a]) axes.push_back(a);
  return axes;
}

struct VmgOut {
  int status;
  long sweeps;
  double delta;
  int cycles;
  double prev;
};

// multigrid3d.solve3d_vmg (multigrid3d.py:602-731) on a prepared fine grid.
VmgOut vmg_loop(ThreadCtx& c, FineGrid& g, VCycle& v, double tol,
                int max_cycles, int accept_stagnation,
                const std::vector<int>& sym) {
  const size_t n = g.d.n();
  const int kind = sweep_kind(g.theta, g.stencil);
  const int rkind = g.theta ? kind : (g.stencil == 0 ? kPlain : kPlainSWResid);
  DBuf<double> r(n, c.s), phi_c0(n, c.s);
  ErrLevel& e0 = v.lv[0];
  long sweeps = 0;
  double prev = std::numeric_limits<double>::infinity();
  double cycle_d = std::numeric_limits<double>::infinity();
  for (int cyc = 0; cyc < max_cycles; cyc++) {
    if (g_stop.load()) return {IG_INTERRUPTED, sweeps, prev, cyc, prev};
    CK(cudaMemcpyAsync(phi_c0.p, g.phi.p, n * 8, cudaMemcpyDeviceToDevice, c.s));
    for (int q = 0; q < v.nu1; q++) {
      for (int colour = 0; colour < 2; colour++)
        fine_sweep(c.s, g.phi.p, g.fixed.p, g.th.p, g.plan, kind, g.d, 1.0, colour, nullptr, 0);
      sweeps++;
    }
    CK(cudaGetLastError());
    if (g_stop.load()) {
      CK(cudaStreamSynchronize(c.s));
      return {IG_INTERRUPTED, sweeps, prev, cyc, prev};
    }
    if (g.plan.on())
      launch_residual_plan(c.s, g.phi.p, g.plan.plan, rkind, g.d, r.p);
    else
      launch_residual(c.s, g.phi.p, g.fixed.p, g.th.p, rkind, g.d, r.p, nullptr);
    launch_restrict(c.s, r.p, g.d, e0.f.p, e0.d, 1);
    CK(cudaGetLastError());
    // a first level small enough for one launch is checked here; a larger
    // one reads its own max|f|
    const double f0 = !e0.bottom && e0.d.n() <= kTailNodes
                          ? device_absmax(c, e0.f.p, nullptr, e0.d.n(), v.red)
                          : std::numeric_limits<double>::infinity();
    solve_err(c, v, 0, f0);
    launch_prolong_add(c.s, e0.e.p, e0.d, g.phi.p, g.fixed.p, g.d);
    for (int q = 0; q < v.nu2; q++) {
      for (int colour = 0; colour < 2; colour++)
        fine_sweep(c.s, g.phi.p, g.fixed.p, g.th.p, g.plan, kind, g.d, 1.0, colour, nullptr, 0);
      sweeps++;
    }
    for (int a : sym) launch_sym_project(c.s, g.phi.p, g.d, a);
    CK(cudaGetLastError());
    cycle_d = device_absmax(c, g.phi.p, phi_c0.p, n, v.red);
    if (cycle_d < tol) return {IG_OK, sweeps, cycle_d, cyc + 1, prev};
    if (cycle_d >= prev) {
      if (accept_stagnation) return {IG_OK, sweeps, cycle_d, cyc + 1, prev};
      return {IG_STAGNATED, sweeps, cycle_d, cyc, prev};
    }
    prev = cycle_d;
  }
  return {IG_CYCLE_CAP, sweeps, cycle_d, max_cycles, prev};
}

void prepare_vcycle(ThreadCtx& c, VCycle& v, FineGrid& g, int nu1, int nu2,
                    double bottom_omega) {
  v.nu1 = nu1;
  v.nu2 = nu2;
  build_err_levels(c, v, g.fixed.p, g.d);
  v.bottom_omega = bottom_omega > 0 ? bottom_omega : optimal_omega_libm(v.lv.back().d);
  v.slots.alloc(2, c.s);
  v.red.alloc(2, c.s);
  v.ctl.alloc(1, c.s);
}

void load_fine(ThreadCtx& c, FineGrid& g, const uint8_t* fixed,
               const float* theta, long nx, long ny, long nz, int stencil) {
  check_dims(nx, ny, nz);
  g.d = Dims{nx, ny, nz};
  g.stencil = stencil_check(stencil);
  const size_t n = g.d.n();
  g.fixed.alloc(n, c.s);
  CK(cudaMemcpyAsync(g.fixed.p, fixed, n, cudaMemcpyDefault, c.s));
  g.phi.alloc(n, c.s);
  if (theta) {
    g.theta = true;
    g.th.alloc(6 * n, c.s);
    CK(cudaMemcpyAsync(g.th.p, theta, 6 * n * 4, cudaMemcpyDefault, c.s));
    plan_theta(c, g.plan, g.th, g.fixed.p, g.d, g.stencil);
  }
}

// Brings the pages of a call's pageable output array in while the GPU
// solves.  A fresh array's pages are otherwise faulted in by the copy at the
// end, which the bases of a door call do at the same time and on one lock:
// eight copies of 14.5 MB took 1 to 17 ms, into touched pages 1 to 2.
struct PageTouch {
  std::thread t;
  PageTouch(void* p, size_t bytes) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    if (a.type != cudaMemoryTypeUnregistered || bytes < (size_t(1) << 20)) return;
    try {
      t = std::thread([p, bytes] {
        volatile unsigned char* q = static_cast<unsigned char*>(p);
        for (size_t o = 0; o < bytes; o += 4096) q[o] = q[o];
      });
    } catch (const std::system_error&) {  // no thread: the copy faults them in
    }
  }
  void join() {
    if (t.joinable()) t.join();
  }
  ~PageTouch() { join(); }
};

void copy_out(ThreadCtx& c, const double* d, double* h, size_t n) {
  CK(cudaMemcpyAsync(h, d, n * 8, cudaMemcpyDefault, c.s));
  CK(cudaStreamSynchronize(c.s));
}

// ---------------------------------------------------------------- cascadic
struct MgLevel {
  Dims d;
  DBuf<uint8_t> fixed;
  DBuf<double> val;
};

std::vector<MgLevel> build_mg_levels(ThreadCtx& c, const uint8_t* fixed_h,
                                     const double* val_h, Dims d,
                                     int min_coarse, int max_levels) {
  std::vector<MgLevel> lv;
  MgLevel f0;
  f0.d = d;
  f0.fixed.alloc(d.n(), c.s);
  f0.val.alloc(d.n(), c.s);
  CK(cudaMemcpyAsync(f0.fixed.p, fixed_h, d.n(), cudaMemcpyDefault, c.s));
  CK(cudaMemcpyAsync(f0.val.p, val_h, d.n() * 8, cudaMemcpyDefault, c.s));
  lv.push_back(std::move(f0));
  while ((int)lv.size() < max_levels) {
    const Dims& a = lv.back().d;
    const Dims b = coarse_of(a);
    if (std::min({a.nx, a.ny, a.nz}) <= min_coarse || std::min({b.nx, b.ny, b.nz}) < 3) break;
    MgLevel L;
    L.d = b;
    L.fixed.alloc(b.n(), c.s);
    L.val.alloc(b.n(), c.s);
    launch_coarsen_mask(c.s, lv.back().fixed.p, lv.back().val.p, a, L.fixed.p, L.val.p, b);
    lv.push_back(std::move(L));
  }
  CK(cudaGetLastError());
  return lv;
}

// ---------------------------------------------------------------- C-ABI glue
template <class F>
int guard(F&& f) {
  try {
    t_err.clear();
    return f();
  } catch (const Status& s) {
    t_err = s.what();
    return s.code;
  } catch (const std::exception& e) {
    t_err = e.what();
    return IG_CUDA_ERROR;
  }
}

cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// ig_solve3d on the values `b`.
int sor_call(const uint8_t* fixed, const Dirichlet& b, const float* theta, long nx, long ny,
             long nz, double tol, long max_sweeps, double omega, const double* phi0, int stencil,
             double* phi_out, long* sweeps_out, double* delta_out) {
  if (!fixed || !(b.val || b.mask) || !phi_out) throw Status(IG_BAD_ARG, "null array");
  ThreadCtx& c = ctx();
  const CallInFlight call(kSorCall);
  FineGrid g;
  load_fine(c, g, fixed, theta, nx, ny, nz, stencil);
  DirichletDev bd;
  init_phi(c, g, b, phi0, bd);
  DBuf<PairCtl> ctl(1, c.s);
  const PairsResult r = sor_loop(c, g.phi.p, g.fixed.p, g.th.p, g.plan, g.stencil, g.d, omega,
                                 tol, max_sweeps, ctl.p);
  copy_out(c, g.phi.p, phi_out, g.d.n());
  if (sweeps_out) *sweeps_out = r.pairs;
  if (delta_out) *delta_out = r.delta;
  if (!r.converged) {
    t_err = "SOR reached its sweep cap";
    return (int)IG_NOT_CONVERGED;
  }
  return (int)IG_OK;
}

// ig_solve3d_vmg on the values `b`.
int vmg_call(const uint8_t* fixed, const Dirichlet& b, const float* theta, long nx, long ny,
             long nz, double tol, int max_cycles, int nu1, int nu2, int stencil,
             const double* phi0, int accept_stagnation, double bottom_omega, double* phi_out,
             long* sweeps_out, double* delta_out, int* cycles_out, double* prev_delta_out) {
  if (!fixed || !(b.val || b.mask) || !phi_out) throw Status(IG_BAD_ARG, "null array");
  if (nu1 < 0 || nu2 < 0) throw Status(IG_BAD_ARG, "nu1 and nu2 must be >= 0");
  ThreadCtx& c = ctx();
  const CallInFlight call(kOtherCall);
  FineGrid g;
  load_fine(c, g, fixed, theta, nx, ny, nz, stencil);
  PageTouch touch(phi_out, g.d.n() * 8);
  std::vector<int> sym;
  {
    DirichletDev bd;
    init_phi(c, g, b, phi0, bd);
    if (!theta) sym = sym_axes(c, g, b, bd);
  }
  VCycle v;
  prepare_vcycle(c, v, g, nu1, nu2, bottom_omega);
  const VmgOut o = vmg_loop(c, g, v, tol, max_cycles, accept_stagnation, sym);
  touch.join();
  copy_out(c, g.phi.p, phi_out, g.d.n());
  if (sweeps_out) *sweeps_out = o.sweeps;
  if (delta_out) *delta_out = o.delta;
  if (cycles_out) *cycles_out = o.cycles;
  if (prev_delta_out) *prev_delta_out = o.prev;
  if (o.status != IG_OK) t_err = "V-cycle did not reach tol";
  return o.status;
}

}  // namespace
}  // namespace ig

using namespace ig;

void ig::set_last_error(const std::string& m) { t_err = m; }

ig::CallInFlight::CallInFlight(CallKind kind)
    : n_(kind == kSorCall ? &device_calls().sor : &device_calls().other) {
  n_->fetch_add(1);
}
ig::CallInFlight::~CallInFlight() { n_->fetch_sub(1); }

bool ig::device_range(const void* p, size_t bytes, size_t align) {
  cudaPointerAttributes a;
  int dev = -1;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  if (a.type != cudaMemoryTypeDevice || a.device != dev || at % align) return false;
  // CUDA's own record of the allocation's extent
  using RangeFn = int (*)(unsigned long long*, size_t*, unsigned long long);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult found;
  if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &fn, 3020, cudaEnableDefault,
                                       &found) != cudaSuccess ||
      found != cudaDriverEntryPointSuccess || !fn) {
    cudaGetLastError();
    return false;
  }
  unsigned long long base = 0;
  size_t size = 0;
  if (reinterpret_cast<RangeFn>(fn)(&base, &size, at) != 0) return false;
  return at >= base && at - base <= size && bytes <= size - (at - base);
}

int ig::call_stream(cudaStream_t* s) {
  return guard([&] {
    *s = ctx().s;
    return (int)IG_OK;
  });
}

extern "C" {

const char* ig_last_error(void) { return t_err.c_str(); }
int ig_abi_version(void) { return 2; }
int ig_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

void ig_request_stop(void) { g_stop.store(1); }
void ig_clear_stop(void) { g_stop.store(0); }
int ig_stop_requested(void) { return g_stop.load(); }

void ig_prof_enable(int on) { g_prof.on.store(on ? 1 : 0); }
void ig_prof_reset(void) {
  g_prof.ms = 0.0;
  g_prof.launches = 0;
  g_prof.nodes = 0;
}
long ig_launch_count(void) { return launch_total(); }
void ig_prof_read(double* ms, long* launches, long* nodes) {
  if (ms) *ms = g_prof.ms;
  if (launches) *launches = g_prof.launches;
  if (nodes) *nodes = g_prof.nodes;
}

int ig_solve3d(const uint8_t* fixed, const double* val, const float* theta,
               long nx, long ny, long nz, double tol, long max_sweeps,
               double omega, const double* phi0, int stencil, double* phi_out,
               long* sweeps_out, double* delta_out) {
  Dirichlet b;
  b.val = val;
  return guard([&] {
    return sor_call(fixed, b, theta, nx, ny, nz, tol, max_sweeps, omega, phi0, stencil, phi_out,
                    sweeps_out, delta_out);
  });
}

int ig_solve_basis_sor(const uint8_t* metal, const uint8_t* mask,
                       double v_basis, const float* theta, long nx, long ny,
                       long nz, double tol, long max_sweeps, double omega,
                       int stencil, double* phi_out, long* sweeps_out,
                       double* delta_out) {
  Dirichlet b;
  b.mask = mask;
  b.v = v_basis;
  return guard([&] {
    return sor_call(metal, b, theta, nx, ny, nz, tol, max_sweeps, omega, nullptr, stencil,
                    phi_out, sweeps_out, delta_out);
  });
}

int ig_solve3d_mg(const uint8_t* fixed, const double* val, const float* theta,
                  long nx, long ny, long nz, double tol, long max_sweeps,
                  int stencil, int min_coarse, int max_levels,
                  double level_tol_factor, const double* level_omega,
                  int n_level_omega, double* phi_out, long* sweeps_out,
                  double* delta_out) {
  return guard([&] {
    if (!fixed || !val || !phi_out) throw Status(IG_BAD_ARG, "null array");
    check_dims(nx, ny, nz);
    stencil_check(stencil);
    ThreadCtx& c = ctx();
    const CallInFlight call(kSorCall);
    const Dims d0{nx, ny, nz};
    std::vector<MgLevel> lv = build_mg_levels(c, fixed, val, d0, min_coarse, std::max(1, max_levels));
    const int nl = (int)lv.size();
    auto omega_of = [&](int L) {
      if (level_omega && L < n_level_omega) return level_omega[L];
      return optimal_omega_libm(lv[L].d);
    };
    DBuf<PairCtl> ctl(1, c.s);
    DBuf<float> th_d;
    Theta plan;
    const Theta none;
    if (theta) {
      th_d.alloc(6 * d0.n(), c.s);
      CK(cudaMemcpyAsync(th_d.p, theta, 6 * d0.n() * 4, cudaMemcpyDefault, c.s));
      plan_theta(c, plan, th_d, lv[0].fixed.p, d0, stencil);
    }
    // coarsest level: cold solve with theta None (multigrid3d.py:200-204);
    // then each finer level from the prolongated guess (multigrid3d.py:206-226)
    DBuf<double> cur;
    Dims cd{0, 0, 0};
    for (int L = nl - 1; L >= 0; L--) {
      MgLevel& M = lv[L];
      const size_t n = M.d.n();
      DBuf<double> phi(n, c.s);
      if (L == nl - 1)
        CK(cudaMemsetAsync(phi.p, 0, n * 8, c.s));
      else
        launch_prolongate(c.s, cur.p, cd, phi.p, M.d);
      launch_set_fixed(c.s, phi.p, M.fixed.p, M.val.p, n);
      // the coarsest solve always uses the plain stencil; with a one-level
      // hierarchy the reference then solves the fine grid again from zero
      // with theta (multigrid3d.py:201-203, 220-226)
      const bool with_theta = L == 0 && nl > 1;
      const double ltol = (L == 0 || L == nl - 1) ? tol : tol * level_tol_factor;
      PairsResult r = sor_loop(c, phi.p, M.fixed.p, with_theta ? th_d.p : nullptr,
                               with_theta ? plan : none, stencil, M.d, omega_of(L), ltol,
                               max_sweeps, ctl.p);
      if (nl == 1 && r.converged && theta) {
        CK(cudaMemsetAsync(phi.p, 0, n * 8, c.s));
        launch_set_fixed(c.s, phi.p, M.fixed.p, M.val.p, n);
        r = sor_loop(c, phi.p, M.fixed.p, th_d.p, plan, stencil, M.d, omega_of(0),
                     tol, max_sweeps, ctl.p);
      }
      if (!r.converged || L == 0) {
        if (sweeps_out) *sweeps_out = r.pairs;
        if (delta_out) *delta_out = r.delta;
      }
      if (!r.converged) {
        if (L == 0) copy_out(c, phi.p, phi_out, n);
        t_err = "SOR reached its sweep cap on cascadic level " + std::to_string(L);
        return (int)IG_NOT_CONVERGED;
      }
      if (L == 0) {
        copy_out(c, phi.p, phi_out, n);
        return (int)IG_OK;
      }
      cur = std::move(phi);
      cd = M.d;
    }
    return (int)IG_OK;
  });
}

int ig_solve3d_vmg(const uint8_t* fixed, const double* val, const float* theta,
                   long nx, long ny, long nz, double tol, int max_cycles,
                   int nu1, int nu2, int stencil, const double* phi0,
                   int accept_stagnation, double bottom_omega, double* phi_out,
                   long* sweeps_out, double* delta_out, int* cycles_out,
                   double* prev_delta_out) {
  Dirichlet b;
  b.val = val;
  return guard([&] {
    return vmg_call(fixed, b, theta, nx, ny, nz, tol, max_cycles, nu1, nu2, stencil, phi0,
                    accept_stagnation, bottom_omega, phi_out, sweeps_out, delta_out, cycles_out,
                    prev_delta_out);
  });
}

int ig_solve_basis_vmg(const uint8_t* metal, const uint8_t* mask,
                       double v_basis, const float* theta, long nx, long ny,
                       long nz, double tol, int max_cycles, int nu1, int nu2,
                       int stencil, double bottom_omega, double* phi_out,
                       long* sweeps_out, double* delta_out, int* cycles_out,
                       double* prev_delta_out) {
  Dirichlet b;
  b.mask = mask;
  b.v = v_basis;
  return guard([&] {
    return vmg_call(metal, b, theta, nx, ny, nz, tol, max_cycles, nu1, nu2, stencil, nullptr, 0,
                    bottom_omega, phi_out, sweeps_out, delta_out, cycles_out, prev_delta_out);
  });
}

int ig_cascadic_relres(const uint8_t* fixed, const double* val, long nx,
                       long ny, long nz, double rel_tol, long max_sweeps,
                       int min_coarse, int max_levels, double level_tol_factor,
                       const double* level_omega, int n_level_omega,
                       int check_every, double* phi_out, long* sweeps_out,
                       double* relres_out, long* total_pairs_out,
                       int* levels_out) {
  return guard([&] {
    if (!fixed || !val || !phi_out) throw Status(IG_BAD_ARG, "null array");
    if (check_every < 1) throw Status(IG_BAD_ARG, "check_every must be >= 1");
    check_dims(nx, ny, nz);
    ThreadCtx& c = ctx();
    const CallInFlight call(kOtherCall);
    const Dims d0{nx, ny, nz};
    std::vector<MgLevel> lv = build_mg_levels(c, fixed, val, d0, min_coarse, std::max(1, max_levels));
    const int nl = (int)lv.size();
    if (levels_out) *levels_out = nl;
    DBuf<unsigned long long> red(2, c.s);
    DBuf<double> cur, nxt;
    Dims cd{0, 0, 0};
    long total = 0;
    const bool prof = g_prof.on.load() != 0;
    for (int L = nl - 1; L >= 0; L--) {
      MgLevel& M = lv[L];
      const size_t n = M.d.n();
      nxt.alloc(n, c.s);
      // ||b||: residual of the Dirichlet values with zeros elsewhere
      CK(cudaMemsetAsync(nxt.p, 0, n * 8, c.s));
      launch_set_fixed(c.s, nxt.p, M.fixed.p, M.val.p, n);
      CK(cudaMemsetAsync(red.p, 0, 16, c.s));
      launch_residual(c.s, nxt.p, M.fixed.p, nullptr, kPlain, M.d, nullptr, red.p);
      const double bnorm = read_absmax(c, red.p, false);
      if (L < nl - 1) {
        launch_prolongate(c.s, cur.p, cd, nxt.p, M.d);
        launch_set_fixed(c.s, nxt.p, M.fixed.p, M.val.p, n);
      }
      const double om = (level_omega && L < n_level_omega) ? level_omega[L] : optimal_omega_libm(M.d);
      const double ltol = (L == 0 || L == nl - 1) ? rel_tol : rel_tol * level_tol_factor;
      long pairs = 0;
      double rr = std::numeric_limits<double>::infinity();
      while (true) {
        CK(cudaMemsetAsync(red.p, 0, 16, c.s));
        launch_residual(c.s, nxt.p, M.fixed.p, nullptr, kPlain, M.d, nullptr, red.p);
        const double rmax = read_absmax(c, red.p, false);
        rr = bnorm > 0 ? rmax / bnorm : rmax;
        if (rr < ltol || pairs >= max_sweeps) break;
        const int chunk = (int)std::min<long>(check_every, max_sweeps - pairs);
        if (prof) CK(cudaEventRecord(c.ev0, c.s));
        for (int q = 0; q < chunk; q++) {
          launch_sweep(c.s, nxt.p, M.fixed.p, nullptr, kPlain, M.d, om, 0, nullptr, nullptr, 0);
          launch_sweep(c.s, nxt.p, M.fixed.p, nullptr, kPlain, M.d, om, 1, nullptr, nullptr, 0);
        }
        CK(cudaGetLastError());
        if (prof) {
          CK(cudaEventRecord(c.ev1, c.s));
          CK(cudaEventSynchronize(c.ev1));
          float ms = 0.f;
          CK(cudaEventElapsedTime(&ms, c.ev0, c.ev1));
          g_prof.ms += ms;
          g_prof.launches += 2L * chunk;
          g_prof.nodes += (long)n * chunk;
        }
        pairs += chunk;
      }
      total += pairs;
      if (L == 0) {
        copy_out(c, nxt.p, phi_out, n);
        if (sweeps_out) *sweeps_out = pairs;
        if (relres_out) *relres_out = rr;
        if (total_pairs_out) *total_pairs_out = total;
        if (!(rr < ltol)) {
          t_err = "cascadic solve reached its sweep cap";
          return (int)IG_NOT_CONVERGED;
        }
        return (int)IG_OK;
      }
      cur = std::move(nxt);
      cd = M.d;
    }
    return (int)IG_OK;
  });
}

// ---- single kernels ----------------------------------------------------

namespace {
struct KScratch {
  int dev = -1;
  unsigned long long* d = nullptr;
};
thread_local KScratch t_ks;

unsigned long long* kscratch() {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (t_ks.dev != dev) {
    CK(cudaMalloc(&t_ks.d, 16));
    t_ks.dev = dev;
  }
  return t_ks.d;
}

double finish_max(cudaStream_t s, unsigned long long* slot) {
  unsigned long long b = 0;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(&b, slot, 8, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return bits_to_double(b);
}
}  // namespace

int ig_sweep_dev(double* phi, const uint8_t* fixed, const float* theta,
                 long nx, long ny, long nz, double omega, int colour,
                 int stencil, double* dmax_out, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    stencil_check(stencil);
    cudaStream_t s = as_stream(stream);
    unsigned long long* slot = kscratch();
    CK(cudaMemsetAsync(slot, 0, 8, s));
    launch_sweep(s, phi, fixed, theta, sweep_kind(theta != nullptr, stencil), Dims{nx, ny, nz},
                 omega, colour & 1, slot, nullptr, 0);
    const double d = finish_max(s, slot);
    if (dmax_out) *dmax_out = d;
    return (int)IG_OK;
  });
}

int ig_residual_dev(const double* phi, const uint8_t* fixed, const float* theta,
                    long nx, long ny, long nz, int stencil, double* out,
                    void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    stencil_check(stencil);
    const int kind = theta ? sweep_kind(theta != nullptr, stencil) : (stencil == 0 ? kPlain : kPlainSWResid);
    launch_residual(as_stream(stream), phi, fixed, theta, kind, Dims{nx, ny, nz}, out, nullptr);
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_sweep_rhs_dev(double* e, const uint8_t* fixed, const double* f, long nx,
                     long ny, long nz, double omega, int colour,
                     double* dmax_out, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    cudaStream_t s = as_stream(stream);
    unsigned long long* slot = kscratch();
    CK(cudaMemsetAsync(slot, 0, 8, s));
    launch_sweep_rhs(s, e, fixed, f, Dims{nx, ny, nz}, omega, colour & 1, slot, nullptr, 0);
    const double d = finish_max(s, slot);
    if (dmax_out) *dmax_out = d;
    return (int)IG_OK;
  });
}

int ig_residual_rhs_dev(const double* e, const uint8_t* fixed, const double* f,
                        long nx, long ny, long nz, double* out, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    launch_residual_rhs(as_stream(stream), e, fixed, f, Dims{nx, ny, nz}, out);
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_restrict_fw_dev(const double* fine, long nx, long ny, long nz,
                       double* out, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    const Dims d{nx, ny, nz};
    launch_restrict(as_stream(stream), fine, d, out, coarse_of(d), 0);
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_prolong_add_dev(const double* coarse, long cx, long cy, long cz,
                       double* out, const uint8_t* fixed, long nx, long ny,
                       long nz, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    check_dims(cx, cy, cz);
    launch_prolong_add(as_stream(stream), coarse, Dims{cx, cy, cz}, out, fixed, Dims{nx, ny, nz});
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_prolongate_dev(const double* coarse, long cx, long cy, long cz,
                      double* out, long nx, long ny, long nz, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    check_dims(cx, cy, cz);
    launch_prolongate(as_stream(stream), coarse, Dims{cx, cy, cz}, out, Dims{nx, ny, nz});
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_coarsen_fixed_any_dev(const uint8_t* fixed, long nx, long ny, long nz,
                             uint8_t* out, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    const Dims d{nx, ny, nz};
    launch_coarsen_any(as_stream(stream), fixed, d, out, coarse_of(d));
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_coarsen_mask_dev(const uint8_t* fixed, const double* val, long nx,
                        long ny, long nz, uint8_t* fc, double* vc,
                        void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    const Dims d{nx, ny, nz};
    launch_coarsen_mask(as_stream(stream), fixed, val, d, fc, vc, coarse_of(d));
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_residual_audit_dev(const double* u, const uint8_t* fixed,
                          const float* theta, long nx, long ny, long nz,
                          double* out, void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    if (nx < 2 || ny < 2 || nz < 2)
      throw Status(IG_BAD_ARG, "the audit residual needs every axis >= 2");
    if (!theta) throw Status(IG_BAD_ARG, "the audit residual needs theta");
    launch_residual_audit(as_stream(stream), u, fixed, theta, Dims{nx, ny, nz}, out);
    CK(cudaGetLastError());
    return (int)IG_OK;
  });
}

int ig_err_sweep_dev(double* e, const uint8_t* fixed, const float* theta,
                     const double* rhs, long nx, long ny, long nz,
                     double omega, int colour, double* dmax_out,
                     void* stream) {
  return guard([&] {
    check_dims(nx, ny, nz);
    if (nx < 2 || ny < 2 || nz < 2)
      throw Status(IG_BAD_ARG, "the error sweep needs every axis >= 2");
    if (!theta) throw Status(IG_BAD_ARG, "the error sweep needs theta");
    cudaStream_t s = as_stream(stream);
    unsigned long long* slot = kscratch();
    CK(cudaMemsetAsync(slot, 0, 8, s));
    launch_err_sweep(s, e, fixed, theta, rhs, Dims{nx, ny, nz}, omega, colour & 1, slot);
    const double d = finish_max(s, slot);
    if (dmax_out) *dmax_out = d;
    return (int)IG_OK;
  });
}

}  // extern "C"

extern "C" long long ig_device_free_bytes(void) {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return 0;
  }
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return (long long)free_b;
}
