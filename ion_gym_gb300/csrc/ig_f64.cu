// ig_f64.cu -- exact FP64 kernels of the 3-D Laplace solve on sm_103a.
//
// Each kernel returns the bits the reference's compiled float64 kernels
// return on the same input (ion_gym physics/solver3d.py and
// physics/multigrid3d.py, cited per kernel).  FP64 is the scarce pipe on
// GB300 (about 1/64 of the FP32 rate), so the kernels spend it only where the
// reference does: masks, indices, maxima and absolute values run on the
// integer pipe, and the theta == 1 stencil divides by 6 on the integer pipe
// (ig::div6) instead of a full division and the relaxation step runs there
// too (ig::sor_apply).
//
// Layout: C-order (nx, ny, nz), z contiguous; theta (6, nx, ny, nz) float32.
// Sweeps map one thread to one (i, j, k-pair) cell so a warp reads 64
// consecutive doubles of a row and every lane does useful FP64 work; the
// flattened index is split with 32-bit multiplicative division.
#include <algorithm>
#include <atomic>
#include <mutex>

#include <cooperative_groups.h>

#include "ig_common.cuh"
#include "ig_internal.h"

namespace ig {

std::atomic<long> g_launches{0};
long launch_total() { return g_launches.load(); }
static thread_local long t_launches = 0;
long launch_total_thread() { return t_launches; }
void note_launches(long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

namespace {

constexpr int kThreads = 256;

inline void counted() {
  t_launches++;
  g_launches.fetch_add(1, std::memory_order_relaxed);
}

__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
  return (__umulhi(n, f.m) + n) >> f.s;
}

struct SweepGeom {
  long nx, ny, nz;
  FastDiv div_kk, div_ny;
  uint32_t total;  // ceil(nx/U)*ny*nkk threads
};

// U: consecutive x-planes per thread.
inline SweepGeom sweep_geom(Dims d, int U = 1) {
  SweepGeom g;
  g.nx = d.nx;
  g.ny = d.ny;
  g.nz = d.nz;
  const long nkk = (d.nz + 1) / 2;
  g.div_kk = FastDiv((uint32_t)nkk);
  g.div_ny = FastDiv((uint32_t)d.ny);
  g.total = (uint32_t)((d.nx + U - 1) / U * d.ny * nkk);
  return g;
}

// Planes per sweep thread: 2 where the colour still fills the GPU's threads
// (152 SMs x 2048) with half as many, else 1 (a small level waits for its
// loads, and more threads have more of them in flight).  The 257^3
// quadrupole's cascadic solve with 1 / 2 / 4 planes on its large levels: 249
// / 243 / 303 ms (four planes leave too few warps).
inline int sweep_planes(Dims d) {
  return d.nx * d.ny * ((d.nz + 1) / 2) >= 2L * 152 * 2048 ? 2 : 1;
}

// Threads per block of the sweeps: the pipe-bound blocks of 256 run in step
// (all in their loads, then all in their sums); the same solve with 64 / 128
// / 256 threads: 244 / 243 / 254 ms.
constexpr int kSweepThreads = 128;
inline unsigned sweep_blocks(const SweepGeom& g) {
  return (g.total + kSweepThreads - 1) / kSweepThreads;
}

struct FlatGeom {
  long nx, ny, nz;
  FastDiv div_nz, div_ny;
  uint32_t total;
};

inline FlatGeom flat_geom(Dims d) {
  FlatGeom g;
  g.nx = d.nx;
  g.ny = d.ny;
  g.nz = d.nz;
  g.div_nz = FastDiv((uint32_t)d.nz);
  g.div_ny = FastDiv((uint32_t)d.ny);
  g.total = (uint32_t)d.n();
  return g;
}

inline unsigned blocks_for(size_t n) {
  return (unsigned)((n + kThreads - 1) / kThreads);
}

// Early-exit test of the exact SOR loop (PairCtl in ig_internal.h).  Uniform
// over the block, so a returning block skips the block reduction as a whole.
__device__ __forceinline__ bool pair_skip(PairCtl* ctl, int colour, int lp) {
  volatile PairCtl* c = ctl;
  if (c->done) return true;
  if (lp >= c->limit) return true;
  if (colour == 0) {
    unsigned long long a = 0, b = 0;
    bool have = false;
    if (lp > 0) {
      a = c->slot[2 * lp - 2];
      b = c->slot[2 * lp - 1];
      have = true;
    } else if (c->has_prev) {
      a = c->prev[0];
      b = c->prev[1];
      have = true;
    }
    if (have) {
      const double d = bits_to_double(a > b ? a : b);
      if (d < c->tol) {
        if (blockIdx.x == 0 && threadIdx.x == 0) c->done = 1;
        return true;
      }
    }
  }
  return false;
}

// Node indices fit 32 bits (grids are below 2^31 nodes).
struct Nb {
  uint32_t xm, xp, ym, yp, zm, zp;
};

// The six neighbours of node p = (i, j, k) as offsets from p, with the
// even-reflection rule at the faces (the ghost at -1 is node 1, the ghost at
// n is node n-2; a size-1 axis uses the node itself) as selects, so the
// interior and the faces run the same instructions.
__device__ __forceinline__ Nb neighbours(uint32_t i, uint32_t j, uint32_t k, uint32_t nx,
                                         uint32_t ny, uint32_t nz) {
  const uint32_t sy = nz, sx = ny * nz;
  const uint32_t p = (i * ny + j) * nz + k;
  const uint32_t rx = nx > 1 ? sx : 0u, ry = ny > 1 ? sy : 0u, rz = nz > 1 ? 1u : 0u;
  Nb n;
  n.xm = i > 0 ? p - sx : p + rx;
  n.xp = i + 1 < nx ? p + sx : p - rx;
  n.ym = j > 0 ? p - sy : p + ry;
  n.yp = j + 1 < ny ? p + sy : p - ry;
  n.zm = k > 0 ? p - 1 : p + rz;
  n.zp = k + 1 < nz ? p + 1 : p - rz;
  return n;
}

// The stencil weights of one node exactly as the reference forms them
// (solver3d.py:169-191, multigrid3d.py:329-353): ghost_linear w[d] =
// 1/theta_d and their sum; sw the products a neighbour's value is divided
// by (float32, as the compiled reference types them) and den.
template <int KIND>
__device__ __forceinline__ double theta_weights(const float t[6], double w[6]) {
  if (KIND == kThetaGhost) {
#pragma unroll
    for (int d = 0; d < 6; d++) w[d] = __drcp_rn((double)t[d]);
    return __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(w[0], w[1]), w[2]), w[3]), w[4]),
                     w[5]);
  }
  const float sx = __fadd_rn(t[0], t[1]), sy = __fadd_rn(t[2], t[3]), sz = __fadd_rn(t[4], t[5]);
  w[0] = (double)__fmul_rn(t[0], sx);
  w[1] = (double)__fmul_rn(t[1], sx);
  w[2] = (double)__fmul_rn(t[2], sy);
  w[3] = (double)__fmul_rn(t[3], sy);
  w[4] = (double)__fmul_rn(t[4], sz);
  w[5] = (double)__fmul_rn(t[5], sz);
  const double px = __drcp_rn((double)__fmul_rn(t[0], t[1]));
  const double py = __drcp_rn((double)__fmul_rn(t[2], t[3]));
  const double pz = __drcp_rn((double)__fmul_rn(t[4], t[5]));
  return __dadd_rn(__dadd_rn(px, py), pz);
}

// num of the theta-weighted stencil from those weights.
template <int KIND>
__device__ __forceinline__ double theta_num(const double v[6], const double w[6]) {
  double num = KIND == kThetaGhost ? __dmul_rn(v[0], w[0]) : __ddiv_rn(v[0], w[0]);
#pragma unroll
  for (int d = 1; d < 6; d++)
    num = __dadd_rn(num, KIND == kThetaGhost ? __dmul_rn(v[d], w[d]) : __ddiv_rn(v[d], w[d]));
  return num;
}

template <int KIND>
__device__ __forceinline__ void theta_num_den(const double v[6],
                                              const float* __restrict__ th,
                                              size_t N, size_t p, double& num,
                                              double& den) {
  float t[6];
  double w[6];
#pragma unroll
  for (int d = 0; d < 6; d++) t[d] = th[d * N + p];
  den = theta_weights<KIND>(t, w);
  num = theta_num<KIND>(v, w);
}

__device__ __forceinline__ double sum6(const double v[6]) {
  return __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(v[0], v[1]), v[2]), v[3]), v[4]), v[5]);
}

// CG: the value comes from L2, for data that other SMs write within the
// same kernel.
template <bool CG>
__device__ __forceinline__ double ldv(const double* a, size_t o) {
  return CG ? __ldcg(a + o) : a[o];
}

template <bool CG = false>
__device__ __forceinline__ void load6(const double* __restrict__ a, const Nb& n,
                                      double v[6]) {
  v[0] = ldv<CG>(a, n.xm);
  v[1] = ldv<CG>(a, n.xp);
  v[2] = ldv<CG>(a, n.ym);
  v[3] = ldv<CG>(a, n.yp);
  v[4] = ldv<CG>(a, n.zm);
  v[5] = ldv<CG>(a, n.zp);
}

// The nodes of one colour a sweep thread owns: the same y, z slot kk and U
// consecutive x-planes (the colour's node alternates between k = 2 kk and
// 2 kk + 1), so that one index split and one pair of y-neighbour offsets
// serve U nodes.
template <int U>
struct SweepNodes {
  uint32_t i0, j, kk, par, sx;
  int ym, yp;  // y-neighbours, relative
  uint32_t nx, nz;
  __device__ __forceinline__ SweepNodes(const SweepGeom& g, uint32_t t, int colour) {
    const uint32_t ij = fdiv(t, g.div_kk), ny = (uint32_t)g.ny;
    nx = (uint32_t)g.nx;
    nz = (uint32_t)g.nz;
    kk = t - ij * g.div_kk.d;
    const uint32_t ib = fdiv(ij, g.div_ny);
    j = ij - ib * g.div_ny.d;
    i0 = ib * U;
    par = (i0 + j + (uint32_t)colour) & 1u;
    sx = ny * nz;
    const int ry = ny > 1 ? (int)nz : 0;
    ym = j > 0 ? -(int)nz : ry;
    yp = j + 1 < ny ? (int)nz : -ry;
  }
  __device__ __forceinline__ uint32_t k(int u) const { return 2 * kk + (par ^ (u & 1)); }
  __device__ __forceinline__ bool valid(int u) const { return i0 + u < nx && k(u) < nz; }
  __device__ __forceinline__ uint32_t at(int u) const {
    return (i0 + u) * sx + j * nz + k(u);
  }
  __device__ __forceinline__ Nb nb(int u, uint32_t p) const {
    const uint32_t i = i0 + u, kz = k(u);
    const uint32_t rx = nx > 1 ? sx : 0u, rz = nz > 1 ? 1u : 0u;
    Nb n;
    n.xm = i > 0 ? p - sx : p + rx;
    n.xp = i + 1 < nx ? p + sx : p - rx;
    n.ym = p + ym;
    n.yp = p + yp;
    n.zm = kz > 0 ? p - 1 : p + rz;
    n.zp = kz + 1 < nz ? p + 1 : p - rz;
    return n;
  }
};

// solver3d._sweep (solver3d.py:131-198).  ONE: omega is 1.
template <int KIND, bool CTL, bool DELTA, bool ONE, int U>
__global__ void __launch_bounds__(kSweepThreads)
k_sweep(double* __restrict__ phi, const uint8_t* __restrict__ fixed,
        const float* __restrict__ th, SweepGeom g, double omega, int colour,
        unsigned long long* dslot, PairCtl* ctl, int lp) {
  if (CTL) {
    if (pair_skip(ctl, colour, lp)) return;
    dslot = &ctl->slot[2 * lp + colour];
  }
  const uint32_t t = blockIdx.x * kSweepThreads + threadIdx.x;
  unsigned long long mb = 0;
  if (t < g.total) {
    const SweepNodes<U> sn(g, t, colour);
    bool go[U];
    double q[U], old[U];
#pragma unroll
    for (int u = 0; u < U; u++) go[u] = sn.valid(u) && !fixed[sn.at(u)];
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (!go[u]) continue;
      const uint32_t p = sn.at(u);
      double v[6];
      load6(phi, sn.nb(u, p), v);
      old[u] = phi[p];
      if (KIND == kPlain) {
        q[u] = sum6(v);
      } else {
        double num, den;
        theta_num_den<KIND>(v, th, (size_t)g.nx * g.ny * g.nz, p, num, den);
        q[u] = __ddiv_rn(num, den);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (!go[u]) continue;
      unsigned long long key = 0;
      phi[sn.at(u)] = sor_apply<DELTA, ONE>(old[u], KIND == kPlain ? div6(q[u]) : q[u], omega,
                                            &key);
      if (DELTA && key > mb) mb = key;
    }
  }
  // without a slot (DELTA false) nobody reads the max |update|: skip it and
  // the block reduction
  if (DELTA) block_max_to(mb, dslot);
}

// multigrid3d._residual (multigrid3d.py:305-354): num - den*phi, 0 at fixed.
// A thread owns the nodes (i0 .. i0 + U - 1, j, k): its x-neighbours are its
// own column, so U nodes take 5 U + 2 loads and one index split.
constexpr int kResidPlanes = 4;
template <int KIND>
__global__ void __launch_bounds__(kSweepThreads)
k_residual(const double* __restrict__ phi, const uint8_t* __restrict__ fixed,
           const float* __restrict__ th, FlatGeom g, double* __restrict__ out,
           unsigned long long* absmax) {
  constexpr int U = kResidPlanes;
  const uint32_t t = blockIdx.x * kSweepThreads + threadIdx.x;
  const uint32_t nx = (uint32_t)g.nx, ny = (uint32_t)g.ny, nz = (uint32_t)g.nz;
  unsigned long long mb = 0;
  const uint32_t ij = fdiv(t, g.div_nz);
  const uint32_t k = t - ij * g.div_nz.d;
  const uint32_t ib = fdiv(ij, g.div_ny);
  const uint32_t j = ij - ib * g.div_ny.d;
  const uint32_t i0 = ib * U;
  if (i0 < nx) {
    const Nb n = neighbours(i0, j, k, nx, ny, nz);
    const uint32_t sx = ny * nz, p0 = i0 * sx + j * nz + k;
    double c[U + 2];
    c[0] = phi[n.xm];
#pragma unroll
    for (int u = 0; u <= U; u++) {
      const uint32_t i = i0 + u;  // past the last plane: the reflected one
      c[u + 1] = i < nx ? phi[p0 + u * sx] : (i == nx ? phi[nx > 1 ? p0 + (u - 2) * sx : p0] : 0.0);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (i0 + u >= nx) break;
      const uint32_t o = u * sx, p = p0 + o;
      double r = 0.0;
      if (!fixed[p]) {
        const double v[6] = {c[u], c[u + 2], phi[n.ym + o], phi[n.yp + o], phi[n.zm + o],
                             phi[n.zp + o]};
        if (KIND == kPlain) {
          r = resid6(sum6(v), c[u + 1]);
        } else if (KIND == kPlainSW) {
          // unit legs: num = sum of v/2 (== sum/2 exactly), den = 3
          r = __dsub_rn(__dmul_rn(sum6(v), 0.5), __dmul_rn(3.0, c[u + 1]));
        } else {
          double num, den;
          theta_num_den<KIND>(v, th, (size_t)nx * ny * nz, p, num, den);
          r = __dsub_rn(num, __dmul_rn(den, c[u + 1]));
        }
      }
      if (out) out[p] = r;
      const unsigned long long key = absbits(r);
      if (key > mb) mb = key;
    }
  }
  if (absmax) block_max_to(mb, absmax);
}

// ---- theta solves by a plan -----------------------------------------------
//
// The general theta kernels spend 6 reciprocals (ghost_linear) or 6
// divisions and 3 reciprocals (sw) on every node, although only nodes beside
// a surface have a leg shorter than 1 (0.4 % of a 57 x 71 x 90 deck).  The
// FP64 pipe bounds them (2 lanes per clock and SM): 43 us a half-sweep on
// that deck, either stencil.  A solve therefore sorts its nodes once:
// nodes with six unit legs take the plain update, whose result is the
// general one's -- ghost_linear: every weight is 1 and den 6; sw: every
// product is 2 and den 3, and halving commutes with rounding unless
// something is subnormal or overflows, where plain_sw_num takes the
// divisions as written -- and the cut nodes are listed by colour with their
// weights.  One launch does both: the first blocks the list, the rest the
// grid; nodes of one colour do not read each other.

// num / den of a node with six unit legs under sw, as the general kernel
// evaluates it.
__device__ __noinline__ double plain_sw_num(const double v[6]) {
  double num = __ddiv_rn(v[0], 2.0);
  for (int d = 1; d < 6; d++) num = __dadd_rn(num, __ddiv_rn(v[d], 2.0));
  return num;
}

// Whether sum6's S of the values v may be halved after the fact: |S| >=
// 2^-900 and finite (values small enough for v / 2 to round are below
// 2^-1021 and vanish in such a sum, halved or not), or every value is zero.
__device__ __forceinline__ bool sw_halves(double S, const double v[6]) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(S));
  const unsigned eb = static_cast<unsigned>(b >> 52) & 0x7ffu;
  if (eb - 123u <= 2040u - 123u) return true;
  unsigned long long any = 0;
#pragma unroll
  for (int d = 0; d < 6; d++) any |= static_cast<unsigned long long>(__double_as_longlong(v[d]));
  return (any << 1) == 0ULL;
}

__global__ void __launch_bounds__(kThreads)
k_theta_class(const uint8_t* __restrict__ fixed, const float* __restrict__ th, FlatGeom g,
              uint8_t* __restrict__ cls, uint32_t* counts) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  int cut = -1;  // the colour of a cut node
  if (t < g.total) {
    uint8_t c = 1;
    if (!fixed[t]) {
      bool unit = true;
#pragma unroll
      for (int d = 0; d < 6; d++) unit = unit && th[(size_t)d * g.total + t] == 1.0f;
      c = unit ? 0 : 2;
    }
    cls[t] = c;
    if (c == 2) {
      const uint32_t ij = fdiv(t, g.div_nz);
      const uint32_t i = fdiv(ij, g.div_ny);
      cut = (int)((i + (ij - i * g.div_ny.d) + (t - ij * g.div_nz.d)) & 1u);
    }
  }
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const int n = __syncthreads_count(cut == c);
    if (threadIdx.x == 0 && n) atomicAdd(counts + c, (uint32_t)n);
  }
}

// The list position of a cut node comes from an atomic counter: the order of
// a colour's nodes in the list changes no result.
template <int KIND>
__global__ void __launch_bounds__(kThreads)
k_theta_fill(const uint8_t* __restrict__ cls, const float* __restrict__ th, FlatGeom g,
             uint32_t n0, uint32_t total, uint32_t* cursor, uint32_t* __restrict__ idx,
             double* __restrict__ w) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= g.total || cls[t] != 2) return;
  const uint32_t ij = fdiv(t, g.div_nz);
  const uint32_t i = fdiv(ij, g.div_ny);
  const uint32_t c = (i + (ij - i * g.div_ny.d) + (t - ij * g.div_nz.d)) & 1u;
  const uint32_t e = (c ? n0 : 0u) + atomicAdd(cursor + c, 1u);
  float tv[6];
  double wv[6];
#pragma unroll
  for (int d = 0; d < 6; d++) tv[d] = th[(size_t)d * g.total + t];
  const double den = theta_weights<KIND>(tv, wv);
  idx[e] = t;
#pragma unroll
  for (int d = 0; d < 6; d++) w[(size_t)d * total + e] = wv[d];
  w[(size_t)6 * total + e] = den;
}

// Node e of the cut list: its index, neighbour values and weights.
template <int KIND>
__device__ __forceinline__ uint32_t cut_node(const double* __restrict__ phi,
                                             const ThetaPlan& P, uint32_t e, const FastDiv& dnz,
                                             const FastDiv& dny, uint32_t nx, double& num,
                                             double& den) {
  const uint32_t p = P.idx[e], total = P.total();
  const uint32_t ij = fdiv(p, dnz);
  const uint32_t i = fdiv(ij, dny);
  const Nb n = neighbours(i, ij - i * dny.d, p - ij * dnz.d, nx, dny.d, dnz.d);
  double v[6], w[6];
  load6(phi, n, v);
#pragma unroll
  for (int d = 0; d < 6; d++) w[d] = P.w[(size_t)d * total + e];
  den = P.w[(size_t)6 * total + e];
  num = theta_num<KIND>(v, w);
  return p;
}

// One colour of the theta sweep (k_sweep<KIND>'s bits).  Whole solves, the
// general kernels against the plan (GB300): solve3d, sw, 57 x 71 x 90 with
// 0.4 % cut nodes 22.6 -> 7.6 ms; the basis door, ghost_linear, four bases of
// a 65 x 65 x 129 ring deck 71.5 -> 49.3 ms.
template <int KIND, bool CTL, bool DELTA, bool ONE>
__global__ void __launch_bounds__(kThreads)
k_sweep_plan(double* __restrict__ phi, const ThetaPlan P, SweepGeom g, FastDiv dnz,
             uint32_t list_blocks, double omega, int colour, unsigned long long* dslot,
             PairCtl* ctl, int lp) {
  if (CTL) {
    if (pair_skip(ctl, colour, lp)) return;
    dslot = &ctl->slot[2 * lp + colour];
  }
  unsigned long long mb = 0;
  uint32_t p = 0xffffffffu;
  double q = 0.0;
  if (blockIdx.x < list_blocks) {
    const uint32_t e = blockIdx.x * kThreads + threadIdx.x;
    if (e < P.count[colour]) {
      double num, den;
      p = cut_node<KIND>(phi, P, (colour ? P.count[0] : 0u) + e, dnz, g.div_ny,
                         (uint32_t)g.nx, num, den);
      q = __ddiv_rn(num, den);
    }
  } else {
    const uint32_t t = (blockIdx.x - list_blocks) * kThreads + threadIdx.x;
    if (t < g.total) {
      const uint32_t ij = fdiv(t, g.div_kk);
      const uint32_t kk = t - ij * g.div_kk.d;
      const uint32_t i = fdiv(ij, g.div_ny);
      const uint32_t j = ij - i * g.div_ny.d;
      const uint32_t k = 2 * kk + ((i + j + colour) & 1);
      const uint32_t o = (i * (uint32_t)g.ny + j) * (uint32_t)g.nz + k;
      if (k < (uint32_t)g.nz && P.cls[o] == 0) {
        const Nb n = neighbours(i, j, k, g.nx, g.ny, g.nz);
        double v[6];
        load6(phi, n, v);
        const double S = sum6(v);
        p = o;
        if (KIND == kThetaSW && !sw_halves(S, v))
          q = __ddiv_rn(plain_sw_num(v), 3.0);
        else
          q = div6(S);
      }
    }
  }
  if (p != 0xffffffffu) {
    const double old = phi[p];
    phi[p] = sor_apply<DELTA, ONE>(old, q, omega, &mb);
  }
  if (DELTA) block_max_to(mb, dslot);
}

// The fine residual num - den phi (k_residual<KIND>'s bits).
template <int KIND>
__global__ void __launch_bounds__(kThreads)
k_residual_plan(const double* __restrict__ phi, const ThetaPlan P, FlatGeom g,
                uint32_t list_blocks, double* __restrict__ out) {
  if (blockIdx.x < list_blocks) {
    const uint32_t e = blockIdx.x * kThreads + threadIdx.x;
    if (e >= P.total()) return;
    double num, den;
    const uint32_t p = cut_node<KIND>(phi, P, e, g.div_nz, g.div_ny, (uint32_t)g.nx, num, den);
    out[p] = __dsub_rn(num, __dmul_rn(den, phi[p]));
    return;
  }
  const uint32_t t = (blockIdx.x - list_blocks) * kThreads + threadIdx.x;
  if (t >= g.total) return;
  const uint8_t c = P.cls[t];
  if (c == 2) return;  // the list's
  double r = 0.0;
  if (c == 0) {
    const uint32_t ij = fdiv(t, g.div_nz);
    const uint32_t i = fdiv(ij, g.div_ny);
    const Nb n = neighbours(i, ij - i * g.div_ny.d, t - ij * g.div_nz.d, g.nx, g.ny, g.nz);
    double v[6];
    load6(phi, n, v);
    const double S = sum6(v);
    if (KIND == kThetaGhost)
      r = resid6(S, phi[t]);
    else if (sw_halves(S, v))
      r = __dsub_rn(__dmul_rn(S, 0.5), __dmul_rn(3.0, phi[t]));
    else
      r = __dsub_rn(plain_sw_num(v), __dmul_rn(3.0, phi[t]));
  }
  out[t] = r;
}

// ---- SOR to its tolerance in one launch ------------------------------------
//
// A grid of some 10^5 nodes is 1.4 us of FP64 work a half-sweep, and a
// launch 7 us of latency around it (control block, mask, values, sum, block
// maximum, each waiting for the one before; 43 us with theta's divisions on
// the last block's chain).  Here one CTA per SM stays for as many pairs as the
// call's turn has (a cooperative launch, so that all of them are resident).  The node arithmetic
// is the launched sweeps'.
//
// A grid barrier after each half-sweep would be four trips to L2 one after
// the other (the values' stores, the arrival, the poll, the next loads), 4000
// clocks at 65^3 beside 7500 of work that all warps do in step, the FP64 pipe
// idle while they are in the integer part.  So there is none: a node's value
// travels with its version, the number of updates it has had, in one 16-byte
// word (a 128-bit access is single).  Colour 0 of pair n takes colour-1
// neighbours of version n, colour 1 colour-0 ones of version n + 1, each lane
// waiting for its own six.  No node can get further ahead: its next update
// waits for neighbours that have read it.  So every CTA runs on as its own
// neighbours allow.
//
// The reference's test after each pair is made a pair late: a CTA publishes
// its maximum of pair n and goes on, and at the end of pair n + 1 reads all
// of pair n; when that met tol, pair n + 1 is undone (prev holds each node's
// value before its last update).  All CTAs see the same maxima and stop
// alike.
//
// A CTA has an even share of the slots in a row; where a thread's neighbours
// lie is worked out once, into shared memory (1500 clocks a half-sweep of
// divisions and masks otherwise).  Words lie by colour and slot, so a warp's
// loads are contiguous.  A cut node of a theta plan goes to six lanes, one
// per leg (its division or product), and the lanes add the six in the
// reference's order: the FP64 pipe takes a warp's instruction as long for two
// lanes as for 32, so six legs side by side are a sixth of the divisions in
// line.
//
// What is left at 65^3 is a half-sweep's chain: the neighbours' words 0.8 us,
// sums and integer step 2.0 (28 warps an SM, FP64 alone 1.4).  solve3d at 65^3
// 4.73 ms launched, 2.75 with grid barriers, 1.78 with a block barrier a
// pair, 1.65 so; with theta (sw, 57 x 71 x 90) 22.5, 6.0, 3.3 and 2.95 (the
// cut nodes in warps of their own).
//
// Waits are bounded (kCoopWait clocks, seconds): a warp that gives up raises
// *status and leaves, the others follow, and the call reports an error.
constexpr long long kCoopWait = 8000000000LL;

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Every CTA of the grid; false when the wait was given up.
__device__ __forceinline__ bool coop_barrier(CoopCtl* c, unsigned target, int* ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&c->arrived, 1u);
    const long long t0 = clock64();
    int good = 1;
    for (unsigned polls = 1; ld_acquire(&c->arrived) < target; polls++) {
      if ((polls & 255u) == 0 &&
          (clock64() - t0 > kCoopWait || *reinterpret_cast<volatile int*>(&c->status))) {
        c->status = 1;
        good = 0;
        break;
      }
    }
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

constexpr size_t kFlowBytes = 20;  // of shared memory a slot
struct FlowGeom {
  SweepGeom g;
  FastDiv dnz;
  uint32_t share;    // slots a CTA
  uint32_t workers;  // threads that have them; the warps after have cut nodes alone
  int rounds;        // slots a worker
  ulonglong2* word;  // 2 * g.total
  double* prev;      // 2 * g.total
};

__device__ __forceinline__ void ld_word(const ulonglong2* p, unsigned long long& v,
                                        unsigned long long& n) {
  asm volatile("{ .reg .b128 w; ld.relaxed.gpu.global.b128 w, [%2]; mov.b128 {%0, %1}, w; }"
               : "=l"(v), "=l"(n) : "l"(p));
}
__device__ __forceinline__ void st_word(ulonglong2* p, unsigned long long v,
                                        unsigned long long n) {
  asm volatile("{ .reg .b128 w; mov.b128 w, {%1, %2}; st.relaxed.gpu.global.b128 [%0], w; }"
               ::"l"(p), "l"(v), "l"(n) : "memory");
}

// Polls until done() (every lane of the warp calls it); false: given up.
template <class F>
__device__ __forceinline__ bool flow_wait(CoopCtl* c, F&& done) {
  if (__all_sync(0xffffffffu, done())) return true;
  const long long t0 = clock64();
  for (unsigned polls = 1; !__all_sync(0xffffffffu, done()); polls++)
    if ((polls & 255u) == 0 &&
        __any_sync(0xffffffffu, clock64() - t0 > kCoopWait ||
                                    *reinterpret_cast<volatile int*>(&c->status))) {
      c->status = 1;
      return false;
    }
  return true;
}

// A node of colour c at slot t = (row ij, kk): its k and its neighbours' slots
// of the other colour (t itself along a size-1 axis).
struct FlowNode {
  uint32_t k, o, t[6];
};
__device__ __forceinline__ FlowNode flow_node(const FlowGeom& G, uint32_t t, int c) {
  const uint32_t nkk = G.g.div_kk.d, ny = G.g.div_ny.d;
  const uint32_t nx = (uint32_t)G.g.nx, nz = (uint32_t)G.g.nz;
  const uint32_t ij = fdiv(t, G.g.div_kk), kk = t - ij * nkk;
  const uint32_t i = fdiv(ij, G.g.div_ny), j = ij - i * ny;
  FlowNode f;
  f.k = 2 * kk + ((i + j + (uint32_t)c) & 1u);
  f.o = ij * nz + f.k;
  const uint32_t sx = ny * nkk, r = ij * nkk;
  const uint32_t rx = nx > 1 ? sx : 0u, ry = ny > 1 ? nkk : 0u;
  f.t[0] = i > 0 ? t - sx : t + rx;
  f.t[1] = i + 1 < nx ? t + sx : t - rx;
  f.t[2] = j > 0 ? t - nkk : t + ry;
  f.t[3] = j + 1 < ny ? t + nkk : t - ry;
  f.t[4] = r + ((f.k > 0 ? f.k - 1 : 1u) >> 1);
  f.t[5] = r + (nz == 1 ? 0u : (f.k + 1 < nz ? f.k + 1 : f.k - 1) >> 1);
  return f;
}

template <int KIND>
__global__ void __launch_bounds__(kCoopThreads, 1)
k_sor_flow(double* phi, const uint8_t* __restrict__ cls, const ThetaPlan P, FlowGeom G,
           double omega, double tol, int pairs, CoopCtl* ctl) {
  // this thread's slots: the x and y neighbours', and bits: plain of either
  // colour (0, 1), z neighbours' distances + 1 (two bits each from 2)
  extern __shared__ uint4 near_xy[];
  uint32_t* near_z = reinterpret_cast<uint32_t*>(near_xy + (size_t)G.rounds * G.workers);
  // pair n in slot n & 3: the warps' maxima and how many are in, whether a
  // warp reads the other CTAs', and the maximum of all once it is known
  __shared__ volatile unsigned long long red[4][32], all[4];
  __shared__ unsigned in[4], asked[4];
  __shared__ volatile unsigned known[4];
  __shared__ int ok;
  if (threadIdx.x < 4)
    in[threadIdx.x] = asked[threadIdx.x] = known[threadIdx.x] = 0;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
  const uint32_t nt = G.workers;
  const int rounds = threadIdx.x < nt ? G.rounds : 0;  // uniform over a warp
  const uint32_t S = G.g.total, nz = (uint32_t)G.g.nz;
  const unsigned same = (G.g.nx > 1 ? 0u : 3u) | (G.g.ny > 1 ? 0u : 12u) | (nz > 1 ? 0u : 48u);
  // slot r of this thread: t0 + r nt, below t1
  const uint32_t t0 = blockIdx.x * G.share + threadIdx.x;
  const uint32_t t1 = min(S, (blockIdx.x + 1) * G.share);
  const uint32_t cw = (uint32_t)(nw - 1 - wid) * gridDim.x + blockIdx.x;
  for (int r = 0; r < rounds; r++) {
    const uint32_t t = t0 + (uint32_t)r * nt;
    uint32_t bits = 0;
    for (int c = 0; c < 2 && t < t1; c++) {
      const FlowNode f = flow_node(G, t, c);
      unsigned long long v = 0, n = ~0ULL;
      if (f.k < nz) {
        v = static_cast<unsigned long long>(__double_as_longlong(phi[f.o]));
        const uint8_t k = cls[f.o];
        n = k == 0 || (KIND != kPlain && k == 2) ? 0ULL : ~0ULL;  // metal: any version
        bits |= (k == 0 ? 1u << c : 0u) | (f.t[4] - t + 1u) << (2 + 4 * c) |
                (f.t[5] - t + 1u) << (4 + 4 * c);
      }
      st_word(G.word + (size_t)c * S + t, v, n);
      near_xy[r * nt + threadIdx.x] = make_uint4(f.t[0], f.t[1], f.t[2], f.t[3]);
    }
    near_z[r * nt + threadIdx.x] = bits;
  }
  if (!coop_barrier(ctl, gridDim.x, &ok)) return;

  int pr = 0;
  bool hit = false, undo = false;
  unsigned long long key = 0;
  // all CTAs' maximum of pair q; false: given up
  auto maxima = [&](int q, unsigned long long* out) {
    unsigned long long m = 0;
    const bool good = flow_wait(ctl, [&] {
      m = 0;
      bool all = true;
      const ulonglong2* w = reinterpret_cast<const ulonglong2*>(ctl->word[q & 3]);
      for (uint32_t b0 = lane; b0 < gridDim.x; b0 += 160) {
        unsigned long long v[5], n[5];
#pragma unroll
        for (int d = 0; d < 5; d++) ld_word(w + min(b0 + 32 * d, gridDim.x - 1), v[d], n[d]);
#pragma unroll
        for (int d = 0; d < 5; d++) {
          m = max(m, v[d]);
          all = all && n[d] == (unsigned long long)(q + 1);
        }
      }
      return all;
    });
    *out = warp_max_u64(m);
    return good;
  };
  // the same, read from the others by the CTA's first warp to ask and from
  // shared memory by the rest
  auto maximum = [&](int q, unsigned long long* out) {
    const unsigned id = (unsigned)(q + 1);
    unsigned before = 0;
    if (lane == 0) before = atomicExch(&asked[q & 3], id);
    if (__shfl_sync(0xffffffffu, before, 0) != id) {
      if (!maxima(q, out)) return false;
      if (lane == 0) {
        all[q & 3] = *out;
        __threadfence_block();
        known[q & 3] = id;
      }
      return true;
    }
    if (!flow_wait(ctl, [&] {
          if (known[q & 3] == id) return true;
          __nanosleep(32);
          return false;
        }))
      return false;
    __threadfence_block();
    *out = all[q & 3];
    return true;
  };
  for (; pr < pairs && !hit; pr++) {
    unsigned long long mb = 0;
    for (int c = 0; c < 2; c++) {
      const unsigned long long want = (unsigned long long)(pr + c);
      ulonglong2* own = G.word + (size_t)c * S;
      const ulonglong2* oth = G.word + (size_t)(1 - c) * S;
      double* prev = G.prev + (size_t)c * S;
      if (KIND != kPlain) {
        // the cut nodes from the CTA's last warps on, which have fewer of the rest
        const uint32_t first = c ? P.count[0] : 0u, total = P.total();
        for (uint32_t q = cw * 5u; q < P.count[c]; q += gridDim.x * (uint32_t)nw * 5u) {
          const int who = lane / 6, leg = lane - 6 * who;
          const bool act = who < 5 && q + who < P.count[c];
          const uint32_t e = first + q + (act ? who : 0);
          const uint32_t p = P.idx[e], ij = fdiv(p, G.dnz);
          const uint32_t t = ij * G.g.div_kk.d + ((p - ij * nz) >> 1);
          const FlowNode f = flow_node(G, t, c);
          const bool self = (same >> leg) & 1u;
          uint32_t u = f.t[0];
#pragma unroll
          for (int d = 1; d < 6; d++) u = leg == d ? f.t[d] : u;
          const ulonglong2* src = self ? own + t : oth + u;
          unsigned long long vb, n, ob, on;
          ld_word(own + t, ob, on);
          const double w = P.w[(size_t)leg * total + e], den = P.w[(size_t)6 * total + e];
          bool have = false;
          if (!flow_wait(ctl, [&] {
                if (!have) {
                  ld_word(src, vb, n);
                  have = self || !act || n >= want;
                }
                return have;
              }))
            return;
          const int l0 = lane < 30 ? 6 * who : 24;
          // along an axis of one node a leg is the node itself: its value from
          // the lane that stored it (l0), since nothing orders this lane's own
          // read of the word behind that store
          const unsigned long long mine = __shfl_sync(0xffffffffu, ob, l0);
          const double v = __longlong_as_double((long long)(self ? mine : vb));
          const double old = __longlong_as_double((long long)mine);
          const double term = KIND == kThetaGhost ? __dmul_rn(v, w) : __ddiv_rn(v, w);
          double num = __shfl_sync(0xffffffffu, term, l0);
#pragma unroll
          for (int d = 1; d < 6; d++)
            num = __dadd_rn(num, __shfl_sync(0xffffffffu, term, l0 + d));
          unsigned long long k = 0;
          const double nv = sor_apply<true, false>(old, __ddiv_rn(num, den), omega, &k);
          if (act && leg == 0) {
            st_word(own + t, (unsigned long long)__double_as_longlong(nv), pr + 1ULL);
            prev[t] = old;
            if (k > mb) mb = k;
          }
        }
      }
      for (int r = 0; r < rounds; r++) {
        const uint32_t t = t0 + (uint32_t)r * nt;
        const uint4 xy = near_xy[r * nt + threadIdx.x];
        const uint32_t bits = near_z[r * nt + threadIdx.x] >> c;
        const bool go = bits & 1u;
        const uint32_t z = bits >> (2 + 3 * c);
        const uint32_t nt[6] = {xy.x, xy.y, xy.z, xy.w, t + (z & 3u) - 1u,
                                t + ((z >> 2) & 3u) - 1u};
        unsigned long long b[6], ob = 0, on;
        bool have = !go;
        if (go) ld_word(own + t, ob, on);
        if (!flow_wait(ctl, [&] {
              if (!have) {
                unsigned long long n[6];
#pragma unroll
                for (int d = 0; d < 6; d++) ld_word(oth + nt[d], b[d], n[d]);
                have = true;
#pragma unroll
                for (int d = 0; d < 6; d++) have = have && (n[d] >= want || ((same >> d) & 1u));
              }
              return have;
            }))
          return;
        if (!go) continue;
        double v[6];
#pragma unroll
        for (int d = 0; d < 6; d++)
          v[d] = __longlong_as_double((long long)((same >> d) & 1u ? ob : b[d]));
        const double old = __longlong_as_double((long long)ob), sum = sum6(v);
        double q;
        if (KIND == kThetaSW && !sw_halves(sum, v))
          q = __ddiv_rn(plain_sw_num(v), 3.0);
        else
          q = div6(sum);
        unsigned long long k = 0;
        const double nv = sor_apply<true, false>(old, q, omega, &k);
        st_word(own + t, (unsigned long long)__double_as_longlong(nv), pr + 1ULL);
        prev[t] = old;
        if (k > mb) mb = k;
      }
    }
    // this pair's maximum out, by the CTA's last warp, and the last pair's in
    mb = warp_max_u64(mb);
    unsigned before = 0;
    if (lane == 0) {
      red[pr & 3][wid] = mb;
      __threadfence_block();
      before = atomicAdd(&in[pr & 3], 1u);
      __threadfence_block();
    }
    // a slot's count goes up by nw every four pairs and is never reset
    if (__shfl_sync(0xffffffffu, before, 0) == (unsigned)(nw * (pr >> 2) + nw - 1)) {
      __syncwarp();
      mb = warp_max_u64(lane < nw ? red[pr & 3][lane] : 0ULL);
      if (lane == 0)
        st_word(reinterpret_cast<ulonglong2*>(ctl->word[pr & 3]) + blockIdx.x, mb, pr + 1ULL);
    }
    if (pr > 0) {
      if (!maximum(pr - 1, &key)) return;
      hit = undo = bits_to_double(key) < tol;
    }
  }
  if (!hit) {
    // the last pair's own test
    if (!maximum(pairs - 1, &key)) return;
    hit = bits_to_double(key) < tol;
  }
  auto put = [&](uint32_t o, uint32_t t, int c) {
    unsigned long long v, n;
    ld_word(G.word + (size_t)c * S + t, v, n);
    phi[o] = undo ? G.prev[(size_t)c * S + t] : __longlong_as_double((long long)v);
  };
  for (int c = 0; c < 2; c++) {
    if (KIND != kPlain) {
      for (uint32_t q = cw * 5u; q < P.count[c]; q += gridDim.x * (uint32_t)nw * 5u) {
        const int who = lane / 6;
        if (who < 5 && lane == 6 * who && q + who < P.count[c]) {
          const uint32_t p = P.idx[(c ? P.count[0] : 0u) + q + who], ij = fdiv(p, G.dnz);
          put(p, ij * G.g.div_kk.d + ((p - ij * nz) >> 1), c);
        }
      }
    }
    for (uint32_t t = t0; rounds && t < t1; t += nt) {
      const FlowNode f = flow_node(G, t, c);
      if (f.k < nz && cls[f.o] == 0) put(f.o, t, c);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->pairs = undo ? pr - 1 : pr;
    ctl->hit = hit ? 1 : 0;
    ctl->key = key;
  }
}

// multigrid3d._sweep_rhs (multigrid3d.py:357-391).  ONE: omega is 1.
template <bool CTL, bool DELTA, bool ONE, int U>
__global__ void __launch_bounds__(kSweepThreads)
k_sweep_rhs(double* __restrict__ e, const uint8_t* __restrict__ fixed,
            const double* __restrict__ f, SweepGeom g, double omega,
            int colour, unsigned long long* dslot, PairCtl* ctl, int lp) {
  if (CTL) {
    if (pair_skip(ctl, colour, lp)) return;
    dslot = &ctl->slot[2 * lp + colour];
  }
  const uint32_t t = blockIdx.x * kSweepThreads + threadIdx.x;
  unsigned long long mb = 0;
  if (t < g.total) {
    const SweepNodes<U> sn(g, t, colour);
    bool go[U];
    double q[U], old[U];
#pragma unroll
    for (int u = 0; u < U; u++) go[u] = sn.valid(u) && !fixed[sn.at(u)];
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (!go[u]) continue;
      const uint32_t p = sn.at(u);
      double v[6];
      load6(e, sn.nb(u, p), v);
      old[u] = e[p];
      q[u] = __dsub_rn(sum6(v), f[p]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (!go[u]) continue;
      unsigned long long key = 0;
      e[sn.at(u)] = sor_apply<DELTA, ONE>(old[u], div6(q[u]), omega, &key);
      if (DELTA && key > mb) mb = key;
    }
  }
  if (DELTA) block_max_to(mb, dslot);
}

// A level's values by (row, k), row the grid row's index ij = i ny + j: a
// flat array.
struct FlatRows {
  const double* __restrict__ a;
  uint32_t nz;
  typedef const double* Row;
  __device__ __forceinline__ Row row(uint32_t ij) const { return a + (size_t)ij * nz; }
  __device__ __forceinline__ double at(Row r, int k) const { return r[k]; }
};

// multigrid3d._restrict_fw_njit (multigrid3d.py:420-455) at coarse node
// (ic, jc, kc): 27-point full weighting with clamped edges, /8, and
// -4x when neg4 (the caller's scaling).
//
// The weights are powers of two, so RN(acc + RN(w x)) is one fused
// multiply-add as long as w x is exact: always, unless x is subnormal or
// within a factor of 8 of it (restrict_slow).  27 FP64 instructions a node
// instead of 54 on a pipe of 2 lanes per clock and SM: 8.9 -> 4.9 us a
// launch, averaged over a 97 x 97 x 193 deck's levels.
template <class A>
static __device__ __noinline__ double restrict_slow(const A fine, int nx, int ny, int nz, int i,
                                                    int j, int k) {
  double acc = 0.0;
  for (int di = -1; di <= 1; di++)
    for (int dj = -1; dj <= 1; dj++)
      for (int dk = -1; dk <= 1; dk++) {
        const int ii = min(max(i + di, 0), nx - 1), jj = min(max(j + dj, 0), ny - 1);
        const int kk = min(max(k + dk, 0), nz - 1);
        const double w = (di ? 0.5 : 1.0) * (dj ? 0.5 : 1.0) * (dk ? 0.5 : 1.0);
        acc = __dadd_rn(acc, __dmul_rn(w, fine.at(fine.row((uint32_t)(ii * ny + jj)), kk)));
      }
  return acc;
}

template <class A>
__device__ __forceinline__ double restrict_node(const A& fine, int nx, int ny, int nz, int ic,
                                                int jc, int kc, int neg4) {
  const int i = 2 * ic, j = 2 * jc, k = 2 * kc;
  const int km = max(k - 1, 0), kp = min(k + 1, nz - 1);
  double acc = 0.0;
  unsigned tiny = 0xffffffffu;  // smallest |x| key but for zeros
#pragma unroll
  for (int di = -1; di <= 1; di++) {
    const int ii = min(max(i + di, 0), nx - 1);
    const double wi = di == 0 ? 1.0 : 0.5;
#pragma unroll
    for (int dj = -1; dj <= 1; dj++) {
      const int jj = min(max(j + dj, 0), ny - 1);
      const double wj = dj == 0 ? 1.0 : 0.5;
      const typename A::Row row = fine.row((uint32_t)(ii * ny + jj));
      const double x[3] = {fine.at(row, km), fine.at(row, k), fine.at(row, kp)};
#pragma unroll
      for (int q = 0; q < 3; q++) {
        // (high word << 1 | low word != 0) - 1: zeros wrap to the top
        const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x[q]));
        const unsigned key = (static_cast<unsigned>(b >> 32) << 1) |
                             (static_cast<unsigned>(b) ? 1u : 0u);
        tiny = min(tiny, key - 1u);
        acc = __fma_rn(wi * wj * (q == 1 ? 1.0 : 0.5), x[q], acc);
      }
    }
  }
  if (tiny < 0x00800000u) acc = restrict_slow<A>(fine, nx, ny, nz, i, j, k);  // 2^-1019
  double r = __dmul_rn(acc, 0.125);  // == acc / 8.0 (power-of-two scale)
  if (neg4) r = -__dmul_rn(r, 4.0);
  return r;
}

// A prolongation axis: fine node i sits at i / 2 in coarse units, so its
// weight on a1 is 0, 1/2 or 1 (half = 0, 1, 2) and on a0 the rest.
struct Lerp {
  int a0, a1, half;
  __device__ __forceinline__ double t() const { return 0.5 * half; }
};

// multigrid3d.py:465-481 (prolong-add coordinates: a0 kept below the top)
__device__ __forceinline__ Lerp pa_axis(int i, int c) {
  Lerp l;
  const bool over = i > 2 * (c - 1);
  l.a0 = over ? c - 1 : i >> 1;
  l.half = over ? 0 : i & 1;
  if (l.a0 > c - 2) {
    l.half = c > 1 ? l.half + 2 * (l.a0 - (c - 2)) : l.half + 2 * l.a0;
    l.a0 = c > 1 ? c - 2 : 0;
  }
  l.a1 = c > 1 ? l.a0 + 1 : l.a0;
  return l;
}

// multigrid3d.py:144-156 (cascadic prolongation coordinates)
__device__ __forceinline__ Lerp pl_axis(int i, int c) {
  Lerp l;
  const bool over = i > 2 * (c - 1);
  l.a0 = over ? c - 1 : i >> 1;
  l.half = over ? 0 : i & 1;
  l.a1 = min(l.a0 + 1, c - 1);
  return l;
}

__device__ __forceinline__ double lerp_ref(double a, double b, double t) {
  // a*(1-t) + b*t, evaluated as the reference writes it
  return __dadd_rn(__dmul_rn(a, __dsub_rn(1.0, t)), __dmul_rn(b, t));
}

template <class A>
static __device__ __noinline__ double trilinear_slow(const A c, int cy, Lerp x, Lerp y, Lerp z) {
#define C(a, b, d) c.at(c.row((uint32_t)((a) * cy + (b))), d)
  const double c00 = lerp_ref(C(x.a0, y.a0, z.a0), C(x.a1, y.a0, z.a0), x.t());
  const double c10 = lerp_ref(C(x.a0, y.a1, z.a0), C(x.a1, y.a1, z.a0), x.t());
  const double c01 = lerp_ref(C(x.a0, y.a0, z.a1), C(x.a1, y.a0, z.a1), x.t());
  const double c11 = lerp_ref(C(x.a0, y.a1, z.a1), C(x.a1, y.a1, z.a1), x.t());
#undef C
  return lerp_ref(lerp_ref(c00, c10, y.t()), lerp_ref(c01, c11, y.t()), z.t());
}

// The trilinear value of the reference's nested lerps (28 FP64 instructions
// and more for the coordinates) with at most 7 additions: a weight 0 or 1
// picks one value, and the halvings of a mean commute with its rounding, so
// sums are formed and scaled once at the end.  Holds while every value is
// +0 or has an exponent that leaves room for three halvings and two
// doublings (no subnormal, overflow, infinity or NaN, skipped weight-0
// values included, since 0 x inf is NaN); -0 also takes the nested form.
// The prolongation's launch, averaged over the same levels: 16.5 -> 4.2 us.
template <class A>
__device__ __forceinline__ double trilinear(const A& c, int cy, const Lerp& x, const Lerp& y,
                                            const Lerp& z) {
  double v[8];
  bool ok = x.half <= 2 && y.half <= 2 && z.half <= 2;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    v[q] = c.at(c.row((uint32_t)((q & 4 ? x.a1 : x.a0) * cy + (q & 2 ? y.a1 : y.a0))),
                q & 1 ? z.a1 : z.a0);
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v[q]));
    ok = ok && ((static_cast<unsigned>(b >> 52) & 0x7ffu) - 64u <= 1976u || b == 0ULL);
  }
  if (!ok) return trilinear_slow<A>(c, cy, x, y, z);
  double p[4];
  if (x.half == 1) {
#pragma unroll
    for (int q = 0; q < 4; q++) p[q] = __dadd_rn(v[q], v[4 + q]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++) p[q] = x.half ? v[4 + q] : v[q];
  }
  if (y.half == 1) {
    p[0] = __dadd_rn(p[0], p[2]);
    p[1] = __dadd_rn(p[1], p[3]);
  } else if (y.half) {
    p[0] = p[2];
    p[1] = p[3];
  }
  // a single z value is doubled, so that every lane of a row takes one
  // addition and one halving more
  const double r = __dadd_rn(z.half == 2 ? p[1] : p[0], z.half ? p[1] : p[0]);
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(r));
  const unsigned long long halvings =
      1u + (x.half == 1 ? 1u : 0u) + (y.half == 1 ? 1u : 0u);
  return (b << 1) ? __longlong_as_double(static_cast<long long>(b - (halvings << 52))) : r;
}

// One CTA solving the bottom of multigrid3d._solve_err
// (multigrid3d.py:575-580) from shared memory: every node update is the
// launched kernel's arithmetic and the maxima are order-free, so the result
// and the pair count equal the launched loop's, without a launch per pair or
// a host synchronisation per batch.
//
// What bounds it is one SM's FP64 pipe (2 lanes per clock, 6 instructions a
// node) and the latency of a half-sweep's chain, so everything else is taken
// out of the pairs: the free nodes of each colour are listed once (their
// order changes no result), a thread keeps its first node of each colour
// with its neighbours' slots in registers (bottoms up to 2048 nodes need no
// other), and a pair has two barriers, its maximum going through the second.
// 637 nodes (7 x 7 x 13): 50 -> 31.5 us a solve, most of it pairs.
constexpr int kBottomCta = 1024;

// A node of the shared-memory level: its slot and its neighbours'.
struct BottomNode {
  int p = -1;
  Nb n;
};

struct BottomGeom {
  int nx, ny, nz;
  FastDiv dny, dnz;
};

__device__ __forceinline__ BottomNode bottom_node(int p, const BottomGeom& g) {
  BottomNode b;
  b.p = p;
  const uint32_t ij = fdiv((uint32_t)p, g.dnz);
  const uint32_t i = fdiv(ij, g.dny);
  b.n = neighbours(i, ij - i * g.dny.d, (uint32_t)p - ij * g.dnz.d, (uint32_t)g.nx,
                   (uint32_t)g.ny, (uint32_t)g.nz);
  return b;
}

__device__ __forceinline__ unsigned long long bottom_update(double* e, const double* f,
                                                            const BottomNode& b, double omega) {
  double v[6];
  load6(e, b.n, v);
  unsigned long long key = 0;
  e[b.p] = sor_apply<true, false>(e[b.p], div6(__dsub_rn(sum6(v), f[b.p])), omega, &key);
  return key;
}

// Block-wide maximum of a key; red: two rows of 32, alternated by the caller
// (row), so that one barrier orders the write and the next call's.
__device__ __forceinline__ unsigned long long cta_max(unsigned long long v,
                                                      unsigned long long* red, int row) {
  v = warp_max_u64(v);
  const int lane = threadIdx.x & 31;
  if (lane == 0) red[32 * row + (threadIdx.x >> 5)] = v;
  __syncthreads();
  return warp_max_u64(lane < (int)(blockDim.x >> 5) ? red[32 * row + lane] : 0ULL);
}

// The whole bottom solve by the calling CTA: sm holds 18 bytes a node, red
// and count are its scratch; f(t, ij, k) reads and put(t, ij, k, e) takes the
// value of node t = ij nz + k.  Every thread must call it.
template <class F, class P>
__device__ __forceinline__ void bottom_solve(const F& f_of, const P& put,
                                             const uint8_t* __restrict__ fixed_g,
                                             const BottomGeom& g, double rel_tol, double omega,
                                             long max_pairs, double* sm,
                                             unsigned long long* red, int* count) {
  const int n = g.nx * g.ny * g.nz, lane = threadIdx.x & 31;
  double* e = sm;
  double* f = sm + n;
  uint16_t* list = reinterpret_cast<uint16_t*>(sm + 2 * n);  // colour 0 up, colour 1 down
  if (threadIdx.x < 2) count[threadIdx.x] = 0;
  __syncthreads();
  // e = 0, f, the free nodes by colour, and max|f| (NaN in f makes it NaN,
  // as numpy's max does)
  unsigned long long fk = 0;
  bool nan = false;
  for (int t0 = 0; t0 < n; t0 += blockDim.x) {
    const int t = t0 + threadIdx.x;
    int c = -1;
    if (t < n) {
      const uint32_t ij = fdiv((uint32_t)t, g.dnz), k = (uint32_t)t - ij * g.dnz.d;
      const double x = f_of((uint32_t)t, ij, k);
      f[t] = x;
      e[t] = 0.0;
      const unsigned long long b =
          static_cast<unsigned long long>(__double_as_longlong(x)) & 0x7fffffffffffffffULL;
      if (b > 0x7ff0000000000000ULL) nan = true;
      else if (b > fk) fk = b;
      if (!fixed_g[t]) {
        const uint32_t i = fdiv(ij, g.dny);
        c = (int)((i + (ij - i * g.dny.d) + k) & 1u);
      }
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const unsigned m = __ballot_sync(0xffffffffu, c == q);
      int base = 0;
      if (lane == 0 && m) base = atomicAdd(&count[q], __popc(m));
      base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
      if (c == q) list[q ? n - 1 - base : base] = (uint16_t)t;
    }
  }
  nan = __syncthreads_or(nan);
  fk = cta_max(fk, red, 0);
  double scale = nan ? __longlong_as_double(0x7ff8000000000000LL) : bits_to_double(fk);
  scale = (1e-300 > scale) ? 1e-300 : scale;  // max(|f|.max(), 1e-300)
  // SOR pairs at omega until the larger of a pair's two max |update| is
  // below 0.02 * (rel_tol * scale / 6), at most max_pairs pairs
  const double tol = __dmul_rn(0.02, __ddiv_rn(__dmul_rn(rel_tol, scale), 6.0));
  const int n0 = count[0], n1 = count[1], tid = (int)threadIdx.x, nt = (int)blockDim.x;
  BottomNode own[2];
  if (tid < n0) own[0] = bottom_node(list[tid], g);
  if (tid < n1) own[1] = bottom_node(list[n - 1 - tid], g);
  for (long pr = 0; pr < max_pairs; pr++) {
    unsigned long long mb = 0;
#pragma unroll
    for (int c = 0; c < 2; c++) {
      if (own[c].p >= 0) mb = max(mb, bottom_update(e, f, own[c], omega));
      for (int q = tid + nt; q < (c ? n1 : n0); q += nt)
        mb = max(mb, bottom_update(e, f, bottom_node(list[c ? n - 1 - q : q], g), omega));
      if (c == 0) __syncthreads();
    }
    mb = cta_max(mb, red, (int)(pr & 1) ^ 1);
    if (bits_to_double(mb) < tol) break;
  }
  // the last pair's barrier (cta_max) came after its last update
  if (max_pairs <= 0) __syncthreads();
  for (int t = tid; t < n; t += nt) {
    const uint32_t ij = fdiv((uint32_t)t, g.dnz);
    put((uint32_t)t, ij, (uint32_t)t - ij * g.dnz.d, e[t]);
  }
}

__global__ void __launch_bounds__(kBottomCta)
k_bottom_err(double* __restrict__ e_out, const uint8_t* __restrict__ fixed_g,
             const double* __restrict__ f_g, BottomGeom g, double rel_tol,
             double omega, long max_pairs) {
  extern __shared__ double sm[];
  __shared__ unsigned long long red[64];
  __shared__ int count[2];
  bottom_solve([=](uint32_t t, uint32_t, uint32_t) { return f_g[t]; },
               [=](uint32_t t, uint32_t, uint32_t, double e) { e_out[t] = e; }, fixed_g, g,
               rel_tol, omega, max_pairs, sm, red, count);
}

// ---- the small error levels in one launch ----------------------------------
//
// multigrid3d._solve_err (multigrid3d.py:553-599) from one level down to the
// bottom, by one cluster of CTAs.  On the launched path a level of some
// 10^4 nodes costs about 20 launches, two memsets and two host decisions a
// cycle, each a few microseconds for well under one of work, and the eight
// bases of a door call queue for the driver as well (75,000 launches in 165
// ms).  Here the host decisions are the cluster's: every CTA forms the same
// maxima (exchanged through distributed shared memory) and takes the same
// branches.
//
// A CTA owns some rows (of k) of each level and their work.  DS: it also
// holds them, values, right-hand sides, masks and the residual, in its shared
// memory for the whole solve, and the others read them there: a phase then
// waits for a remote shared load (some 200 clocks) and a barrier with nothing
// of global memory behind it, where the levels in global memory cost two L2
// round trips and a fence, 5200 clocks a half-sweep even on 13 x 13 x 25
// nodes.  Levels too large for that (long rows in few of them) stay in
// global memory, read and written through L2.  Every node's arithmetic is
// the launched kernels', so the bits are theirs.  The bottom is CTA 0's
// (bottom_solve).  16 CTAs of 512 threads: a half-sweep of 25 x 25 x 49
// nodes is then some two nodes a thread and bound by its chain of load, sum
// and barrier rather than by the 16 SMs' FP64 pipes.
// A launch's time, values in global memory and here: 8 bases of a 97 x 97 x
// 193 ring deck 723 -> 576 us beside one another (a third of it the bottom),
// the door 96 -> 82 ms; 4 with theta at 65 x 65 x 129 282 -> 246 us (two
// thirds the bottom), 28.8 -> 27.5 ms.
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// Shared address a of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ double ld_cluster(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// A level's values by row and k wherever they live (FlatRows' interface):
// s the owner's shared address of them (the same in every CTA), or g.
template <bool DS>
struct TailRows;
template <>
struct TailRows<true> {
  uint32_t s, nz;
  FastDiv drow;  // rows a CTA
  typedef uint32_t Row;
  __device__ __forceinline__ Row row(uint32_t ij) const {
    const uint32_t o = fdiv(ij, drow);
    return cluster_addr(s + (ij - o * drow.d) * nz * 8u, o);
  }
  __device__ __forceinline__ double at(Row r, int k) const { return ld_cluster(r + 8u * k); }
  __device__ __forceinline__ void put(Row r, int k, double v) const { st_cluster(r + 8u * k, v); }
};
template <>
struct TailRows<false> {
  double* g;
  uint32_t nz;
  typedef double* Row;
  __device__ __forceinline__ Row row(uint32_t ij) const { return g + (size_t)ij * nz; }
  __device__ __forceinline__ double at(Row r, int k) const { return __ldcg(r + k); }
  __device__ __forceinline__ void put(Row r, int k, double v) const { __stcg(r + k, v); }
};

// What a CTA has of a level: rows [row0, row0 + rows), their arrays.
template <bool DS>
struct TailPart {
  uint32_t row0;
  int rows;
  double *e, *f, *r;
  const uint8_t* fixed;
  // own values: DS in this CTA's shared memory, else through L2
  static __device__ __forceinline__ double ld(const double* p) { return DS ? *p : __ldcg(p); }
  static __device__ __forceinline__ void st(double* p, double v) {
    if (DS) *p = v;
    else __stcg(p, v);
  }
};

template <bool DS>
__device__ __forceinline__ TailPart<DS> tail_part(const TailArgs& A, const TailLevel& L, int rank,
                                                  unsigned char* sm) {
  TailPart<DS> t;
  t.row0 = (uint32_t)rank * L.drow.d;
  t.rows = min((int)L.drow.d, L.nx * L.ny - (int)t.row0);
  const size_t o = (size_t)t.row0 * L.nz;
  t.e = DS ? reinterpret_cast<double*>(sm + L.oe) : L.e + o;
  t.f = DS ? reinterpret_cast<double*>(sm + L.of) : L.f + o;
  t.r = DS ? reinterpret_cast<double*>(sm + A.orr) : L.r + o;
  t.fixed = DS ? sm + L.om : L.fixed + o;
  return t;
}

template <bool DS>
__device__ __forceinline__ TailRows<DS> tail_rows(const TailLevel& L, double* g, uint32_t s) {
  if constexpr (DS) return TailRows<true>{s, (uint32_t)L.nz, L.drow};
  else return TailRows<false>{g, (uint32_t)L.nz};
}

// The six neighbours of node (row ij = (i, j), k) of a level: x and y ones by
// row, z ones in the node's own row (own), as neighbours() has them.
template <bool DS>
__device__ __forceinline__ void tail_load6(const TailRows<DS>& e, const double* own,
                                           const TailLevel& L, uint32_t ij, uint32_t i,
                                           uint32_t j, uint32_t k, double v[6]) {
  const uint32_t ny = (uint32_t)L.ny, nx = (uint32_t)L.nx, nz = (uint32_t)L.nz;
  const uint32_t rx = nx > 1 ? ny : 0u, ry = ny > 1 ? 1u : 0u, rz = nz > 1 ? 1u : 0u;
  v[0] = e.at(e.row(i > 0 ? ij - ny : ij + rx), (int)k);
  v[1] = e.at(e.row(i + 1 < nx ? ij + ny : ij - rx), (int)k);
  v[2] = e.at(e.row(j > 0 ? ij - 1 : ij + ry), (int)k);
  v[3] = e.at(e.row(j + 1 < ny ? ij + 1 : ij - ry), (int)k);
  v[4] = TailPart<DS>::ld(own + (k > 0 ? k - 1 : k + rz));
  v[5] = TailPart<DS>::ld(own + (k + 1 < nz ? k + 1 : k - rz));
}

// One half-sweep at omega 1 of a CTA's rows; the largest |update| key with
// DELTA.
template <bool DS, bool DELTA>
__device__ __forceinline__ unsigned long long tail_sweep(const TailLevel& L,
                                                         const TailPart<DS>& own,
                                                         const TailRows<DS>& e, int colour) {
  unsigned long long mb = 0;
  const int slots = own.rows * (int)L.dkk.d;
  for (int t = (int)threadIdx.x; t < slots; t += kTailThreads) {
    const uint32_t lr = fdiv((uint32_t)t, L.dkk), ij = own.row0 + lr;
    const uint32_t i = fdiv(ij, L.dny);
    const uint32_t j = ij - i * L.dny.d;
    const uint32_t k = 2 * ((uint32_t)t - lr * L.dkk.d) + ((i + j + (uint32_t)colour) & 1u);
    if (k >= (uint32_t)L.nz) continue;
    const uint32_t row = lr * (uint32_t)L.nz;
    if (own.fixed[row + k]) continue;
    double v[6];
    tail_load6<DS>(e, own.e + row, L, ij, i, j, k, v);
    const double f = own.ld(own.f + row + k), old = own.ld(own.e + row + k);
    unsigned long long key = 0;
    own.st(own.e + row + k,
           sor_apply<DELTA, true>(old, div6(__dsub_rn(sum6(v), f)), 1.0, &key));
    if (DELTA && key > mb) mb = key;
  }
  return mb;
}

template <bool DS>
__global__ void __launch_bounds__(kTailThreads)
k_err_tail(const __grid_constant__ TailArgs A) {
  namespace cg = cooperative_groups;
  extern __shared__ double dyn[];
  __shared__ unsigned long long red[64], wred[32], slot[2][kTailCtas];
  __shared__ int count[2];
  unsigned char* sm = reinterpret_cast<unsigned char*>(dyn);
  const uint32_t sb = smem_u32(sm);
  cg::cluster_group cl = cg::this_cluster();
  const int ctas = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int par = 0;
  // the cluster's maximum of a key, ending in a cluster barrier
  auto cluster_max = [&](unsigned long long v) {
    v = warp_max_u64(v);
    if (lane == 0) wred[wid] = v;
    __syncthreads();
    if (wid == 0) {
      v = warp_max_u64(lane < kTailThreads / 32 ? wred[lane] : 0ULL);
      if (lane < ctas) *cl.map_shared_rank(&slot[par][rank], lane) = v;
    }
    cl.sync();
    v = warp_max_u64(lane < ctas ? slot[par][lane] : 0ULL);
    par ^= 1;
    return v;
  };
  // max|f| as a key, ~0 standing for NaN
  auto fkey = [](double f) {
    const unsigned long long b =
        static_cast<unsigned long long>(__double_as_longlong(f)) & 0x7fffffffffffffffULL;
    return b > 0x7ff0000000000000ULL ? ~0ULL : b;
  };
  auto part = [&](const TailLevel& L) { return tail_part<DS>(A, L, rank, sm); };
  auto e_rows = [&](const TailLevel& L) { return tail_rows<DS>(L, L.e, sb + L.oe); };
  double tol[kTailLevels];
  int cyc[kTailLevels];
  auto enter = [&](int l, unsigned long long fk) {
    double scale = fk == ~0ULL ? __longlong_as_double(0x7ff8000000000000LL) : bits_to_double(fk);
    scale = (1e-300 > scale) ? 1e-300 : scale;  // max(|f|.max(), 1e-300)
    tol[l] = __ddiv_rn(__dmul_rn(A.rel_tol, scale), 6.0);
    cyc[l] = 0;
  };
  int l = 0;
  cl.sync();  // every CTA of the cluster runs
  {
    if (DS) {
      // the masks, and the first level's right-hand side
      for (int q = 0; q + 1 < A.nlev; q++) {
        const TailLevel& L = A.lv[q];
        const TailPart<DS> own = part(L);
        for (int t = threadIdx.x; t < own.rows * L.nz; t += kTailThreads)
          sm[L.om + t] = L.fixed[(size_t)own.row0 * L.nz + t];
      }
    }
    const TailLevel& L = A.lv[0];
    const TailPart<DS> own = part(L);
    unsigned long long fk = 0;
    for (int t = threadIdx.x; t < own.rows * L.nz; t += kTailThreads) {
      const double f = __ldcg(L.f + (size_t)own.row0 * L.nz + t);
      fk = max(fk, fkey(f));
      if (DS) own.st(own.f + t, f);
      own.st(own.e + t, 0.0);
    }
    enter(0, cluster_max(fk));
  }
  while (true) {
    // level l: pre-smoothing, and its residual restricted to level l + 1
    const TailLevel& L = A.lv[l];
    const TailLevel& C = A.lv[l + 1];
    {
      const TailPart<DS> own = part(L);
      const TailRows<DS> e = e_rows(L);
      for (int q = 0; q < 2 * A.nu1; q++) {
        tail_sweep<DS, false>(L, own, e, q & 1);
        cl.sync();
      }
      for (int t = threadIdx.x; t < own.rows * L.nz; t += kTailThreads) {
        double r = 0.0;
        if (!own.fixed[t]) {
          const uint32_t lr = fdiv((uint32_t)t, L.dnz), ij = own.row0 + lr;
          const uint32_t i = fdiv(ij, L.dny);
          const uint32_t row = lr * (uint32_t)L.nz;
          double v[6];
          tail_load6<DS>(e, own.e + row, L, ij, i, ij - i * L.dny.d, (uint32_t)t - row, v);
          r = __dsub_rn(resid6(sum6(v), own.ld(own.e + t)), own.ld(own.f + t));
        }
        own.st(own.r + t, r);
      }
      cl.sync();
    }
    {
      const TailPart<DS> own = part(C);
      const TailRows<DS> r = tail_rows<DS>(L, L.r, sb + A.orr);
      unsigned long long fk = 0;
      for (int t = threadIdx.x; t < own.rows * C.nz; t += kTailThreads) {
        const uint32_t lr = fdiv((uint32_t)t, C.dnz), ij = own.row0 + lr;
        const uint32_t ic = fdiv(ij, C.dny);
        const double f = restrict_node(r, L.nx, L.ny, L.nz, (int)ic, (int)(ij - ic * C.dny.d),
                                       (int)((uint32_t)t - lr * C.dnz.d), 1);
        own.st(own.f + t, f);
        own.st(own.e + t, 0.0);
        fk = max(fk, fkey(f));
      }
      enter(l + 1, cluster_max(fk));
    }
    l++;
    if (l + 1 < A.nlev) continue;
    if (rank == 0) {
      BottomGeom b;
      b.nx = C.nx;
      b.ny = C.ny;
      b.nz = C.nz;
      b.dny = C.dny;
      b.dnz = C.dnz;
      const TailRows<DS> e = e_rows(C), f = tail_rows<DS>(C, C.f, sb + C.of);
      bottom_solve(
          [&](uint32_t, uint32_t ij, uint32_t k) { return f.at(f.row(ij), (int)k); },
          [&](uint32_t, uint32_t ij, uint32_t k, double v) { e.put(e.row(ij), (int)k, v); },
          C.fixed, b, A.rel_tol, A.bottom_omega, A.bottom_pairs,
          reinterpret_cast<double*>(sm + A.ob), red, count);
    }
    cl.sync();
    // back up: correction, post-smoothing, and the cycle's decision
    bool done = true;
    while (done && l > 0) {
      const TailLevel& F = A.lv[l - 1];
      const TailLevel& K = A.lv[l];
      const TailPart<DS> own = part(F);
      const TailRows<DS> e = e_rows(F), ec = e_rows(K);
      l--;
      for (int t = threadIdx.x; t < own.rows * F.nz; t += kTailThreads) {
        if (own.fixed[t]) continue;
        const uint32_t lr = fdiv((uint32_t)t, F.dnz), ij = own.row0 + lr;
        const uint32_t i = fdiv(ij, F.dny);
        const Lerp x = pa_axis((int)i, K.nx), y = pa_axis((int)(ij - i * F.dny.d), K.ny);
        const Lerp z = pa_axis((int)((uint32_t)t - lr * F.dnz.d), K.nz);
        own.st(own.e + t, __dadd_rn(own.ld(own.e + t), trilinear(ec, K.ny, x, y, z)));
      }
      cl.sync();
      for (int q = 0; q < 2 * A.nu2 - 2; q++) {
        tail_sweep<DS, false>(F, own, e, q & 1);
        cl.sync();
      }
      unsigned long long mb = tail_sweep<DS, true>(F, own, e, 0);
      cl.sync();
      mb = cluster_max(max(mb, tail_sweep<DS, true>(F, own, e, 1)));
      cyc[l]++;
      done = bits_to_double(mb) < tol[l] || cyc[l] >= A.max_cycles;
    }
    if (done) break;
  }
  if (DS) {
    const TailLevel& L = A.lv[0];
    const TailPart<DS> own = part(L);
    for (int t = threadIdx.x; t < own.rows * L.nz; t += kTailThreads)
      L.e[(size_t)own.row0 * L.nz + t] = own.e[t];
  }
  cl.sync();  // no CTA leaves while another may still reach its shared memory
}

// multigrid3d._residual_rhs (multigrid3d.py:394-417).
__global__ void __launch_bounds__(kThreads)
k_residual_rhs(const double* __restrict__ e, const uint8_t* __restrict__ fixed,
               const double* __restrict__ f, FlatGeom g,
               double* __restrict__ out) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= g.total) return;
  const uint32_t ij = fdiv(t, g.div_nz);
  const uint32_t k = t - ij * g.div_nz.d;
  const uint32_t i = fdiv(ij, g.div_ny);
  const uint32_t j = ij - i * g.div_ny.d;
  double r = 0.0;
  if (!fixed[t]) {
    const Nb n = neighbours(i, j, k, g.nx, g.ny, g.nz);
    double v[6];
    load6(e, n, v);
    r = __dsub_rn(resid6(sum6(v), e[t]), f[t]);
  }
  out[t] = r;
}

__global__ void __launch_bounds__(kSweepThreads)
k_restrict(const double* __restrict__ fine, int nx, int ny, int nz,
           double* __restrict__ out, FlatGeom c, int neg4) {
  const uint32_t t = blockIdx.x * kSweepThreads + threadIdx.x;
  if (t >= c.total) return;
  const uint32_t ij = fdiv(t, c.div_nz);
  const uint32_t ic = fdiv(ij, c.div_ny);
  out[t] = restrict_node(FlatRows{fine, (uint32_t)nz}, nx, ny, nz, (int)ic, (int)(ij - ic * c.div_ny.d),
                         (int)(t - ij * c.div_nz.d), neg4);
}

// multigrid3d._prolong_add_njit (multigrid3d.py:458-499).
__global__ void __launch_bounds__(kSweepThreads)
k_prolong_add(const double* __restrict__ coarse, int cx, int cy, int cz,
              double* __restrict__ out, const uint8_t* __restrict__ fixed,
              FlatGeom g) {
  const uint32_t t = blockIdx.x * kSweepThreads + threadIdx.x;
  if (t >= g.total) return;
  if (fixed[t]) return;
  const uint32_t ij = fdiv(t, g.div_nz);
  const uint32_t i = fdiv(ij, g.div_ny);
  const Lerp x = pa_axis((int)i, cx), y = pa_axis((int)(ij - i * g.div_ny.d), cy);
  const Lerp z = pa_axis((int)(t - ij * g.div_nz.d), cz);
  out[t] = __dadd_rn(out[t], trilinear(FlatRows{coarse, (uint32_t)cz}, cy, x, y, z));
}

// multigrid3d._prolongate (multigrid3d.py:138-171).
__global__ void __launch_bounds__(kSweepThreads)
k_prolongate(const double* __restrict__ coarse, int cx, int cy, int cz,
             double* __restrict__ out, FlatGeom g) {
  const uint32_t t = blockIdx.x * kSweepThreads + threadIdx.x;
  if (t >= g.total) return;
  const uint32_t ij = fdiv(t, g.div_nz);
  const uint32_t i = fdiv(ij, g.div_ny);
  const Lerp x = pl_axis((int)i, cx), y = pl_axis((int)(ij - i * g.div_ny.d), cy);
  const Lerp z = pl_axis((int)(t - ij * g.div_nz.d), cz);
  out[t] = trilinear(FlatRows{coarse, (uint32_t)cz}, cy, x, y, z);
}

// multigrid3d._coarsen_fixed_any (multigrid3d.py:507-526).
__global__ void __launch_bounds__(kThreads)
k_coarsen_any(const uint8_t* __restrict__ fixed, long nx, long ny, long nz,
              uint8_t* __restrict__ out, FlatGeom c) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= c.total) return;
  const uint32_t ij = fdiv(t, c.div_nz);
  const long kc = t - ij * c.div_nz.d;
  const long ic = fdiv(ij, c.div_ny);
  const long jc = ij - ic * c.div_ny.d;
  uint8_t any = 0;
  for (int a = 0; a < 2; a++)
    for (int b = 0; b < 2; b++)
      for (int q = 0; q < 2; q++) {
        const long i = 2 * ic + a, j = 2 * jc + b, k = 2 * kc + q;
        if (i < nx && j < ny && k < nz && fixed[((size_t)i * ny + j) * nz + k]) any = 1;
      }
  out[t] = any;
}

// multigrid3d._coarsen_mask (multigrid3d.py:85-135).
__global__ void __launch_bounds__(kThreads)
k_coarsen_mask(const uint8_t* __restrict__ fixed, const double* __restrict__ val,
               long nx, long ny, long nz, uint8_t* __restrict__ fc,
               double* __restrict__ vc, FlatGeom c) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= c.total) return;
  const uint32_t ij = fdiv(t, c.div_nz);
  const long kc = t - ij * c.div_nz.d;
  const long ic = fdiv(ij, c.div_ny);
  const long jc = ij - ic * c.div_ny.d;
  const size_t p0 = ((size_t)(2 * ic) * ny + 2 * jc) * nz + 2 * kc;
  if (fixed[p0]) {
    fc[t] = 1;
    vc[t] = val[p0];
    return;
  }
  unsigned long long best = 0;
  bool any = false;
  double bv = 0.0;
  for (int a = 0; a < 2; a++)
    for (int b = 0; b < 2; b++)
      for (int q = 0; q < 2; q++) {
        const long i = 2 * ic + a, j = 2 * jc + b, k = 2 * kc + q;
        if (i >= nx || j >= ny || k >= nz) continue;
        const size_t p = ((size_t)i * ny + j) * nz + k;
        if (!fixed[p]) continue;
        const double v = val[p];
        // |v| compared through its bits (first maximum wins, as argmax)
        const unsigned long long m =
            (static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffULL) + 1ULL;
        if (!any || m > best) {
          best = m;
          bv = v;
        }
        any = true;
      }
  fc[t] = any ? 1 : 0;
  vc[t] = any ? bv : val[p0];
}

__global__ void k_set_fixed(double* __restrict__ phi,
                            const uint8_t* __restrict__ fixed,
                            const double* __restrict__ val, size_t n) {
  const size_t t = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (t < n && fixed[t]) phi[t] = val[t];
}

__global__ void k_set_basis(double* __restrict__ phi, const uint8_t* __restrict__ fixed,
                            const uint8_t* __restrict__ mask, double v, size_t n) {
  const size_t t = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (t < n && fixed[t]) phi[t] = mask[t] ? v : 0.0;
}

// The flip test of every axis at once, a node and its three mirror images a
// thread (the host read every node of a symmetric deck once per axis and
// basis before the first launch).
__global__ void __launch_bounds__(kThreads)
k_sym_check(const uint8_t* __restrict__ fixed, const double* __restrict__ val,
            const uint8_t* __restrict__ mask, double v, FlatGeom g, int* flags) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= g.total) return;
  const uint32_t ij = fdiv(t, g.div_nz);
  const uint32_t k = t - ij * g.div_nz.d;
  const uint32_t i = fdiv(ij, g.div_ny);
  const uint32_t j = ij - i * g.div_ny.d;
  const uint32_t nx = (uint32_t)g.nx, ny = (uint32_t)g.ny, nz = (uint32_t)g.nz;
  const uint32_t q[3] = {((nx - 1 - i) * ny + j) * nz + k, (i * ny + ny - 1 - j) * nz + k,
                         ij * nz + nz - 1 - k};
  auto at = [&](uint32_t p) { return val ? val[p] : (mask[p] ? v : 0.0); };
  const bool fx = fixed[t] != 0;
  const double x = at(t);
#pragma unroll
  for (int a = 0; a < 3; a++)
    if ((fixed[q[a]] != 0) != fx || !(at(q[a]) == x)) flags[a] = 1;
}

__global__ void __launch_bounds__(kThreads)
k_absdiff_max(const double* __restrict__ a, const double* __restrict__ b,
              size_t n, unsigned long long* bits, int* nan_flag) {
  unsigned long long mb = 0;
  bool nan = false;
  for (size_t t = (size_t)blockIdx.x * kThreads + threadIdx.x; t < n;
       t += (size_t)gridDim.x * kThreads) {
    const double d = b ? __dsub_rn(a[t], b[t]) : a[t];
    const unsigned long long x =
        static_cast<unsigned long long>(__double_as_longlong(d)) & 0x7fffffffffffffffULL;
    if (x > 0x7ff0000000000000ULL) nan = true;
    else if (x > mb) mb = x;
  }
  if (__syncthreads_or(nan) && threadIdx.x == 0) *nan_flag = 1;
  block_max_to(mb, bits);
}

__global__ void k_report(const unsigned long long* __restrict__ d, unsigned long long* host) {
  if (threadIdx.x < 2) host[threadIdx.x] = d[threadIdx.x];
}

// phi <- (phi + flip(phi, axis)) * 0.5 (multigrid3d.py:689-691); each thread
// owns a mirror pair, so the in-place update reads both values first.
__global__ void __launch_bounds__(kThreads)
k_sym_project(double* __restrict__ phi, FlatGeom g, int axis) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= g.total) return;
  const uint32_t ij = fdiv(t, g.div_nz);
  const long k = t - ij * g.div_nz.d;
  const long i = fdiv(ij, g.div_ny);
  const long j = ij - i * g.div_ny.d;
  long mi = i, mj = j, mk = k;
  if (axis == 0) mi = g.nx - 1 - i;
  else if (axis == 1) mj = g.ny - 1 - j;
  else mk = g.nz - 1 - k;
  const size_t q = ((size_t)mi * g.ny + mj) * g.nz + mk;
  if (q < t) return;  // the partner with the lower index does the pair
  const double s = __dmul_rn(__dadd_rn(phi[t], phi[q]), 0.5);
  phi[t] = s;
  phi[q] = s;
}

// solver3d._residual_kernel (solver3d.py:366-386): num/den - u.
__global__ void __launch_bounds__(kThreads)
k_residual_audit(const double* __restrict__ u, const uint8_t* __restrict__ fixed,
                 const float* __restrict__ th, FlatGeom g,
                 double* __restrict__ out) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= g.total) return;
  const uint32_t ij = fdiv(t, g.div_nz);
  const uint32_t k = t - ij * g.div_nz.d;
  const uint32_t i = fdiv(ij, g.div_ny);
  const uint32_t j = ij - i * g.div_ny.d;
  double r = 0.0;
  if (!fixed[t]) {
    const Nb n = neighbours(i, j, k, g.nx, g.ny, g.nz);
    double v[6], num, den;
    load6(u, n, v);
    theta_num_den<kThetaGhost>(v, th, g.total, t, num, den);
    r = __dsub_rn(__ddiv_rn(num, den), u[t]);
  }
  out[t] = r;
}

// solver3d._err_sweep (solver3d.py:389-417).
__global__ void __launch_bounds__(kThreads)
k_err_sweep(double* __restrict__ e, const uint8_t* __restrict__ fixed,
            const float* __restrict__ th, const double* __restrict__ rhs,
            SweepGeom g, double omega, int colour, unsigned long long* dslot) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  unsigned long long mb = 0;
  if (t < g.total) {
    const uint32_t ij = fdiv(t, g.div_kk);
    const uint32_t kk = t - ij * g.div_kk.d;
    const uint32_t i = fdiv(ij, g.div_ny);
    const uint32_t j = ij - i * g.div_ny.d;
    const uint32_t k = 2 * kk + ((i + j + colour) & 1);
    if (k < (uint32_t)g.nz) {
      const uint32_t p = (i * (uint32_t)g.ny + j) * (uint32_t)g.nz + k;
      if (!fixed[p]) {
        const Nb n = neighbours(i, j, k, g.nx, g.ny, g.nz);
        double v[6], num, den;
        load6(e, n, v);
        theta_num_den<kThetaGhost>(v, th, (size_t)g.nx * g.ny * g.nz, p, num, den);
        const double old = e[p];
        const double inner = __dsub_rn(__dadd_rn(__ddiv_rn(num, den), rhs[p]), old);
        const double nw = __dadd_rn(old, __dmul_rn(omega, inner));
        mb = absbits(__dsub_rn(nw, old));
        e[p] = nw;
      }
    }
  }
  block_max_to(mb, dslot);
}

__global__ void k_fill_ones_f32(float* a, size_t n) {
  const size_t t = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (t < n) a[t] = 1.0f;
}

}  // namespace

void launch_sweep(cudaStream_t s, double* phi, const uint8_t* fixed,
                  const float* th, int kind, Dims d, double omega, int colour,
                  unsigned long long* dslot, PairCtl* ctl, int lp) {
  const int U = kind == kPlain ? sweep_planes(d) : 1;
  const SweepGeom g = sweep_geom(d, U);
  const unsigned nb = sweep_blocks(g);
  if (nb == 0) return;
  counted();
  const bool one = omega == 1.0 && !ctl;
#define IG_SWEEP_T(K, C, D, O, P)                                                            \
  k_sweep<K, C, D, O, P><<<nb, kSweepThreads, 0, s>>>(phi, fixed, th, g, omega, colour, dslot,    \
                                                 ctl, lp)
#define IG_SWEEP(K, P)                                                                       \
  if (ctl) IG_SWEEP_T(K, true, true, false, P);                                              \
  else if (dslot && one) IG_SWEEP_T(K, false, true, true, P);                                \
  else if (dslot) IG_SWEEP_T(K, false, true, false, P);                                      \
  else if (one) IG_SWEEP_T(K, false, false, true, P);                                        \
  else IG_SWEEP_T(K, false, false, false, P);
  if (kind == kPlain && U == 2) { IG_SWEEP(kPlain, 2) }
  else if (kind == kPlain) { IG_SWEEP(kPlain, 1) }
  else if (kind == kThetaGhost) { IG_SWEEP(kThetaGhost, 1) }
  else { IG_SWEEP(kThetaSW, 1) }
#undef IG_SWEEP_T
#undef IG_SWEEP
}

void launch_residual(cudaStream_t s, const double* phi, const uint8_t* fixed,
                     const float* th, int kind, Dims d, double* out,
                     unsigned long long* absmax) {
  const FlatGeom g = flat_geom(d);
  const unsigned nb = (unsigned)((((size_t)(d.nx + kResidPlanes - 1) / kResidPlanes) * d.ny * d.nz +
                                  kSweepThreads - 1) / kSweepThreads);
  if (nb == 0) return;
  counted();
  if (kind == kPlain)
    k_residual<kPlain><<<nb, kSweepThreads, 0, s>>>(phi, fixed, th, g, out, absmax);
  else if (kind == kPlainSW)
    k_residual<kPlainSW><<<nb, kSweepThreads, 0, s>>>(phi, fixed, th, g, out, absmax);
  else if (kind == kThetaGhost)
    k_residual<kThetaGhost><<<nb, kSweepThreads, 0, s>>>(phi, fixed, th, g, out, absmax);
  else
    k_residual<kThetaSW><<<nb, kSweepThreads, 0, s>>>(phi, fixed, th, g, out, absmax);
}

void launch_theta_class(cudaStream_t s, const uint8_t* fixed, const float* th, Dims d,
                        uint8_t* cls, uint32_t* counts) {
  const FlatGeom g = flat_geom(d);
  cudaMemsetAsync(counts, 0, 2 * sizeof(uint32_t), s);
  k_theta_class<<<blocks_for(g.total), kThreads, 0, s>>>(fixed, th, g, cls, counts);
  counted();
}

void launch_theta_fill(cudaStream_t s, const uint8_t* cls, const float* th, int kind, Dims d,
                       const uint32_t count[2], uint32_t* cursor, uint32_t* idx, double* w) {
  const FlatGeom g = flat_geom(d);
  const unsigned nb = blocks_for(g.total);
  const uint32_t total = count[0] + count[1];
  cudaMemsetAsync(cursor, 0, 2 * sizeof(uint32_t), s);
  if (total == 0) return;
  if (kind == kThetaGhost)
    k_theta_fill<kThetaGhost><<<nb, kThreads, 0, s>>>(cls, th, g, count[0], total, cursor, idx, w);
  else
    k_theta_fill<kThetaSW><<<nb, kThreads, 0, s>>>(cls, th, g, count[0], total, cursor, idx, w);
  counted();
}

void launch_sweep_plan(cudaStream_t s, double* phi, const ThetaPlan& plan, int kind, Dims d,
                       double omega, int colour, PairCtl* ctl, int lp) {
  unsigned long long* const dslot = nullptr;  // with ctl the kernel takes its slot from it
  const SweepGeom g = sweep_geom(d);
  const FastDiv dnz((uint32_t)d.nz);
  const uint32_t lb = blocks_for(plan.count[colour]);
  const unsigned nb = lb + blocks_for(g.total);
  counted();
  const bool one = omega == 1.0 && !ctl;
#define IG_SWEEP_T(K, C, D, O)                                                               \
  k_sweep_plan<K, C, D, O><<<nb, kThreads, 0, s>>>(phi, plan, g, dnz, lb, omega, colour,     \
                                                   dslot, ctl, lp)
#define IG_SWEEP(K)                                                                          \
  if (ctl) IG_SWEEP_T(K, true, true, false);                                                 \
  else if (one) IG_SWEEP_T(K, false, false, true);                                           \
  else IG_SWEEP_T(K, false, false, false);
  if (kind == kThetaGhost) { IG_SWEEP(kThetaGhost) }
  else { IG_SWEEP(kThetaSW) }
#undef IG_SWEEP_T
#undef IG_SWEEP
}

void launch_residual_plan(cudaStream_t s, const double* phi, const ThetaPlan& plan, int kind,
                          Dims d, double* out) {
  const FlatGeom g = flat_geom(d);
  const uint32_t lb = blocks_for(plan.total());
  const unsigned nb = lb + blocks_for(g.total);
  counted();
  if (kind == kThetaGhost)
    k_residual_plan<kThetaGhost><<<nb, kThreads, 0, s>>>(phi, plan, g, lb, out);
  else
    k_residual_plan<kThetaSW><<<nb, kThreads, 0, s>>>(phi, plan, g, lb, out);
}

void launch_sweep_rhs(cudaStream_t s, double* e, const uint8_t* fixed,
                      const double* f, Dims d, double omega, int colour,
                      unsigned long long* dslot, PairCtl* ctl, int lp) {
  const int U = sweep_planes(d);
  const SweepGeom g = sweep_geom(d, U);
  const unsigned nb = sweep_blocks(g);
  if (nb == 0) return;
  counted();
  const bool one = omega == 1.0 && !ctl;
#define IG_SWEEP_T(C, D, O, P)                                                               \
  k_sweep_rhs<C, D, O, P><<<nb, kSweepThreads, 0, s>>>(e, fixed, f, g, omega, colour, dslot, ctl, \
                                                  lp)
#define IG_SWEEP(P)                                                                          \
  if (ctl) IG_SWEEP_T(true, true, false, P);                                                 \
  else if (dslot && one) IG_SWEEP_T(false, true, true, P);                                   \
  else if (dslot) IG_SWEEP_T(false, true, false, P);                                         \
  else if (one) IG_SWEEP_T(false, false, true, P);                                           \
  else IG_SWEEP_T(false, false, false, P);
  if (U == 2) { IG_SWEEP(2) }
  else { IG_SWEEP(1) }
#undef IG_SWEEP_T
#undef IG_SWEEP
}

// A number found once for each device: a kernel's attributes and the launches
// that fit belong to the device, and another thread's call may be between
// finding them and launching.
class PerDevice {
 public:
  // find(device) on the current device's first use; 0 where there is no device
  template <class F>
  int get(F&& find) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMost) {
      cudaGetLastError();
      return 0;
    }
    std::lock_guard<std::mutex> lk(mu_);
    if (!found_[dev]) {
      value_[dev] = find(dev);
      found_[dev] = true;
    }
    return value_[dev];
  }

 private:
  static constexpr int kMost = 64;
  std::mutex mu_;
  int value_[kMost] = {0};
  bool found_[kMost] = {false};
};

bool launch_bottom_err(cudaStream_t s, double* e, const uint8_t* fixed, const double* f,
                       Dims d, double rel_tol, double omega, long max_pairs) {
  const size_t n = d.n();
  if (n == 0 || 17 * n > kBottomSmemMax) return false;
  const size_t bytes = 18 * n;
  static PerDevice smem;
  if (!smem.get([](int) {
        const int most = (int)(18 * (kBottomSmemMax / 17));
        const bool ok = cudaFuncSetAttribute(k_bottom_err,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             most) == cudaSuccess;
        if (!ok) cudaGetLastError();
        return ok ? 1 : 0;
      }))
    return false;
  BottomGeom g;
  g.nx = (int)d.nx;
  g.ny = (int)d.ny;
  g.nz = (int)d.nz;
  g.dny = FastDiv((uint32_t)d.ny);
  g.dnz = FastDiv((uint32_t)d.nz);
  // a thread per node of one colour, in whole warps: fewer warps, cheaper
  // barriers
  const int nt = std::min<long>(kBottomCta, std::max<long>(64, ((long)(n + 1) / 2 + 31) / 32 * 32));
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(1);
  c.blockDim = dim3((unsigned)nt);
  c.dynamicSmemBytes = (bytes + 7) / 8 * 8;
  c.stream = s;
  if (cudaLaunchKernelEx(&c, k_bottom_err, e, fixed, f, g, rel_tol, omega, max_pairs) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  counted();
  return true;
}

// The largest dynamic shared memory a CTA of k_sor_flow is launched with: its
// share of the slots of the largest grid on this route (152 SMs).  The
// attribute is set to this once, never to a call's own size: calls of other
// threads launch the same kernels.
constexpr size_t kFlowSmemMax = 8 * kCoopThreads * kFlowBytes;

bool launch_sor_coop(cudaStream_t s, double* phi, const uint8_t* cls, const ThetaPlan* plan,
                     int kind, Dims d, double omega, double tol, int pairs, CoopCtl* ctl,
                     void* word, double* prev) {
  // a whole grid of one CTA per SM
  static PerDevice sms;
  const int n = sms.get([](int dev) {
    int coop = 0, count = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    for (const void* fn : {(const void*)k_sor_flow<kThetaGhost>, (const void*)k_sor_flow<kThetaSW>,
                           (const void*)k_sor_flow<kPlain>})
      if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kFlowSmemMax) != cudaSuccess)
        coop = 0;
    cudaGetLastError();
    return coop ? std::min(count, kCoopCtas) : 0;
  });
  if (n < 1 || !word) return false;
  SweepGeom g = sweep_geom(d);
  FastDiv dnz((uint32_t)d.nz);
  ThetaPlan P = plan ? *plan : ThetaPlan();
  FlowGeom G;
  G.g = g;
  G.dnz = dnz;
  G.share = (g.total + (uint32_t)n - 1) / (uint32_t)n;
  // no more warps than the share has work for: idle ones only ask whether the
  // others are done.  A theta plan's cut nodes (five a warp) get up to four
  // warps of their own, since the nodes of a warp that has both wait behind the
  // divisions (57 x 71 x 90, 0.4 % cut nodes: 3.31 -> 2.98 ms), but none that
  // would cost the others a round (129^3: 20.6 us a half-sweep, 22.0 with
  // four).
  const uint32_t cut = plan ? std::max(plan->count[0], plan->count[1]) : 0u;
  unsigned cutw = std::min(4u, (cut + 5u * (unsigned)n - 1) / (5u * (unsigned)n));
  auto rounds_of = [&](unsigned w) { return (G.share + w - 1) / w; };
  while (cutw && rounds_of(kCoopThreads - 32 * cutw) > rounds_of(kCoopThreads)) cutw--;
  G.workers = std::min((unsigned)kCoopThreads - 32 * cutw,
                       std::max(64u, (G.share + 31) / 32 * 32));
  const unsigned nt = G.workers + 32 * cutw;
  G.rounds = (int)rounds_of(G.workers);
  G.word = static_cast<ulonglong2*>(word);
  G.prev = prev;
  const size_t smem = (size_t)G.rounds * G.workers * kFlowBytes;
  if (smem > kFlowSmemMax || cudaMemsetAsync(ctl, 0, sizeof(CoopCtl), s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  void* args[] = {&phi, &cls, &P, &G, &omega, &tol, &pairs, &ctl};
  const void* fn = kind == kThetaGhost ? (const void*)k_sor_flow<kThetaGhost>
                   : kind == kThetaSW  ? (const void*)k_sor_flow<kThetaSW>
                                       : (const void*)k_sor_flow<kPlain>;
  if (cudaLaunchCooperativeKernel(fn, dim3(n), dim3(nt), args, smem, s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  counted();
  return true;
}

TailLevel tail_level(Dims d, double* e, double* f, double* r, const uint8_t* fixed) {
  TailLevel L;
  L.e = e;
  L.f = f;
  L.r = r;
  L.fixed = fixed;
  L.nx = (int)d.nx;
  L.ny = (int)d.ny;
  L.nz = (int)d.nz;
  L.dkk = FastDiv((uint32_t)((d.nz + 1) / 2));
  L.dny = FastDiv((uint32_t)d.ny);
  L.dnz = FastDiv((uint32_t)d.nz);
  return L;
}

// Gives each CTA its rows and, in shared memory, its part of every level;
// the bytes that takes.
static size_t tail_layout(TailArgs& a, int ctas) {
  size_t o = 0, rmax = 0, m = 0;
  for (int q = 0; q < a.nlev; q++) {
    TailLevel& L = a.lv[q];
    const uint32_t rows = ((uint32_t)(L.nx * L.ny) + ctas - 1) / ctas;
    L.drow = FastDiv(rows);
    const size_t n = (size_t)rows * L.nz;
    L.oe = (uint32_t)o;
    L.of = (uint32_t)(o + 8 * n);
    o += 16 * n;
    if (q + 1 < a.nlev) rmax = std::max(rmax, n);
  }
  a.orr = (uint32_t)o;
  o += 8 * rmax;
  a.ob = (uint32_t)o;  // the bottom's 18 bytes a node, CTA 0's
  const TailLevel& b = a.lv[a.nlev - 1];
  o += ((size_t)b.nx * b.ny * b.nz * 18 + 7) / 8 * 8;
  for (int q = 0; q + 1 < a.nlev; q++) {
    TailLevel& L = a.lv[q];
    L.om = (uint32_t)(o + m);
    m += (size_t)L.drow.d * L.nz;
  }
  return (o + m + 7) / 8 * 8;
}

bool launch_err_tail(cudaStream_t s, TailArgs a) {
  const TailLevel& b = a.lv[a.nlev - 1];
  const size_t nb = (size_t)b.nx * b.ny * b.nz;
  auto config = [](cudaLaunchConfig_t* c, cudaLaunchAttribute* at, int n, size_t smem,
                   cudaStream_t st) {
    *c = cudaLaunchConfig_t{};
    c->gridDim = dim3(n);
    c->blockDim = dim3(kTailThreads);
    c->dynamicSmemBytes = smem;
    c->stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = n;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    c->attrs = at;
    c->numAttrs = 1;
  };
  constexpr size_t most = 18 * (kBottomSmemMax / 17);
  // the cluster size this device takes with all of an SM's shared memory (16
  // CTAs, else the portable 8; 0: neither)
  static PerDevice size;
  const int ctas = size.get([&](int) {
    for (const void* fn : {(const void*)k_err_tail<false>, (const void*)k_err_tail<true>}) {
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
      cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    cudaGetLastError();
    for (int n : {kTailCtas, 8}) {
      cudaLaunchConfig_t c;
      cudaLaunchAttribute at[1];
      config(&c, at, n, most, nullptr);
      int active = 0, other = 0;
      if (cudaOccupancyMaxActiveClusters(&active, k_err_tail<true>, &c) == cudaSuccess &&
          cudaOccupancyMaxActiveClusters(&other, k_err_tail<false>, &c) == cudaSuccess &&
          active > 0 && other > 0)
        return n;
      cudaGetLastError();
    }
    return 0;
  });
  if (!ctas || nb == 0 || 17 * nb > kBottomSmemMax) return false;
  const size_t bytes = tail_layout(a, ctas);
  const bool ds = bytes <= most;
  if (!ds) a.ob = 0;  // the bottom's scratch alone
  cudaLaunchConfig_t c;
  cudaLaunchAttribute at[1];
  config(&c, at, ctas, ds ? bytes : (18 * nb + 7) / 8 * 8, s);
  if (cudaLaunchKernelEx(&c, ds ? k_err_tail<true> : k_err_tail<false>, a) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  counted();
  return true;
}

void launch_residual_rhs(cudaStream_t s, const double* e, const uint8_t* fixed,
                         const double* f, Dims d, double* out) {
  const FlatGeom g = flat_geom(d);
  const unsigned nb = blocks_for(g.total);
  if (nb) {
    k_residual_rhs<<<nb, kThreads, 0, s>>>(e, fixed, f, g, out);
    counted();
  }
}

void launch_restrict(cudaStream_t s, const double* fine, Dims d, double* out,
                     Dims c, int neg4) {
  const FlatGeom g = flat_geom(c);
  const unsigned nb = (g.total + kSweepThreads - 1) / kSweepThreads;
  if (nb) {
    k_restrict<<<nb, kSweepThreads, 0, s>>>(fine, (int)d.nx, (int)d.ny, (int)d.nz, out, g, neg4);
    counted();
  }
}

void launch_prolong_add(cudaStream_t s, const double* coarse, Dims c,
                        double* out, const uint8_t* fixed, Dims d) {
  const FlatGeom g = flat_geom(d);
  const unsigned nb = (g.total + kSweepThreads - 1) / kSweepThreads;
  if (nb) {
    k_prolong_add<<<nb, kSweepThreads, 0, s>>>(coarse, (int)c.nx, (int)c.ny, (int)c.nz, out, fixed, g);
    counted();
  }
}

void launch_prolongate(cudaStream_t s, const double* coarse, Dims c,
                       double* out, Dims d) {
  const FlatGeom g = flat_geom(d);
  const unsigned nb = (g.total + kSweepThreads - 1) / kSweepThreads;
  if (nb) {
    k_prolongate<<<nb, kSweepThreads, 0, s>>>(coarse, (int)c.nx, (int)c.ny, (int)c.nz, out, g);
    counted();
  }
}

void launch_coarsen_any(cudaStream_t s, const uint8_t* fixed, Dims d,
                        uint8_t* out, Dims c) {
  const FlatGeom g = flat_geom(c);
  const unsigned nb = blocks_for(g.total);
  if (nb) {
    k_coarsen_any<<<nb, kThreads, 0, s>>>(fixed, d.nx, d.ny, d.nz, out, g);
    counted();
  }
}

void launch_coarsen_mask(cudaStream_t s, const uint8_t* fixed,
                         const double* val, Dims d, uint8_t* fc, double* vc,
                         Dims c) {
  const FlatGeom g = flat_geom(c);
  const unsigned nb = blocks_for(g.total);
  if (nb) {
    k_coarsen_mask<<<nb, kThreads, 0, s>>>(fixed, val, d.nx, d.ny, d.nz, fc, vc, g);
    counted();
  }
}

void launch_set_fixed(cudaStream_t s, double* phi, const uint8_t* fixed,
                      const double* val, size_t n) {
  const unsigned nb = blocks_for(n);
  if (nb) {
    k_set_fixed<<<nb, kThreads, 0, s>>>(phi, fixed, val, n);
    counted();
  }
}

void launch_set_basis(cudaStream_t s, double* phi, const uint8_t* fixed, const uint8_t* mask,
                      double v, size_t n) {
  const unsigned nb = blocks_for(n);
  if (nb) {
    k_set_basis<<<nb, kThreads, 0, s>>>(phi, fixed, mask, v, n);
    counted();
  }
}

void launch_sym_check(cudaStream_t s, const uint8_t* fixed, const double* val,
                      const uint8_t* mask, double v, Dims d, int* flags) {
  const FlatGeom g = flat_geom(d);
  cudaMemsetAsync(flags, 0, 3 * sizeof(int), s);
  k_sym_check<<<blocks_for(g.total), kThreads, 0, s>>>(fixed, val, mask, v, g, flags);
  counted();
}

void launch_absdiff_max(cudaStream_t s, const double* a, const double* b,
                        size_t n, unsigned long long* bits, int* nan_flag) {
  unsigned nb = blocks_for(n);
  if (nb > 152u * 8u) nb = 152u * 8u;
  if (nb) {
    k_absdiff_max<<<nb, kThreads, 0, s>>>(a, b, n, bits, nan_flag);
    counted();
  }
}

void launch_report(cudaStream_t s, const unsigned long long* d, unsigned long long* host) {
  k_report<<<1, 32, 0, s>>>(d, host);
  counted();
}

void launch_sym_project(cudaStream_t s, double* phi, Dims d, int axis) {
  const FlatGeom g = flat_geom(d);
  const unsigned nb = blocks_for(g.total);
  if (nb) {
    k_sym_project<<<nb, kThreads, 0, s>>>(phi, g, axis);
    counted();
  }
}

void launch_residual_audit(cudaStream_t s, const double* u,
                           const uint8_t* fixed, const float* th, Dims d,
                           double* out) {
  const FlatGeom g = flat_geom(d);
  const unsigned nb = blocks_for(g.total);
  if (nb) {
    k_residual_audit<<<nb, kThreads, 0, s>>>(u, fixed, th, g, out);
    counted();
  }
}

void launch_err_sweep(cudaStream_t s, double* e, const uint8_t* fixed,
                      const float* th, const double* rhs, Dims d, double omega,
                      int colour, unsigned long long* dslot) {
  const SweepGeom g = sweep_geom(d);
  const unsigned nb = blocks_for(g.total);
  if (nb) {
    k_err_sweep<<<nb, kThreads, 0, s>>>(e, fixed, th, rhs, g, omega, colour, dslot);
    counted();
  }
}

void launch_fill_ones_f32(cudaStream_t s, float* a, size_t n) {
  const unsigned nb = blocks_for(n);
  if (nb) {
    k_fill_ones_f32<<<nb, kThreads, 0, s>>>(a, n);
    counted();
  }
}

}  // namespace ig
