// ig_geometry.cu -- analytic scenes on the device: the labelled node raster
// (ion_gym physics/rasterize3d.py:45-109) and the fractional-surface legs
// theta (physics/solver3d.py:46-127), bit-identical to the reference's
// float64 numpy evaluation.
//
// A scene arrives as a flat primitive table in grid units.  Each primitive
// carries its electrode (in raster order), its shape, whether it is a
// `within` or a `notin` solid, and its bounds pre-combined on the host with
// the reference's tolerance exactly as the reference writes them
// (r**2 + eps, (z - length) - eps, x1 - eps, ...), so the kernels only form
// (x - cx)**2 + (y - cy)**2 with round-to-nearest operations and compare.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "ig_common.cuh"
#include "ig_internal.h"
#include "../../include/igsolve.h"

namespace ig {
namespace {

constexpr int kT = 256;

// One primitive: kind (0 cylinder, 1 box), electrode slot, shape id, role (0
// within, 1 notin), then the bounds:
//   cylinder: cx, cy, r2 (r**2 + e), zlo ((z - length) - e), zhi (z + e)
//   box:      x1 - e, x2 + e, y1 - e, y2 + e, z1 - e, z2 + e
// Two copies of the bounds are stored: with e = +eps (inclusive) and with
// e = -eps (strict, used for `notin` solids by the theta inside test).
// node: the inclusive bounds as the nodes see them, the first and last
// integer coordinate inside per axis (a cylinder's x and y ranges are open):
// integer compares leave the FP64 pipe, 2 lanes per clock and SM, to the
// radius test.
struct Prim {
  int kind, elec, shape, role;
  double in[6];
  double st[6];
  int node[6];
};

__device__ __forceinline__ bool inside(const Prim& p, const double* b, double x,
                                       double y, double z) {
  if (p.kind == 0) {
    const double dx = __dsub_rn(x, b[0]);
    const double dy = __dsub_rn(y, b[1]);
    const double rr = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
    return rr <= b[2] && z >= b[3] && z <= b[4];
  }
  return x >= b[0] && x <= b[1] && y >= b[2] && y <= b[3] && z >= b[4] && z <= b[5];
}

__device__ __noinline__ bool in_radius(const Prim& p, int i, int j) {
  const double dx = __dsub_rn((double)i, p.in[0]);
  const double dy = __dsub_rn((double)j, p.in[1]);
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) <= p.in[2];
}

// inside(p, p.in, ...) of node (i, j, k)
__device__ __forceinline__ bool inside_node(const Prim& p, int i, int j, int k) {
  if (i < p.node[0] || i > p.node[1] || j < p.node[2] || j > p.node[3] || k < p.node[4] ||
      k > p.node[5])
    return false;
  return p.kind != 0 || in_radius(p, i, j);
}

// Per electrode, a warp's counts and lowest index with one atomic each (a
// lone atomic per metal node serialises on the electrode's counter).
__device__ __forceinline__ void warp_count(bool hit, unsigned long long* n) {
  const unsigned m = __ballot_sync(0xffffffffu, hit);
  if (m && (threadIdx.x & 31) == 0) atomicAdd(n, (unsigned long long)__popc(m));
}
__device__ __forceinline__ void warp_first(bool hit, size_t t, unsigned long long* first) {
  const unsigned m = __ballot_sync(0xffffffffu, hit);  // t rises with the lane
  if (m && (int)(threadIdx.x & 31) == __ffs(m) - 1) atomicMin(first, (unsigned long long)t);
}

// rasterize3d.rasterize: per node, electrodes in order; shapes union, within
// minus notin (inclusive bounds for both); a node claimed by a second
// electrode index is a clash.  Per electrode: node count, clash count and
// the lowest clashing flat index.  97 x 97 x 193 nodes, 8 rings:
// 364 -> 95 us.
__global__ void __launch_bounds__(kT)
k_rasterize(const Prim* __restrict__ prims, int np, const int* __restrict__ eidx,
            int ne, long nx, long ny, long nz, int16_t* __restrict__ lab,
            unsigned long long* __restrict__ count,
            unsigned long long* __restrict__ clash_count,
            unsigned long long* __restrict__ clash_min) {
  const size_t n = (size_t)nx * ny * nz;
  const size_t t = (size_t)blockIdx.x * kT + threadIdx.x;
  const bool live = t < n;  // every lane stays for the warp's votes
  const int k = live ? (int)(t % nz) : -1;
  const int j = live ? (int)((t / nz) % ny) : -1;
  const int i = live ? (int)(t / ((size_t)nz * ny)) : -1;
  int16_t cur = 0;
  int p = 0;
  for (int e = 0; e < ne; e++) {
    bool m = false;
    while (p < np && prims[p].elec == e) {
      // one shape: its within primitives then its notin primitives
      const int sh = prims[p].shape;
      bool w = false;
      while (p < np && prims[p].elec == e && prims[p].shape == sh) {
        const Prim& q = prims[p];
        const bool hit = live && inside_node(q, i, j, k);
        if (q.role == 0) w = w || hit;
        else w = w && !hit;
        p++;
      }
      m = m || w;
    }
    if (!__any_sync(0xffffffffu, m)) continue;
    const int16_t idx = (int16_t)eidx[e];
    const bool clash = m && cur != 0 && cur != idx;
    warp_count(m, count + e);
    warp_count(clash, clash_count + e);
    warp_first(clash, t, clash_min + e);
    if (m) cur = idx;
  }
  if (live) lab[t] = cur;
}

// solver3d.inside_scene_pts for one point: union over shapes of (any
// within, inclusive) minus (any notin, strict)
__device__ __forceinline__ bool inside_scene(const Prim* __restrict__ prims, int np,
                                             double x, double y, double z) {
  bool total = false;
  int p = 0;
  while (p < np) {
    const int e = prims[p].elec, sh = prims[p].shape;
    bool w = false;
    while (p < np && prims[p].elec == e && prims[p].shape == sh) {
      const Prim& q = prims[p];
      if (q.role == 0) w = w || inside(q, q.in, x, y, z);
      else w = w && !inside(q, q.st, x, y, z);
      p++;
    }
    total = total || w;
  }
  return total;
}

// Whether primitive q can hold a point of the leg from x0 to x1 along axis
// ax (the other coordinates at p): a box or disc overlap with a margin, so
// that a primitive left out is outside at every probe of the leg, whatever
// the rounding.
__device__ __forceinline__ bool leg_near(const Prim& q, const double p[3], int ax, double x0,
                                         double x1) {
  double lo[3] = {p[0], p[1], p[2]}, hi[3] = {p[0], p[1], p[2]};
  lo[ax] = x0;
  hi[ax] = x1;
  const double* b = q.in;
  auto apart = [](double l, double h, double bl, double bh) {
    const double m = 1e-6 * (1.0 + fabs(l) + fabs(h) + fabs(bl) + fabs(bh));
    return l > bh + m || h < bl - m;
  };
  if (q.kind == 0) {
    if (apart(lo[2], hi[2], b[3], b[4])) return false;
    double rr = 0.0, s = 0.0;
    for (int a = 0; a < 2; a++) {
      const double d = b[a] < lo[a] ? lo[a] - b[a] : (b[a] > hi[a] ? b[a] - hi[a] : 0.0);
      rr += d * d;
      s += fabs(lo[a]) + fabs(hi[a]) + fabs(b[a]);
    }
    return !(rr > b[2] + 1e-6 * (1.0 + fabs(b[2]) + s * s));
  }
  return !(apart(lo[0], hi[0], b[0], b[1]) || apart(lo[1], hi[1], b[2], b[3]) ||
           apart(lo[2], hi[2], b[4], b[5]));
}

// inside_scene over the listed primitives (their table order kept).
__device__ __forceinline__ bool inside_listed(const Prim* __restrict__ prims, const int* list,
                                              int nl, double x, double y, double z) {
  bool total = false;
  int q = 0;
  while (q < nl) {
    const int e = prims[list[q]].elec, sh = prims[list[q]].shape;
    bool w = false;
    for (; q < nl && prims[list[q]].elec == e && prims[list[q]].shape == sh; q++) {
      const Prim& r = prims[list[q]];
      if (r.role == 0) w = w || inside(r, r.in, x, y, z);
      else w = w && !inside(r, r.st, x, y, z);
    }
    total = total || w;
  }
  return total;
}

// solver3d.fractions_from_scene: the leg of direction d at every vacuum
// node whose d-neighbour is metal (a low mirror plane sees node 1 from node
// 0), by `iters` bisections of the exact inside test; theta =
// float32(clip(0.5 (lo + hi), 1e-3, 1)), 1 everywhere else.
//
// Legs are few (a percent of the nodes) and cost thousands of FP64
// instructions each, so a block first queues those of its nodes in shared
// memory, writing 1 elsewhere, then gives each queued leg a thread; a leg
// tests only the primitives that can hold one of its points (leg_near),
// usually one or two.  97 x 97 x 193 nodes, 8 rings: 2933 us with
// a thread per node and direction over every primitive (the fill included)
// -> 183 us.
constexpr int kLegPrims = 8;
__global__ void __launch_bounds__(kT)
k_theta(const Prim* __restrict__ prims, int np, const uint8_t* __restrict__ metal,
        long nx, long ny, long nz, int mirror_bits, int iters,
        float* __restrict__ th) {
  __shared__ unsigned short queue[6 * kT];
  __shared__ int queued;
  const size_t n = (size_t)nx * ny * nz;
  const size_t t = (size_t)blockIdx.x * kT + threadIdx.x;
  const long len[3] = {nx, ny, nz};
  if (threadIdx.x == 0) queued = 0;
  __syncthreads();
  if (t < n) {
    const long c[3] = {(long)(t / ((size_t)nz * ny)), (long)((t / nz) % ny), (long)(t % nz)};
    const long step[3] = {ny * nz, nz, 1};
    const bool vacuum = !metal[t];
#pragma unroll
    for (int d = 0; d < 6; d++) {
      const int ax = d >> 1;
      // the neighbour's distance along the axis; a low mirror plane shows
      // node 0 the solid at node 1
      long q = (d & 1) ? 1 : -1;
      if (q < 0 && c[ax] == 0) q = ((mirror_bits >> ax) & 1) && len[ax] > 1 ? 1 : 0;
      if (q > 0 && c[ax] + q >= len[ax]) q = 0;
      if (vacuum && q != 0 && metal[t + q * step[ax]])
        queue[atomicAdd(&queued, 1)] = (unsigned short)(d * kT + threadIdx.x);
      else
        th[(size_t)d * n + t] = 1.0f;
    }
  }
  __syncthreads();
  const int nq = queued;
  for (int w = threadIdx.x; w < nq; w += kT) {
    const int d = queue[w] / kT, ax = d >> 1, step = (d & 1) ? 1 : -1;
    const size_t o = (size_t)blockIdx.x * kT + queue[w] % kT;
    const double p0[3] = {(double)(long)(o / ((size_t)nz * ny)), (double)(long)((o / nz) % ny),
                          (double)(long)(o % nz)};
    const bool mir = ((mirror_bits >> ax) & 1) && step < 0;
    // the probes' range (a mirrored one is reflected into the domain)
    double x0 = step > 0 ? p0[ax] : p0[ax] - 1.0;
    const double x1 = x0 + 1.0;
    if (mir && x0 < 0.0) x0 = 0.0;
    int list[kLegPrims], nl = 0;
    bool all = false;
    for (int q = 0; q < np; q++)
      if (leg_near(prims[q], p0, ax, x0, mir ? fmax(x1, 1.0) : x1)) {
        if (nl == kLegPrims) {
          all = true;
          break;
        }
        list[nl++] = q;
      }
    double lo = 0.0, hi = 1.0;
    for (int it = 0; it < iters; it++) {
      const double mid = __dmul_rn(0.5, __dadd_rn(lo, hi));
      double pr[3] = {p0[0], p0[1], p0[2]};
      pr[ax] = __dadd_rn(p0[ax], step > 0 ? mid : -mid);
      if (mir) pr[ax] = fabs(pr[ax]);
      const bool hit = all ? inside_scene(prims, np, pr[0], pr[1], pr[2])
                           : inside_listed(prims, list, nl, pr[0], pr[1], pr[2]);
      if (hit) hi = mid;
      else lo = mid;
    }
    double v = __dmul_rn(0.5, __dadd_rn(lo, hi));
    v = v < 1e-3 ? 1e-3 : (v > 1.0 ? 1.0 : v);
    th[(size_t)d * n + o] = __double2float_rn(v);
  }
}

// ---- extruded 2-D cross-sections (build_shapes3d.py, raster2d.py) -------
//
// A shape's cross-section is evaluated on its in-plane node coordinates
// (a_i, b_j) with the reference's float64 expressions (raster2d.py:113-
// 230): a rect (optionally rotated about its centre) or an ellipse with
// every edge moved out by the 1e-9 mm tolerance, or a polygon as a closed
// solid (even-odd interior or within 1e-9 mm of an edge).  The host passes
// the scalars already combined as the reference writes them.
struct XSec {
  int type;          // 0 rect, 1 ellipse, 2 polygon
  int rotated;       // rect
  double p[10];      // rect: cx, cy, ca, sa, xlo, xhi, ylo, yhi
                     // ellipse: cx, cy, rxT, ryT; polygon: tol2
};

__global__ void __launch_bounds__(kT)
k_xsection(XSec S, const double* __restrict__ poly, int npts, const double* __restrict__ a,
           long na, const double* __restrict__ b, long nb, uint8_t* __restrict__ out) {
  const size_t n = (size_t)na * nb;
  const size_t t = (size_t)blockIdx.x * kT + threadIdx.x;
  if (t >= n) return;
  const double X = a[t / nb], Y = b[t % nb];
  bool in = false;
  if (S.type == 0) {
    double xr = X, yr = Y;
    if (S.rotated) {
      const double cx = S.p[0], cy = S.p[1], ca = S.p[2], sa = S.p[3];
      const double dx = __dsub_rn(X, cx), dy = __dsub_rn(Y, cy);
      xr = __dsub_rn(__dadd_rn(cx, __dmul_rn(dx, ca)), __dmul_rn(dy, sa));
      yr = __dadd_rn(__dadd_rn(cy, __dmul_rn(dx, sa)), __dmul_rn(dy, ca));
    }
    in = xr >= S.p[4] && xr <= S.p[5] && yr >= S.p[6] && yr <= S.p[7];
  } else if (S.type == 1) {
    const double u = __ddiv_rn(__dsub_rn(X, S.p[0]), S.p[2]);
    const double v = __ddiv_rn(__dsub_rn(Y, S.p[1]), S.p[3]);
    in = __dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)) <= 1.0;
  } else {
    // poly rows: x0, y0, x1, y1, ex, ey, seg2 (7 x npts)
    const double* x0 = poly;
    const double* y0 = poly + npts;
    const double* x1 = poly + 2 * npts;
    const double* y1 = poly + 3 * npts;
    const double* ex = poly + 4 * npts;
    const double* ey = poly + 5 * npts;
    const double* sg = poly + 6 * npts;
    bool inside = false;
    for (int e = 0; e < npts; e++) {
      const double ax = x0[e], ay = y0[e], bx = x1[e], by = y1[e];
      if (ay == by) continue;
      const bool straddles = (ay > Y) != (by > Y);
      const double xint = __dadd_rn(
          ax, __ddiv_rn(__dmul_rn(__dsub_rn(Y, ay), __dsub_rn(bx, ax)), __dsub_rn(by, ay)));
      inside ^= straddles && (X < xint);
    }
    double d2 = __longlong_as_double(0x7ff0000000000000LL);  // +inf
    for (int e = 0; e < npts; e++) {
      double dj2;
      const double dx = __dsub_rn(X, x0[e]), dy = __dsub_rn(Y, y0[e]);
      if (sg[e] == 0.0) {
        dj2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
      } else {
        double tt = __ddiv_rn(__dadd_rn(__dmul_rn(dx, ex[e]), __dmul_rn(dy, ey[e])), sg[e]);
        tt = tt < 0.0 ? 0.0 : (tt > 1.0 ? 1.0 : tt);
        const double px = __dadd_rn(x0[e], __dmul_rn(tt, ex[e]));
        const double py = __dadd_rn(y0[e], __dmul_rn(tt, ey[e]));
        const double qx = __dsub_rn(X, px), qy = __dsub_rn(Y, py);
        dj2 = __dadd_rn(__dmul_rn(qx, qx), __dmul_rn(qy, qy));
      }
      d2 = dj2 < d2 ? dj2 : d2;
    }
    in = inside || d2 <= S.p[0];
  }
  out[t] = in ? 1 : 0;
}

// One extruded shape of the 3-D assembly: its electrode slot, extrusion
// axis (in-plane axes are the next two, cyclically), whether it is a
// cutout, and where its cross-section (na x nb bytes) and its range along
// the axis (one byte per node of that axis) start in the shared buffers.
struct ShapeRec {
  int slot, axis, cutout, pad;
  long long xs_off, rng_off;
  int na, nb;
};

// build_shapes3d.shapes_masks_3d + electrode_mask_3d: per node, electrodes
// in order; an electrode's shapes in order, additive shapes OR their
// volume in, cutouts AND NOT theirs; the node's label is the last
// electrode that claims it and a claim over an earlier one is a clash.
__global__ void __launch_bounds__(kT)
k_shapes_label(const ShapeRec* __restrict__ recs, int nrec, const uint8_t* __restrict__ xs,
               const uint8_t* __restrict__ rng, const int* __restrict__ eidx, int ne, long nx,
               long ny, long nz, int16_t* __restrict__ lab, unsigned long long* __restrict__ count,
               unsigned long long* __restrict__ clash_count,
               unsigned long long* __restrict__ clash_min) {
  const size_t n = (size_t)nx * ny * nz;
  const size_t t = (size_t)blockIdx.x * kT + threadIdx.x;
  const bool live = t < n;  // every lane stays for the warp's votes
  const size_t u = live ? t : 0;
  const long idx[3] = {(long)(u / ((size_t)nz * ny)), (long)((u / nz) % ny), (long)(u % nz)};
  int16_t cur = 0;
  int r = 0;
  for (int e = 0; e < ne; e++) {
    bool m = false;
    for (; r < nrec && recs[r].slot == e; r++) {
      const ShapeRec& q = recs[r];
      const int a1 = (q.axis + 1) % 3, a2 = (q.axis + 2) % 3;
      const bool v = live && rng[q.rng_off + idx[q.axis]] &&
                     xs[q.xs_off + (long long)idx[a1] * q.nb + idx[a2]];
      if (q.cutout)
        m = m && !v;
      else
        m = m || v;
    }
    m = m && live;
    if (!__any_sync(0xffffffffu, m)) continue;
    const bool clash = m && cur != 0;
    warp_count(m, count + e);
    warp_count(clash, clash_count + e);
    warp_first(clash, t, clash_min + e);
    if (m) cur = (int16_t)eidx[e];
  }
  if (live) lab[t] = cur;
}

}  // namespace
}  // namespace ig

using namespace ig;

namespace {
#define GK(x)                                                            \
  do {                                                                   \
    cudaError_t e_ = (x);                                                \
    if (e_ != cudaSuccess) {                                             \
      set_last_error(std::string(#x) + ": " + cudaGetErrorString(e_));   \
      return IG_CUDA_ERROR;                                              \
    }                                                                    \
  } while (0)

int check_table(const double* table, int n_prims) {
  for (int p = 0; p < n_prims; p++) {
    const double* r = table + 16 * p;
    if ((r[0] != 0.0 && r[0] != 1.0) || r[1] < 0 || (r[3] != 0.0 && r[3] != 1.0)) {
      set_last_error("malformed primitive table");
      return IG_BAD_ARG;
    }
    if (p > 0 && r[1] < table[16 * (p - 1) + 1]) {
      set_last_error("primitive table not in electrode order");
      return IG_BAD_ARG;
    }
  }
  return IG_OK;
}

// h: the host copy, which has to live until the stream is synchronised.
int upload_prims(const double* table, int n_prims, std::vector<Prim>& h, CallBuf& dev,
                 cudaStream_t s) {
  // table rows: kind, elec, shape, role, in[6], st[6]  (16 doubles)
  h.resize((size_t)(n_prims > 0 ? n_prims : 1));
  // a double bound as the first / last integer coordinate inside it (NaN:
  // none)
  auto first = [](double b) {
    return b != b ? INT_MAX : (int)std::max(-1e9, std::min(1e9, std::ceil(b)));
  };
  auto last = [](double b) {
    return b != b ? INT_MIN : (int)std::max(-1e9, std::min(1e9, std::floor(b)));
  };
  for (int p = 0; p < n_prims; p++) {
    const double* r = table + 16 * p;
    const double* in = r + 4;
    const bool box = r[0] != 0.0;
    for (int a = 0; a < 2; a++) {
      h[p].node[2 * a] = box ? first(in[2 * a]) : INT_MIN;
      h[p].node[2 * a + 1] = box ? last(in[2 * a + 1]) : INT_MAX;
    }
    h[p].node[4] = first(in[box ? 4 : 3]);
    h[p].node[5] = last(in[box ? 5 : 4]);
    h[p].kind = (int)r[0];
    h[p].elec = (int)r[1];
    h[p].shape = (int)r[2];
    h[p].role = (int)r[3];
    for (int a = 0; a < 6; a++) {
      h[p].in[a] = r[4 + a];
      h[p].st[a] = r[10 + a];
    }
  }
  cudaError_t e = dev.alloc(sizeof(Prim) * h.size(), s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(dev.p, h.data(), sizeof(Prim) * n_prims, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) {
    set_last_error(std::string("primitive upload: ") + cudaGetErrorString(e));
    return IG_CUDA_ERROR;
  }
  return IG_OK;
}
}  // namespace

extern "C" int ig_rasterize(const double* table, int n_prims,
                            const int* electrode_index, int n_electrodes,
                            long nx, long ny, long nz, int16_t* labels_out,
                            unsigned long long* counts_out,
                            unsigned long long* clash_counts_out,
                            unsigned long long* clash_first_out) {
  set_last_error("");
  if (!table || !electrode_index || !labels_out || n_prims < 0 || n_electrodes < 1 ||
      nx < 1 || ny < 1 || nz < 1) {
    set_last_error("invalid raster arguments");
    return IG_BAD_ARG;
  }
  if (int st = check_table(table, n_prims)) return st;
  cudaStream_t s = nullptr;
  if (int st = call_stream(&s)) return st;
  const CallInFlight call(kOtherCall);
  const size_t n = (size_t)nx * ny * nz;
  std::vector<Prim> host;
  CallBuf prims, eidx, lab, cnt;
  const CallSync sync{s};
  if (int st = upload_prims(table, n_prims, host, prims, s)) return st;
  GK(eidx.alloc(sizeof(int) * n_electrodes, s));
  GK(cudaMemcpyAsync(eidx.p, electrode_index, sizeof(int) * n_electrodes, cudaMemcpyHostToDevice, s));
  GK(lab.alloc(2 * n, s));
  GK(cnt.alloc(3 * 8 * (size_t)n_electrodes, s));
  unsigned long long* c = static_cast<unsigned long long*>(cnt.p);
  GK(cudaMemsetAsync(c, 0, 2 * 8 * (size_t)n_electrodes, s));
  GK(cudaMemsetAsync(c + 2 * n_electrodes, 0xff, 8 * (size_t)n_electrodes, s));
  const unsigned nb = (unsigned)((n + kT - 1) / kT);
  k_rasterize<<<nb, kT, 0, s>>>(static_cast<Prim*>(prims.p), n_prims,
                                static_cast<int*>(eidx.p), n_electrodes, nx, ny, nz,
                                static_cast<int16_t*>(lab.p), c, c + n_electrodes,
                                c + 2 * n_electrodes);
  GK(cudaGetLastError());
  GK(cudaMemcpyAsync(labels_out, lab.p, 2 * n, cudaMemcpyDeviceToHost, s));
  if (counts_out) GK(cudaMemcpyAsync(counts_out, c, 8 * n_electrodes, cudaMemcpyDeviceToHost, s));
  if (clash_counts_out)
    GK(cudaMemcpyAsync(clash_counts_out, c + n_electrodes, 8 * n_electrodes, cudaMemcpyDeviceToHost, s));
  if (clash_first_out)
    GK(cudaMemcpyAsync(clash_first_out, c + 2 * n_electrodes, 8 * n_electrodes,
                       cudaMemcpyDeviceToHost, s));
  GK(cudaStreamSynchronize(s));
  return IG_OK;
}

extern "C" int ig_theta_scene(const double* table, int n_prims, const uint8_t* metal,
                              long nx, long ny, long nz, int mirror_bits, int iters,
                              float* theta_out) {
  set_last_error("");
  if (!table || !metal || !theta_out || n_prims < 0 || nx < 1 || ny < 1 || nz < 1 ||
      iters < 0) {
    set_last_error("invalid theta arguments");
    return IG_BAD_ARG;
  }
  if (int st = check_table(table, n_prims)) return st;
  cudaStream_t s = nullptr;
  if (int st = call_stream(&s)) return st;
  const CallInFlight call(kOtherCall);
  const size_t n = (size_t)nx * ny * nz;
  std::vector<Prim> host;
  CallBuf prims, m, th;
  const CallSync sync{s};
  if (int st = upload_prims(table, n_prims, host, prims, s)) return st;
  GK(m.alloc(n, s));
  GK(cudaMemcpyAsync(m.p, metal, n, cudaMemcpyHostToDevice, s));
  GK(th.alloc(6 * n * 4, s));
  k_theta<<<(unsigned)((n + kT - 1) / kT), kT, 0, s>>>(
      static_cast<Prim*>(prims.p), n_prims, static_cast<uint8_t*>(m.p), nx, ny, nz, mirror_bits,
      iters, static_cast<float*>(th.p));
  GK(cudaGetLastError());
  GK(cudaMemcpyAsync(theta_out, th.p, 6 * n * 4, cudaMemcpyDeviceToHost, s));
  GK(cudaStreamSynchronize(s));
  return IG_OK;
}

extern "C" int ig_shape_xsection(int type, const double* params, int n_params,
                                 const double* poly, int n_points, const double* a, long na,
                                 const double* b, long nb, uint8_t* out) {
  set_last_error("");
  if (type < 0 || type > 2 || !params || n_params < 1 || n_params > 10 || !a || !b || !out ||
      na < 1 || nb < 1 || (type == 2 && (!poly || n_points < 1))) {
    set_last_error("invalid cross-section arguments");
    return IG_BAD_ARG;
  }
  cudaStream_t s = nullptr;
  if (int st = call_stream(&s)) return st;
  const CallInFlight call(kOtherCall);
  XSec S{};
  S.type = type;
  for (int q = 0; q < n_params; q++) S.p[q] = params[q];
  S.rotated = type == 0 && n_params >= 9 && params[8] != 0.0;
  const size_t n = (size_t)na * nb;
  CallBuf dp, da, db, dout;
  const CallSync sync{s};
  if (type == 2) {
    GK(dp.alloc(7 * sizeof(double) * n_points, s));
    GK(cudaMemcpyAsync(dp.p, poly, 7 * sizeof(double) * n_points, cudaMemcpyHostToDevice, s));
  }
  GK(da.alloc(8 * na, s));
  GK(db.alloc(8 * nb, s));
  GK(cudaMemcpyAsync(da.p, a, 8 * na, cudaMemcpyHostToDevice, s));
  GK(cudaMemcpyAsync(db.p, b, 8 * nb, cudaMemcpyHostToDevice, s));
  GK(dout.alloc(n, s));
  k_xsection<<<(unsigned)((n + kT - 1) / kT), kT, 0, s>>>(
      S, static_cast<double*>(dp.p), n_points, static_cast<double*>(da.p), na,
      static_cast<double*>(db.p), nb, static_cast<uint8_t*>(dout.p));
  GK(cudaGetLastError());
  note_launches(1);
  GK(cudaMemcpyAsync(out, dout.p, n, cudaMemcpyDeviceToHost, s));
  GK(cudaStreamSynchronize(s));
  return IG_OK;
}

extern "C" int ig_shapes_label(const long long* table, int n_shapes, const uint8_t* xs,
                               long long xs_len, const uint8_t* rng, long long rng_len,
                               const int* electrode_index, int n_electrodes, long nx, long ny,
                               long nz, int16_t* labels_out, unsigned long long* counts_out,
                               unsigned long long* clash_counts_out,
                               unsigned long long* clash_first_out) {
  set_last_error("");
  if (!table || n_shapes < 0 || !xs || !rng || !electrode_index || n_electrodes < 1 ||
      !labels_out || nx < 1 || ny < 1 || nz < 1) {
    set_last_error("invalid shape-label arguments");
    return IG_BAD_ARG;
  }
  const long len[3] = {nx, ny, nz};
  std::vector<ShapeRec> recs((size_t)(n_shapes > 0 ? n_shapes : 1));
  for (int q = 0; q < n_shapes; q++) {
    // rows: slot, axis, cutout, xs_off, rng_off (7 long longs with na, nb)
    const long long* r = table + 7 * q;
    ShapeRec& R = recs[q];
    R.slot = (int)r[0];
    R.axis = (int)r[1];
    R.cutout = (int)r[2];
    R.xs_off = r[3];
    R.rng_off = r[4];
    R.na = (int)r[5];
    R.nb = (int)r[6];
    const int a1 = (R.axis + 1) % 3, a2 = (R.axis + 2) % 3;
    if (R.axis < 0 || R.axis > 2 || R.slot < 0 || R.slot >= n_electrodes ||
        (q > 0 && R.slot < recs[q - 1].slot) || R.na != len[a1] || R.nb != len[a2] ||
        R.xs_off < 0 || R.xs_off + (long long)R.na * R.nb > xs_len || R.rng_off < 0 ||
        R.rng_off + len[R.axis] > rng_len) {
      set_last_error("malformed shape table");
      return IG_BAD_ARG;
    }
  }
  cudaStream_t s = nullptr;
  if (int st = call_stream(&s)) return st;
  const CallInFlight call(kOtherCall);
  const size_t n = (size_t)nx * ny * nz;
  CallBuf drec, dxs, drng, deidx, dlab, dcnt;
  const CallSync sync{s};
  GK(drec.alloc(sizeof(ShapeRec) * recs.size(), s));
  GK(cudaMemcpyAsync(drec.p, recs.data(), sizeof(ShapeRec) * recs.size(), cudaMemcpyHostToDevice, s));
  GK(dxs.alloc(xs_len > 0 ? xs_len : 1, s));
  if (xs_len > 0) GK(cudaMemcpyAsync(dxs.p, xs, xs_len, cudaMemcpyHostToDevice, s));
  GK(drng.alloc(rng_len > 0 ? rng_len : 1, s));
  if (rng_len > 0) GK(cudaMemcpyAsync(drng.p, rng, rng_len, cudaMemcpyHostToDevice, s));
  GK(deidx.alloc(sizeof(int) * n_electrodes, s));
  GK(cudaMemcpyAsync(deidx.p, electrode_index, sizeof(int) * n_electrodes, cudaMemcpyHostToDevice, s));
  GK(dlab.alloc(2 * n, s));
  GK(dcnt.alloc(3 * 8 * (size_t)n_electrodes, s));
  unsigned long long* c = static_cast<unsigned long long*>(dcnt.p);
  GK(cudaMemsetAsync(c, 0, 2 * 8 * (size_t)n_electrodes, s));
  GK(cudaMemsetAsync(c + 2 * n_electrodes, 0xff, 8 * (size_t)n_electrodes, s));
  k_shapes_label<<<(unsigned)((n + kT - 1) / kT), kT, 0, s>>>(
      static_cast<ShapeRec*>(drec.p), n_shapes, static_cast<uint8_t*>(dxs.p),
      static_cast<uint8_t*>(drng.p), static_cast<int*>(deidx.p), n_electrodes, nx, ny, nz,
      static_cast<int16_t*>(dlab.p), c, c + n_electrodes, c + 2 * n_electrodes);
  GK(cudaGetLastError());
  note_launches(1);
  GK(cudaMemcpyAsync(labels_out, dlab.p, 2 * n, cudaMemcpyDeviceToHost, s));
  if (counts_out) GK(cudaMemcpyAsync(counts_out, c, 8 * n_electrodes, cudaMemcpyDeviceToHost, s));
  if (clash_counts_out)
    GK(cudaMemcpyAsync(clash_counts_out, c + n_electrodes, 8 * n_electrodes, cudaMemcpyDeviceToHost, s));
  if (clash_first_out)
    GK(cudaMemcpyAsync(clash_first_out, c + 2 * n_electrodes, 8 * n_electrodes,
                       cudaMemcpyDeviceToHost, s));
  GK(cudaStreamSynchronize(s));
  return IG_OK;
}
