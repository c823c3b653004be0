// ig_common.cuh -- shared device helpers for the ion_gym field-solve kernels.
//
// Exactness contract of the FP64 kernels: every FP64 operation is an explicit
// round-to-nearest intrinsic (__dadd_rn, __dmul_rn, __fma_rn, __ddiv_rn,
// __drcp_rn), so nothing is contracted or reassociated and each kernel returns
// the bits of the reference's float64 arithmetic (left-to-right evaluation,
// float32 theta products kept in float32, as the compiled reference types
// them).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ig {

// Even-reflection neighbour rule at every outer face (the ghost at -1 is
// node 1, the ghost at n is node n-2; a size-1 axis uses the node itself).
__host__ __device__ __forceinline__ long lo_nb(long i, long n) {
  return i > 0 ? i - 1 : (n > 1 ? 1 : i);
}
__host__ __device__ __forceinline__ long hi_nb(long i, long n) {
  return i < n - 1 ? i + 1 : (n > 1 ? n - 2 : i);
}

// x / 6.0 correctly rounded without the FP64 pipe (GB300 runs FP64 at
// about 1/64 of its integer rate, and the theta-free sweep is bound by it).
// x = M * 2^(E-52) with a 53-bit integer significand M, so x/6 =
// (N/3) * 2^(E-53-k) with N = M * 2^k, k = 1 when M >= 1.5 * 2^52 and 2
// otherwise, which puts N/3 in [2^52, 2^53).  Q = floor(N/3) (one 64-bit
// multiply-high by ceil(2^65/3)) and the remainder r = N - 3Q is 0, 1 or 2:
// the discarded fraction r/3 is never one half, so RN(N/3) is Q + (r == 2),
// and Q + 1 never reaches 2^53 (that would need N = 3*2^53 - 1, odd).  The
// result is Q with the biased exponent lowered by 1 + k.  Zeros return
// themselves (sign kept; cold starts are mostly zeros); exponents whose
// quotient would be subnormal (biased below 4), infinities and NaNs take the
// hardware division.  Checked bit-for-bit against x/6.0 by the test-suite.
__device__ __forceinline__ double div6(double x) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
  const unsigned eb = (static_cast<unsigned>(b >> 32) >> 20) & 0x7ffu;
  if (eb - 4u > 2042u) {
    if ((b << 1) == 0ULL) return x;
    return __ddiv_rn(x, 6.0);
  }
  const unsigned long long m = (b & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
  const unsigned k = m >= 0x0018000000000000ULL ? 1u : 2u;
  const unsigned long long n = m << k;
  const unsigned long long q0 = __umul64hi(n, 0xAAAAAAAAAAAAAAABULL) >> 1;
  const unsigned r = static_cast<unsigned>(n) - 3u * static_cast<unsigned>(q0);
  const unsigned long long q = q0 + (r == 2u ? 1ULL : 0ULL);
  // q carries the implicit bit 2^52, so adding it to the exponent field
  // (eb - 2 - k) << 52 sets the exponent to eb - 1 - k
  const unsigned long long mag =
      (static_cast<unsigned long long>(eb - 2u - k) << 52) + q;
  return __longlong_as_double(static_cast<long long>((b & 0x8000000000000000ULL) | mag));
}

// |d| as an order-preserving 64-bit key (d >= 0, so the IEEE bit pattern
// orders like the value).  NaN maps to 0: the reference's "if d > dmax"
// never takes a NaN.
__device__ __forceinline__ unsigned long long absbits(double d) {
  unsigned long long b =
      static_cast<unsigned long long>(__double_as_longlong(d)) & 0x7fffffffffffffffULL;
  return b > 0x7ff0000000000000ULL ? 0ULL : b;
}

// The FP64 operations behind the integer forms below, as calls: written in
// line, a fallback this short is predicated instead of branched around, and
// instructions that every lane has switched off still take their turn in
// the FP64 pipe -- 3 on top of the sum's 5.
static __device__ __noinline__ double sor_slow(double old, double q, double omega) {
  return __dadd_rn(old, __dmul_rn(omega, __dsub_rn(q, old)));
}
static __device__ __noinline__ double sub_slow(double a, double b) { return __dsub_rn(a, b); }
static __device__ __noinline__ double resid_slow(double S, double phi) {
  return __dsub_rn(S, __dmul_rn(6.0, phi));
}

// One node of a sweep from its quotient q: nw = RN(old + RN(omega * RN(q -
// old))), the key of |RN(nw - old)| to *key when DELTA, on the integer pipe
// where that is exact, so that a node costs the FP64 pipe its neighbour sum
// alone (the pipe does 2 lanes per clock and SM, the integer pipe 64; the
// sweep is bound by the former).
//
//  * difference: q = Mq*2^(eq-1075) and old = Mo*2^(eo-1075) (53-bit integer
//    significands, biased exponents no more than one apart) differ by the
//    exact integer D = +-Mq*2^(eq-e) -+ Mo*2^(eo-e), e the smaller exponent;
//    when |D| < 2^53 it is RN(q - old) itself.
//  * omega 1 (ONE): then old + D is q, exactly.
//  * step: omega's significand W times |D| is formed with both normalised,
//    so its top bit is one of two places, and rounded once to the 53 bits m
//    (to nearest, ties to even; a set low bit stands for every bit below).
//  * sum: in units of old's ulp / 512, old is Mo*2^9 and the step m*2^9
//    shifted right by the exponents' distance, again with a low bit for
//    what is shifted out (an even half-way point is never mistaken for
//    it); while the sum keeps old's exponent its rounding to a multiple of
//    2^9 is RN(old + step), and the integer |rr - Mo| is |nw - old|.
//    (Leaving the half-way cases to the FP64 operations saves ten integer
//    instructions and loses: omega 1.85 is 37/20, whose products are halves
//    once in twenty lanes, so most warps would run both paths: 68 against 52
//    us a half-sweep of a 257^3 quadrupole.)
//
// Zero on zero stays +0 (cold starts are mostly zeros).  Everything else
// (other zeros, subnormals, exponents further apart, a rounded difference, a
// subnormal step, a sum that leaves old's binade, omega not a positive
// normal number) takes the FP64 operations as the reference writes them.
// Checked bit-for-bit against those by the test-suite.
//
// The 257^3 quadrupole's cascadic solve (omega 1.85): 278 ms with the
// difference and the product alone on the integer pipe (6 FP64 instructions
// a node), 250 ms now (5, the neighbour sum).  The FP64 pipe is then 72 %
// busy and the integer pipe 60 % (counters of a 257^3 half-sweep), so an
// addition of the sum moved over would cost there what it saves here.
__device__ __forceinline__ unsigned long long sor_key(unsigned long long ad, int e) {
  // the IEEE bits of ad * 2^(e - 1075), 0 < ad < 2^54, where that is normal;
  // ~0 where it is not
  const int lz = __clzll(static_cast<long long>(ad)) - 11;
  const unsigned long long m = lz >= 0 ? ad << lz : ad >> 1;  // lz = -1: ad is even
  return e - lz >= 1 ? (static_cast<unsigned long long>(e - lz - 1) << 52) + m : ~0ULL;
}

template <bool DELTA, bool ONE>
__device__ __forceinline__ double sor_apply(double old, double q, double omega,
                                            unsigned long long* key) {
  constexpr unsigned long long kFrac = 0x000fffffffffffffULL, kHid = 0x0010000000000000ULL;
  const unsigned long long bq = static_cast<unsigned long long>(__double_as_longlong(q));
  const unsigned long long bo = static_cast<unsigned long long>(__double_as_longlong(old));
  const unsigned long long bw = static_cast<unsigned long long>(__double_as_longlong(omega));
  const int eq = static_cast<int>(bq >> 52) & 0x7ff, eo = static_cast<int>(bo >> 52) & 0x7ff;
  const int ew = static_cast<int>(bw >> 52);  // sign bit included
  const int emin = min(eq, eo), de = eq - eo;
  const bool wok = ONE || static_cast<unsigned>(ew - 1) < 2046u;
  const unsigned long long mo = (bo & kFrac) | kHid, mq = (bq & kFrac) | kHid;
  const unsigned long long a = de > 0 ? mq << 1 : mq, b = de < 0 ? mo << 1 : mo;
  const bool opp = static_cast<long long>(bq ^ bo) < 0;
  const long long dd = static_cast<long long>(opp ? a + b : a - b);
  const unsigned long long ad = static_cast<unsigned long long>(dd < 0 ? -dd : dd);
  bool ok = wok && static_cast<unsigned>(eq - 1) < 2046u && static_cast<unsigned>(eo - 1) < 2046u &&
            static_cast<unsigned>(de + 1) <= 2u && (ad >> 53) == 0ULL;
  unsigned long long k = 0;
  double nw;
  if (ONE) {
    nw = q;
    if (DELTA && ad) {
      k = sor_key(ad, emin);
      ok = ok && k != ~0ULL;
    }
  } else {
    const int lz = __clzll(static_cast<long long>(ad | 1ULL));
    const unsigned long long an = ad << lz, wn = ((bw & kFrac) | kHid) << 10;
    const unsigned long long hi = __umul64hi(wn, an), lo = wn * an;
    const int s = 9 + static_cast<int>(hi >> 62);
    const unsigned long long h = hi | (lo ? 1ULL : 0ULL);
    const unsigned long long m = (h + ((1ULL << (s - 1)) - 1ULL) + ((h >> s) & 1ULL)) >> s;
    const int eu = emin + ew + s - lz - 1021;  // the step is m * 2^(eu - 1075)
    const int sh = min(eo - eu, 63);
    const unsigned long long m9 = m << 9, t0 = m9 >> (sh & 63);
    const unsigned long long t = t0 | ((t0 << (sh & 63)) != m9 ? 1ULL : 0ULL);
    const unsigned long long A = mo << 9;
    // the step has q's sign if |q|'s side of the difference won, and old's
    // side if not: it adds to |old| when q and old agree and |q| is larger
    const unsigned long long R = (!opp && dd > 0) ? A + t : A - t;
    const unsigned long long rr = (R + 255ULL + ((R >> 9) & 1ULL)) >> 9;
    const unsigned long long out = (bo & 0x8000000000000000ULL) |
                                   ((static_cast<unsigned long long>(eo - 1) << 52) + rr);
    nw = ad ? __longlong_as_double(static_cast<long long>(out)) : old;
    ok = ok && (!ad || (eu >= 1 && sh >= 0 && (R >> 61) == 1ULL));
    if (DELTA && ad && rr != mo) {
      k = sor_key(rr > mo ? rr - mo : mo - rr, eo);
      ok = ok && k != ~0ULL;
    }
  }
  if (!ok) {
    if (wok && ((bq | bo) << 1) == 0ULL) {
      nw = 0.0;
      k = 0;
    } else {
      nw = sor_slow(old, q, ONE ? 1.0 : omega);
      if (DELTA) k = absbits(sub_slow(nw, old));
    }
  }
  if (DELTA) *key = k;
  return nw;
}

// RN(S - RN(6 phi)), the residual of a node whose legs are all 1, on the
// integer pipe where that is exact: 6 phi's significand is 3 Mo rounded by
// one or two bits, and the difference of two numbers at most one binade
// apart is an exact integer (see sor_apply).  Zero minus zero, and every
// case that is not exact, take the FP64 operations.  Checked against them
// by the test-suite.
__device__ __forceinline__ double resid6(double S, double phi) {
  constexpr unsigned long long kFrac = 0x000fffffffffffffULL, kHid = 0x0010000000000000ULL;
  const unsigned long long bs = static_cast<unsigned long long>(__double_as_longlong(S));
  const unsigned long long bo = static_cast<unsigned long long>(__double_as_longlong(phi));
  const int es = static_cast<int>(bs >> 52) & 0x7ff, eo = static_cast<int>(bo >> 52) & 0x7ff;
  const unsigned long long m3 = 3ULL * ((bo & kFrac) | kHid);  // [3, 6) * 2^52
  const int sh = 1 + static_cast<int>(m3 >> 54);
  const unsigned long long mp =
      (m3 + ((1ULL << (sh - 1)) - 1ULL) + ((m3 >> sh) & 1ULL)) >> sh;  // up to 2^53
  const int ep = eo + 1 + sh;  // 6 phi = mp * 2^(ep - 1075)
  const unsigned long long ms = (bs & kFrac) | kHid;
  const int emin = min(es, ep), de = es - ep;
  const unsigned long long a = de > 0 ? ms << 1 : ms, b = de < 0 ? mp << 1 : mp;
  const bool opp = static_cast<long long>(bs ^ bo) < 0;
  const long long dd = static_cast<long long>(opp ? a + b : a - b);
  const unsigned long long ad = static_cast<unsigned long long>(dd < 0 ? -dd : dd);
  const bool ok = static_cast<unsigned>(es - 1) < 2046u && static_cast<unsigned>(eo - 1) < 2040u &&
                  static_cast<unsigned>(de + 1) <= 2u && (ad >> 53) == 0ULL;
  const unsigned long long k = ad ? sor_key(ad, emin) : 0ULL;
  if (ok && k != ~0ULL)  // an exact zero difference is +0
    return __longlong_as_double(static_cast<long long>(
        k | (ad ? (bs ^ (dd < 0 ? 0x8000000000000000ULL : 0ULL)) & 0x8000000000000000ULL
                : 0ULL)));
  return resid_slow(S, phi);
}

// Warp max of a 64-bit key with two 32-bit warp reductions (REDUX): the
// largest high word, then the largest low word among the lanes holding it.
// Every lane of the warp must call it.
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32));
  const unsigned lo =
      __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0u);
  return ((unsigned long long)hi << 32) | lo;
}

// Block-wide max of a 64-bit key, then one atomicMax into *dst -- only when
// it beats the value already there, so the tens of thousands of blocks of a
// launch do not all queue atomics on one address.  Every thread of the
// block must call it.
__device__ __forceinline__ void block_max_to(unsigned long long v,
                                             unsigned long long* dst) {
  __shared__ unsigned long long red[32];
  v = warp_max_u64(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? red[lane] : 0ULL;
    v = warp_max_u64(v);
    if (lane == 0 && v && v > *reinterpret_cast<volatile unsigned long long*>(dst))
      atomicMax(dst, v);
  }
}

// float -> double by its bits for zeros and normal floats (exponent rebias,
// significand moved up 29 bits); subnormals, infinities and NaN convert on
// the FP64 pipe (a call, so that they alone pay for it).
static __device__ __noinline__ double widen_slow(float d) { return (double)d; }
__device__ __forceinline__ double widen(float d) {
  const unsigned fb = __float_as_uint(d);
  const unsigned ef = (fb >> 23) & 0xffu;
  if (ef - 1u < 254u)
    return __longlong_as_double(static_cast<long long>(
        (static_cast<unsigned long long>(fb & 0x80000000u) << 32) |
        (static_cast<unsigned long long>(ef + 896u) << 52) |
        (static_cast<unsigned long long>(fb & 0x7fffffu) << 29)));
  if ((fb & 0x7fffffffu) == 0u)
    return __longlong_as_double(static_cast<long long>(static_cast<unsigned long long>(fb) << 32));
  return widen_slow(d);
}

__host__ __device__ __forceinline__ double bits_to_double(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(b));
#else
  double d;
  __builtin_memcpy(&d, &b, 8);
  return d;
#endif
}

}  // namespace ig
