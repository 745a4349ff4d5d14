// fp64_int.cuh -- IEEE-754 binary64 square root, division and comparisons,
// round to nearest even, computed on the integer pipes.
//
// GB300 executes 2 FP64 operations per SM per clock (one warp instruction
// holds an SM sub-partition's FP64 pipe for 64 cycles), against 64 integer
// operations per SM per clock.  The hardware's correctly rounded sqrt and
// division are sequences of ~10 and ~7 FP64-pipe operations; the force law
// needs 7 and more of them per contact and is FP64-pipe bound with most issue
// slots idle.  The versions here take an FP32 seed, refine it in fixed point and
// settle the last bit with an exact integer rounding test, so they run
// beside the FP64 pipe instead of on it.  Results are bit-identical to the
// hardware's __dsqrt_rn / __ddiv_rn for every input: normal operands and zeros
// take the integer path; subnormal, infinite and NaN operands, and results
// outside the normal range, take the hardware instruction.  (Plain additions
// and multiplications stay on the FP64 pipe: one instruction there beats the
// ~30-40 integer instructions of an exact emulation, measured on GB300.)
//
// The functions are __host__ __device__ so that the CPU tests compare them
// with the host's IEEE arithmetic on billions of operands, including exact
// squares and quotients, ties, exponent extremes and deliberately degraded
// seeds.
#pragma once
#include <stdint.h>
#include <string.h>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline __attribute__((always_inline))
#endif

namespace fpi {

constexpr uint64_t kSign = 0x8000000000000000ull;
constexpr uint64_t kMant = 0x000FFFFFFFFFFFFFull;
constexpr uint64_t kHid = 0x0010000000000000ull;

__host__ __device__ __forceinline__ uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
__host__ __device__ __forceinline__ double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
__host__ __device__ __forceinline__ uint64_t mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
__host__ __device__ __forceinline__ int clz64(uint64_t v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
// the hardware operations, for the rare operands the integer paths leave out
__host__ __device__ __forceinline__ double hw_sqrt(double x) {
#ifdef __CUDA_ARCH__
  return __dsqrt_rn(x);
#else
  return __builtin_sqrt(x);
#endif
}
__host__ __device__ __forceinline__ double hw_div(double x, double y) {
#ifdef __CUDA_ARCH__
  return __ddiv_rn(x, y);
#else
  return x / y;
#endif
}
__host__ __device__ __forceinline__ uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return u;
#endif
}
__host__ __device__ __forceinline__ float ffrom(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}
// single-precision seeds: ~22 correct bits are all the refinement needs
__host__ __device__ __forceinline__ float rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  float r = 1.0f / __builtin_sqrtf(x);
#ifdef FPI_HOST_SEED_HOOK
  r = FPI_HOST_SEED_HOOK(r);
#endif
  return r;
#endif
}
__host__ __device__ __forceinline__ float rcp_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  float r = 1.0f / x;
#ifdef FPI_HOST_SEED_HOOK
  r = FPI_HOST_SEED_HOOK(r);
#endif
  return r;
#endif
}
__host__ __device__ __forceinline__ float log2_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return __builtin_log2f(x);
#endif
}
__host__ __device__ __forceinline__ float exp2_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  float r = __builtin_exp2f(x);
#ifdef FPI_HOST_SEED_HOOK
  r = FPI_HOST_SEED_HOOK(r);
#endif
  return r;
#endif
}
__host__ __device__ __forceinline__ int64_t smulhi(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (int64_t)(((__int128)a * b) >> 64);
#endif
}
// Q1.31 fixed point of a single-precision seed r in [1/4, 2)
__host__ __device__ __forceinline__ uint32_t q31_from_seed(float r) {
  const uint32_t rb = fbits(r);
  return ((rb << 8) | 0x80000000u) >> (127u - (rb >> 23));
}
__host__ __device__ __forceinline__ uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
__host__ __device__ __forceinline__ int64_t swide(int32_t a, int32_t b) { return (int64_t)a * b; }

// The refinements below run in 32x32-bit products: an operand enters a step
// with the bits the step's result can hold, and the residual of the last step
// (A - g^2, a*2^30 - q*b) is exact modulo 2^64 and small.  One lane's chain is
// what a small bed waits for (a warp of the force law runs 6 square roots and
// 9 quotients, one after the other), and at 1M spheres fewer instructions leave
// the FP64 pipe fewer gaps.
// The errors, with e0 the seed's: 2^-22 on the GPU, and still sound at 2^-17.

// sqrt(x), correctly rounded, for positive normal x: x = M * 2^(2h) with M in
// [1, 4).  r, a single-precision seed of 1/sqrt(M), takes one Newton step
// (r <- r + r*(1 - M r^2)/2) to within 2^-29; g = M r is corrected by the exact
// residual, g <- g + r*(M - g^2)/2 (Markstein, IBM J. Res. Dev. 34(1), 1990),
// to within 2^-56.  The candidate S = round(g * 2^52) is then settled by the
// exact integer test of round-to-nearest, S^2 - S < M*2^104 <= S^2 + S, and
// moved by one unit if it fails.
__host__ __device__ __forceinline__ uint64_t sqrt_normal(uint64_t u) {
  const uint64_t f = u & kMant;
  const int E = (int)((uint32_t)(u >> 52) & 0x7FFu) - 1023;
  const uint32_t odd = (uint32_t)E & 1u;
  const uint64_t A = ((f | kHid) << 10) << odd;            // M in Q2.62
  const uint32_t m = (uint32_t)(A >> 32);                  // M in Q2.30
  const uint32_t r0 = q31_from_seed(rsqrt_seed(ffrom(((127u + odd) << 23) | (uint32_t)(f >> 29))));
  const uint32_t p = (uint32_t)(wide(r0, r0) >> 31);       // r^2 in Q1.31
  const int32_t d = (int32_t)((int64_t)((1ull << 61) - wide(m, p)) >> 16);   // 1 - M r^2 in Q.45
  const uint32_t r = r0 + (uint32_t)(swide((int32_t)(r0 >> 1), d) >> 45);    // Q.75 / 2 to Q1.31
  const uint32_t g = (uint32_t)(wide(m, r) >> 31);         // ~sqrt(M) in Q2.30
  const int64_t res = (int64_t)(A - (wide(g, g) << 2));    // M - g^2 in Q.62, exact, below 2^37
  const int64_t c = swide((int32_t)(res >> 7), (int32_t)(r >> 1));            // Q.85
  uint64_t S = (((uint64_t)g << 31) + (uint64_t)(c >> 25) + (1u << 8)) >> 9;  // ~sqrt(M) * 2^52
  // D = M*2^104 - S^2, exact in 64 bits while S is within a few units
  const int64_t D = (int64_t)((A << 42) - S * S);
  S += (uint64_t)(D > (int64_t)S) - (uint64_t)(D <= -(int64_t)S);
  const int er = ((E - (int)odd) >> 1) + 1023;
  return (((uint64_t)(er - 1)) << 52) + S;
}
// operands for sqrt_normal: positive and normal
__host__ __device__ __forceinline__ bool sqrt_special(uint64_t u) { return (uint32_t)(u >> 52) - 1u >= 2046u; }
// the others: zeros, subnormals, negatives, infinities, NaN
__host__ __device__ __forceinline__ double sqrt_other(double x) {
  return (bits(x) << 1) == 0 ? x : hw_sqrt(x);   // sqrt(+-0) = +-0
}
__host__ __device__ __forceinline__ double sqrt_rn(double x) {
  const uint64_t u = bits(x);
  if (sqrt_special(u)) return sqrt_other(x);
  return from_bits(sqrt_normal(u));
}

// x / y, correctly rounded.  Normal x and y with a normal quotient take the
// integer path: the significand ratio Q = (mx/my) * 2^k in [1, 2) starts as
// q = mx * z with z a reciprocal of my to within 2^-29, is corrected by the exact
// remainder, q + (mx - q*my)*z, to within 2^-56, and the candidate
// S = round(Q * 2^52) is settled by the exact remainder R = mx*2^(52+k) - S*my
// (round to nearest: |R| < my/2; a quotient of two 53-bit significands never
// lies half-way) and moved by one unit if the test fails.  Zeros, subnormals,
// infinities, NaNs and quotients outside the normal range take the hardware
// division.  The refined reciprocal depends on y only, so several quotients by
// one divisor share it (Divisor).
struct Divisor {
  double y;
  uint64_t mb;    // significand of y, [2^52, 2^53)
  int64_t z;      // ~1/my in Q2.62
  uint32_t upper; // the same in Q1.31, within 2^-29
  uint32_t eb;    // biased exponent of y
  bool normal;
};

__host__ __device__ __forceinline__ Divisor divisor(double y) {
  Divisor v;
  v.y = y;
  const uint64_t b = bits(y);
  v.eb = (uint32_t)(b >> 52) & 0x7FFu;
  v.normal = v.eb - 1u < 2046u;
  v.mb = (b & kMant) | kHid;
  const uint32_t b31 = (uint32_t)(v.mb >> 21);             // my in Q1.31
  const float fb = ffrom((127u << 23) | (uint32_t)((v.mb & kMant) >> 29));
  const uint32_t z0 = q31_from_seed(rcp_seed(fb));
  // two Newton steps z <- z + z*(1 - my*z), the first in 32 bits.  div_by reads
  // the upper half only; where nothing else does, the second is not compiled.
  const int32_t d0 = (int32_t)((int64_t)((1ull << 62) - wide(b31, z0)) >> 17);   // Q.45
  const uint32_t z1 = z0 + (uint32_t)(swide((int32_t)(z0 >> 1), d0) >> 44);       // Q.75 to Q1.31
  const uint64_t B = v.mb << 11;                           // my in Q1.63
  const uint64_t t = wide((uint32_t)(B >> 32), z1) + (wide((uint32_t)B, z1) >> 32);   // my*z in Q2.62
  const int32_t d1 = (int32_t)((int64_t)((1ull << 62) - t) >> 5);                 // Q.57
  v.z = (int64_t)((uint64_t)z1 << 31) + (swide((int32_t)(z1 >> 1), d1) >> 25);    // Q.87 to Q2.62
  v.upper = z1;
  return v;
}

// bits of x / v.y; special: the quotient is not one of the integer path's
__host__ __device__ __forceinline__ uint64_t div_normal(uint64_t a, const Divisor& v, bool& special) {
  const uint32_t ea = (uint32_t)(a >> 52) & 0x7FFu;
  const uint64_t ma = (a & kMant) | kHid, mb = v.mb;
  const uint32_t k = ma < mb ? 1u : 0u;                    // Q = ma*2^k/mb in [1, 2)
  const int eq = (int)ea - (int)v.eb + 1023 - (int)k;
  special = ea - 1u >= 2046u || !v.normal || (uint32_t)(eq - 1) >= 2046u;
  const uint64_t mx = ma << k;
  const uint32_t q = (uint32_t)(wide((uint32_t)(mx >> 22), v.upper) >> 31);   // ~Q in Q2.30
  const int64_t rem = (int64_t)((mx << 30) - mb * q);      // exact, below 2^56
  const int64_t c = swide((int32_t)(rem >> 26), (int32_t)(v.upper >> 1));
  uint64_t S = ((uint64_t)q << 22) + (uint64_t)((c + (1ll << 33)) >> 34);   // ~Q * 2^52
  // R = ma*2^(52+k) - S*mb, exact in 64 bits while S is within a few units
  const int64_t R2 = (int64_t)((mx << 52) - S * mb) * 2, hb = (int64_t)mb;
  S += (uint64_t)(R2 > hb) - (uint64_t)(R2 < -hb);
  return ((a ^ bits(v.y)) & kSign) | ((((uint64_t)(eq - 1)) << 52) + S);
}
__host__ __device__ __forceinline__ double div_other(double x, const Divisor& v) {
  const uint64_t a = bits(x);
  if ((a << 1) == 0 && v.normal) return from_bits((a ^ bits(v.y)) & kSign);   // +-0 / normal
  return hw_div(x, v.y);
}
__host__ __device__ __forceinline__ double div_by(double x, const Divisor& v) {
  bool special;
  const uint64_t q = div_normal(bits(x), v, special);
  if (special) return div_other(x, v);
  return from_bits(q);
}

// x^0.2 and x^0.4 (the exponents as the nearest doubles: 0.2 + 2^-54/5 and its
// double), for positive normal x (+inf gives +inf).  x = M * 2^(5h) with M in
// [1, 32); z, a single-precision seed of M^(-1/5), is within e = 2^-20, and
// t = M z^4 is the root times (1 + e)^4.  d = 1 - t z = 1 - (1 + e)^5 gives the root
// as t (1 - d)^(-4/5), by the binomial series to d^3: the next term is below
// 2^-72.  The exponent's excess over 1/5 is the factor 1 + (2^-54/5) ln x.  The
// root is held in 62 bits: the results are within 0.53 and 0.56 ulp.  Two calls
// of pow keep a warp 11500 cycles (5760 each, measured).
__host__ __device__ __forceinline__ void fifth_powers(double x, double& x02, double& x04) {
  const uint64_t u = bits(x), f = u & kMant;
  const int e = (int)((u >> 52) & 0x7FFu);
  const int h5 = (e + 2) / 5, r = e + 2 - 5 * h5, h = h5 - 205;   // e - 1023 = 5 h + r
  const float fm = ffrom((uint32_t)(127 + r) << 23 | (uint32_t)(f >> 29));
  const float lg = log2_seed(fm);
  const uint32_t z = q31_from_seed(exp2_seed(-0.2f * lg));       // 24 significant bits
  const int s2 = r >= 3;                     // z^2 < 2^-s2: room for s2 more bits
  const uint64_t z2 = wide(z, z) << (1 + s2);                    // z^2 2^s2 in Q1.63, exact
  const uint64_t z4 = mulhi(z2, z2) << (r - 2 * s2);             // z^4 2^r in Q2.62
  const uint64_t t = mulhi((f | kHid) << 11, z4) << 1;           // M z^4 in Q2.62
  const uint64_t tz = (wide((uint32_t)(t >> 32), z) << 1) + (wide((uint32_t)t, z) >> 31);   // Q2.62
  const int64_t d = (int64_t)((1ull << 62) - tz);                // below 2^-17
  // s = d * (4/5 + d * (18/25 + d * 84/125)), Q2.62
  const int32_t d31 = (int32_t)(d >> 15);                        // Q.47
  const int32_t a = 1546188227 + (int32_t)(swide(d31, 1443109012) >> 47);      // 18/25 + .. in Q.31
  const uint64_t b = 0x3333333333333333ull + (uint64_t)(swide(d31, a) >> 16);  // 4/5 + .. in Q2.62
  const int64_t s = (int64_t)((uint64_t)smulhi(d, (int64_t)b) << 2);
  // (2^-54/5) ln x in units of 2^-62: 256/5 ln 2 log2 x = 35.4891... (5h + lg)
  const int32_t lx = h * 5 * 9085 + (int32_t)(fbits(lg * 9085.22f + 12582912.0f) - 0x4B400000u);   // 256 times
  const int64_t corr = s + (lx >> 8);
  const uint64_t T = t + ((uint64_t)smulhi((int64_t)(t >> 1), corr) << 3);   // root of M in Q2.62 (t may pass 2)
  const uint64_t T2 = mulhi(T, T);                               // its square in Q4.60
  // the binades (near a power of two the exponent's excess can cross one)
  const int k1 = clz64(T) - 1, k2 = clz64(T2) - 3;
  x02 = from_bits(((uint64_t)(h + 1022 - k1) << 52) + ((T + (1ull << (9 - k1))) >> (10 - k1)));
  x04 = from_bits(((uint64_t)(2 * h + 1022 - k2) << 52) + ((T2 + (1ull << (7 - k2))) >> (8 - k2)));
  if (e == 0x7FF) x02 = x04 = x;
}

__host__ __device__ __forceinline__ double div_rn(double x, double y) { return div_by(x, divisor(y)); }

// Square roots of N operands, and quotients of N by one divisor: the
// integer chains stand side by side, with one branch behind them for the
// operands that the integer path leaves out, so that they overlap (the branch
// of each call by itself keeps the compiler from that).
template <int N>
__host__ __device__ __forceinline__ void sqrt_many(const double (&x)[N], double (&r)[N]) {
  bool special = false;
#pragma unroll
  for (int i = 0; i < N; i++) {
    r[i] = from_bits(sqrt_normal(bits(x[i])));
    special |= sqrt_special(bits(x[i]));
  }
  if (special) {
#pragma unroll
    for (int i = 0; i < N; i++)
      if (sqrt_special(bits(x[i]))) r[i] = sqrt_other(x[i]);
  }
}
template <int N>
__host__ __device__ __forceinline__ void div_many(const double (&x)[N], const Divisor& v, double (&r)[N]) {
  bool sp[N], special = false;
#pragma unroll
  for (int i = 0; i < N; i++) {
    r[i] = from_bits(div_normal(bits(x[i]), v, sp[i]));
    special |= sp[i];
  }
  if (special) {
#pragma unroll
    for (int i = 0; i < N; i++)
      if (sp[i]) r[i] = div_other(x[i], v);
  }
}

// IEEE comparisons on the integer pipes (false with a NaN; +0 == -0): the
// bit patterns, with the magnitude bits of negatives flipped, order like the
// values.
__host__ __device__ __forceinline__ int64_t order_key(uint64_t u) {
  return (int64_t)(u ^ ((uint64_t)((int64_t)u >> 63) >> 1));
}
__host__ __device__ __forceinline__ bool unordered_or_zeros(uint64_t a, uint64_t b) {
  const uint64_t aa = a << 1, bb = b << 1;     // magnitudes, shifted out sign
  return aa > 0xFFE0000000000000ull || bb > 0xFFE0000000000000ull || (aa | bb) == 0;
}
__host__ __device__ __forceinline__ bool gt(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  return !unordered_or_zeros(a, b) && order_key(a) > order_key(b);
}
__host__ __device__ __forceinline__ bool lt(double x, double y) { return gt(y, x); }
__host__ __device__ __forceinline__ bool ge(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  const uint64_t aa = a << 1, bb = b << 1;
  if (aa > 0xFFE0000000000000ull || bb > 0xFFE0000000000000ull) return false;   // NaN
  if ((aa | bb) == 0) return true;                                                // +-0 >= +-0
  return order_key(a) >= order_key(b);
}
__host__ __device__ __forceinline__ bool le(double x, double y) { return ge(y, x); }

// floor(q) as an int when 0 <= floor(q) < n (q = -0 counts as 0), else -1;
// NaN and infinities give -1.  Integer work only.
__host__ __device__ __forceinline__ int floor_in_range(double q, int n) {
  const uint64_t u = bits(q);
  if ((u << 1) == 0) return n > 0 ? 0 : -1;
  if (u >> 63) return -1;                        // negative
  const uint32_t e = (uint32_t)(u >> 52);
  if (e < 1023u) return n > 0 ? 0 : -1;          // 0 < q < 1
  if (e > 1023u + 30u) return -1;                // >= 2^31, infinity, NaN
  const uint64_t v = ((u & kMant) | kHid) >> (1075u - e);
  return v < (uint64_t)n ? (int)v : -1;
}

// (q - k) in Q1.31, truncated, for the quotient q >= 0 and its floor k
// (0 <= k < 2^31).
__host__ __device__ __forceinline__ int32_t frac31(double q, int k) {
  const uint64_t u = bits(q);
  const uint32_t e = (uint32_t)(u >> 52) & 0x7FFu;
  const uint64_t m = (u & kMant) | (e ? kHid : 0ull);
  const int s = (e ? (int)e : 1) - 1023 - 20;    // q * 2^32 = m * 2^s, s <= 10
  const uint64_t qf = s >= 0 ? (m << s) : (s > -64 ? (m >> -s) : 0ull);
  return (int32_t)((qf - ((uint64_t)k << 32)) >> 1);
}

// floor(x / y) of the IEEE quotient as an int in [0, n), else -1 (as
// floor_in_range of div_by), and where x / y lies inside that unit: off31 =
// (x/y - floor) in Q1.31, within 2^-29 (an estimate for single-precision
// copies, not part of the exact result).  Fast path (positive normal x and y,
// quotient below 2^27): the quotient in Q32.32 from the divisor's reciprocal,
// error below 2^-30; the rounded quotient differs from the exact one by less
// than q*2^-53 < 2^-26, so when the estimate is at least 2^-20 from an integer
// both have the floor of the estimate.  Other operands, and estimates inside
// that band, take the exact division.
__host__ __device__ __forceinline__ int floor_div(double x, const Divisor& v, int n, int32_t& off31) {
  const uint64_t a = bits(x);
  const uint32_t ea = (uint32_t)(a >> 52);     // the sign bit makes negatives large
  const int sh = (int)ea - (int)v.eb;          // x/y = (mx/my) * 2^sh
  if (ea - 1u < 2046u && v.normal && (bits(v.y) >> 63) == 0 && sh <= 26) {
    const uint64_t ma = (a & kMant) | kHid;
    const uint64_t r61 = mulhi(ma << 11, (uint64_t)v.z);   // mx/my in Q3.61
    const int rs = 29 - sh;
    const uint64_t qf = rs >= 64 ? 0ull : (r61 >> rs);     // ~x/y in Q32.32
    const uint32_t fr = (uint32_t)qf;
    if (fr >= (1u << 12) && fr <= 0xFFFFFFFFu - (1u << 12)) {
      off31 = (int32_t)(fr >> 1);
      const uint64_t k = qf >> 32;
      return k < (uint64_t)n ? (int)k : -1;
    }
  }
  const double q = div_by(x, v);
  const int k = floor_in_range(q, n);
  off31 = k >= 0 ? frac31(q, k) : 0;
  return k;
}

// A single-precision copy of x for estimates: truncated (relative error below
// 2^-23) from the bits for normal x in the float range, else converted.
__host__ __device__ __forceinline__ float to_float_trunc(double x) {
  const uint64_t u = bits(x);
  const uint32_t e = (uint32_t)(u >> 52) & 0x7FFu;
  if (e - 897u < 254u)   // 2^-126 <= |x| < 2^128
    return ffrom((uint32_t)(u >> 63) << 31 | (e - 896u) << 23 | (uint32_t)((u & kMant) >> 29));
  return (float)x;
}

// (float)x, round to nearest even, on the integer pipes where x rounds to a
// normal float (the hardware conversion takes the FP64 pipe's rate on GB300);
// zeros, other results, infinities and NaNs take the hardware conversion.
__host__ __device__ __forceinline__ float to_float_rn(double x) {
  const uint64_t u = bits(x);
  const uint32_t e = (uint32_t)(u >> 52) & 0x7FFu;
  if (e - 897u < 253u) {   // 2^-126 <= |x| < 2^127: rounding up a binade stays finite
    const uint64_t m = (u & ~kSign) + 0x0FFFFFFFull + ((u >> 29) & 1ull);
    return ffrom((uint32_t)(u >> 63) << 31 | ((uint32_t)(m >> 29) - (896u << 23)));
  }
  return (float)x;
}

// x * (-0.5): the exponent field drops by one and the sign flips; a subnormal
// half is the rounded half of the bits (to even), infinities and NaN keep
// theirs.  No instruction of the FP64 pipe: the hardware multiplication for the
// rare operands was predicated, not branched over, and kept the pipe all the
// same (12 a sphere beside the update's 30; without it a step of 1M spheres takes
// 640 us instead of 646, of 200k 184 instead of 187.5).
__host__ __device__ __forceinline__ double mul_neg_half(double x) {
  const uint64_t u = bits(x), m = u & ~kSign;
  const uint32_t e = (uint32_t)(m >> 52);
  const uint64_t low = (m >> 1) + (m & (m >> 1) & 1ull);   // e < 2: bits are multiples of the least subnormal
  const uint64_t half = e >= 2047u ? m : (e >= 2u ? m - (1ull << 52) : low);
  return from_bits(half | ((u ^ kSign) & kSign));
}

}  // namespace fpi
