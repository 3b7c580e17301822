// IEEE binary64 division and square root (round to nearest even) computed on the integer pipe.
//
// On GB300 the FP64 unit of an SM sub-partition takes about 64 cycles per warp instruction, and the IEEE
// division and square root are sequences of several such instructions. The integer pipe issues a warp
// instruction every cycle or two. These functions produce the same correctly rounded result with 64-bit
// integer arithmetic and one single-precision approximation instruction, leaving the FP64 unit to the
// products of the solvers.
//
// Method (a Newton-type step in fixed point followed by an exact remainder test, as in Brent and Zimmermann,
// "Modern Computer Arithmetic" (2010), sections 3.4 and 3.5), laid out for a short dependency chain: one
// higher-order step in place of two Newton steps, 32 x 32 -> 64-bit multiply-adds in place of full 64-bit high
// products, and one correction of the last place in place of four.
//   division a / b: with mantissas A, B (53-bit integers, A scaled so that B <= A < 2B) and b = B / 2^53 in
//     [1/2, 1), r0 ~ 1 / b is the single-precision reciprocal. eps = 1 - b r0 is exact (a low 64-bit product),
//     and 1 / b = r0 (1 + eps + eps^2 + eps^3 + ...); the truncated series leaves eps^4 (below 2^-70 even for
//     starting points 40 units off). A r with 8 bits below the last place, biased down, gives the rounded
//     quotient or one less, and the sign of the exact remainder at the halfway point decides.
//   square root of x: with the mantissa M (53-bit integer, doubled when the exponent is odd) and m = M / 2^52 in
//     [1, 4), y0 ~ 1 / sqrt(m) is the single-precision reciprocal square root, eps = 1 - m y0^2,
//     1 / sqrt(m) = y0 (1 + eps / 2 + 3 eps^2 / 8 + 5 eps^3 / 16 + ...), and M y with 7 bits below the last place
//     gives the rounded root or one less; the sign of M 2^52 - (k + 1/2)^2 decides.
// Neither a quotient of normal numbers nor a square root falls halfway between two doubles.
// Cycles on GB300, one warp alone (latency) / per operation of a sub-partition's six warps (throughput): division
// 325 / 152, square root 420 / 159; with two Newton steps and four corrections 496 / 258 and 559 / 269; the FP64
// unit's own sequences 641 / 635 and 599 / 572.
// Infinities, NaNs, subnormal operands, zero divisors and results outside the normal range are passed to the
// hardware operation, which handles them by definition. Zero dividends and square roots of zero, which the
// solvers meet all the time, stay on the fast path: a warp with one such lane would otherwise run both.
//
// Every function is __host__ __device__: on the host the single-precision approximation is the exact
// reciprocal (optionally perturbed by a test), so the same integer steps can be compared against the host's
// IEEE operations.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef BG_HD
#ifdef __CUDACC__
#define BG_HD __host__ __device__ __forceinline__
#else
#define BG_HD inline
#endif
#endif

namespace bogus_gpu {
namespace ipipe {

constexpr uint64_t kMant = (uint64_t(1) << 52) - 1;
constexpr uint64_t kHidden = uint64_t(1) << 52;

// The device moves between a double and its bits are opaque to the optimiser, which would otherwise turn tests and
// sign changes written on the bits back into FP64 comparisons and negations (each an FP64 instruction).
BG_HD uint64_t to_bits(double x) {
#ifdef __CUDA_ARCH__
  uint64_t u;
  asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
  return u;
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
BG_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  double x;
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(u));
  return x;
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
BG_HD uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__float_as_uint(x);
#else
  uint32_t u;
  std::memcpy(&u, &x, 4);
  return u;
#endif
}
BG_HD float bitsf(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}
// high 64 bits of the 128-bit products
BG_HD uint64_t umulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
BG_HD int64_t smulhi(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (int64_t)(((__int128)a * b) >> 64);
#endif
}

// Single-precision approximations of 1/x and 1/sqrt(x) for x in [1/2, 4]. On the device: the approximate
// reciprocal and reciprocal square root instructions (rcp.approx.ftz.f32, rsqrt.approx.ftz.f32). On the
// host: the correctly rounded values moved by `host_ulps` units in the last place (a test sets it to show
// that the iteration tolerates approximations much worse than the hardware's).
#ifndef __CUDA_ARCH__
inline int& host_ulps() {
  static thread_local int u = 0;
  return u;
}
#endif
BG_HD float rcp_approx(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return bitsf(fbits(1.0f / x) + host_ulps());
#endif
}
BG_HD float rsqrt_approx(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return bitsf(fbits(1.0f / std::sqrt(x)) + host_ulps());
#endif
}

// v 2^(151 - f) for a float v in [2^(f - 127), 2^(f - 126)], from the line through its bit patterns there; for a v
// slightly below, the line's value (as far below again: a worse starting point by one bit, not an error)
BG_HD uint32_t fixed_of(float v, uint32_t f) { return 2u * fbits(v) - ((f - 1u) << 24); }
BG_HD uint64_t mul_wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
BG_HD uint32_t lo32(uint64_t v) { return (uint32_t)v; }
BG_HD uint32_t hi32(uint64_t v) { return (uint32_t)(v >> 32); }
BG_HD int32_t mulhi_s(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
// (a b) >> 64 without the low halves' product: low by at most two units
BG_HD uint64_t mulhi_est(uint64_t a, uint64_t b) {
  const uint64_t m1 = mul_wide(hi32(a), lo32(b)), m2 = mul_wide(lo32(a), hi32(b));
  return mul_wide(hi32(a), hi32(b)) + hi32(m1) + hi32(m2);
}
// (s r) >> 32 for a signed s, |s| < 2^62, and r < 2^26
BG_HD int64_t mul_shift32(int64_t s, uint32_t r) {
  return (int64_t)(int32_t)(s >> 32) * (int32_t)r + (int64_t)hi32(mul_wide((uint32_t)s, r));
}
// v + 1, or v when rem < 0
BG_HD uint64_t round_up(uint64_t v, uint64_t rem) { return (v + 1) + (uint64_t)(int64_t)((int32_t)hi32(rem) >> 31); }

// Correctly rounded a / b when b is normal and a is zero, or a and the quotient are normal; `ok` false otherwise
// (the returned value is then meaningless).
BG_HD double div_core(uint64_t ua, uint64_t ub, bool& ok) {
  const uint32_t ea = (uint32_t)(ua >> 52) & 0x7FFu, eb = (uint32_t)(ub >> 52) & 0x7FFu;
  uint64_t A = (ua & kMant) | kHidden;
  const uint64_t B = (ub & kMant) | kHidden;
  const bool lt = A < B;
  A <<= lt ? 1 : 0;  // A / B in [1, 2)
  const int e = (int)ea - (int)eb + 1023 - (lt ? 1 : 0);
  const uint64_t sign = (ua ^ ub) & (uint64_t(1) << 63);
  const bool zero = (ua << 1) == 0;
  ok = (eb - 1u < 2046u) && (zero || ((ea - 1u < 2046u) && (e >= 1) && (e <= 2045)));
  // r0 ~ 1 / b for b = B / 2^53 in [1/2, 1) from the leading 24 bits, as R0 / 2^24 (r0 from just below 1 to 2)
  const uint32_t R0 = fixed_of(rcp_approx(bitsf(0x3F000000u | (uint32_t)((B >> 29) & 0x7FFFFFu))), 127u);
  // eps = 1 - b r0, exact at 2^-77: the product's bits from 2^77 up are those of 1
  const int64_t E = -(int64_t)(B * R0);
  const int32_t Eh = (int32_t)(E >> 32);                // eps 2^45
  const int64_t e2 = (int64_t)Eh * Eh;                  // eps^2 2^90
  const int32_t e3 = mulhi_s((int32_t)(e2 >> 25), Eh);  // eps^3 2^78
  // r = r0 (1 + eps + eps^2 + eps^3) as R / 2^62
  const uint64_t R = ((uint64_t)R0 << 38) + (uint64_t)(mul_shift32(E + (e2 >> 13) + (e3 >> 1), R0) >> 7);
  // the rounded quotient or one less: q = A r 2^7 carries 8 bits below the last place, within 8 units
  const uint64_t m = (mulhi_est(A << 9, R) + (128 - 8)) >> 8;
  // the sign of A / B - (m + 1/2), which is never zero
  const uint64_t mant = round_up(m, (A << 53) - (2 * m + 1) * B);  // in [2^52, 2^53)
  return from_bits(zero ? sign : (sign | ((uint64_t)(uint32_t)(e - 1) << 52)) + mant);
}

// Correctly rounded sqrt(x) for a positive normal x or a zero; `ok` false otherwise.
BG_HD double sqrt_core(uint64_t ux, bool& ok) {
  const uint32_t ex = (uint32_t)(ux >> 52);  // sign included: negative x fails the range test
  const bool zero = (ux << 1) == 0;
  ok = zero || ex - 1u < 2046u;
  const bool odd = !(ex & 1u);  // the unbiased exponent ex - 1023 is odd
  const uint64_t M = ((ux & kMant) | kHidden) << (odd ? 1 : 0);  // m = M / 2^52 in [1, 4)
  // y0 ~ 1 / sqrt(m) from the leading 24 bits, as Y0 / 2^25 (y0 from just below 1/2 to 1)
  const uint32_t Y0 = fixed_of(
      rsqrt_approx(bitsf((odd ? 0x40000000u : 0x3F800000u) | (uint32_t)((ux >> 29) & 0x7FFFFFu))), 126u);
  // eps = 1 - m y0^2 at 2^-70 (the product's last 32 bits dropped)
  const uint64_t Z = mul_wide(Y0, Y0);
  const uint64_t P = hi32(mul_wide(lo32(M), lo32(Z))) + mul_wide(lo32(M), hi32(Z)) + mul_wide(hi32(M), lo32(Z)) +
                     ((uint64_t)(hi32(M) * hi32(Z)) << 32);
  const int64_t E = -(int64_t)P;
  const int32_t Eh = (int32_t)(E >> 26);                // eps 2^44
  const int64_t e2 = (int64_t)Eh * Eh;                  // eps^2 2^88
  const int32_t e3 = mulhi_s((int32_t)(e2 >> 25), Eh);  // eps^3 2^75
  // y = y0 (1 + eps / 2 + 3 eps^2 / 8 + 5 eps^3 / 16) as Y / 2^62; the sum in brackets less 1 at 2^-69
  const int64_t S = (E >> 2) + ((3 * e2) >> 22) + ((5 * e3) >> 10);
  const uint64_t Y = ((uint64_t)Y0 << 37) + (uint64_t)mul_shift32(S, Y0);
  // the rounded root or one less: M y 2^7 carries 7 bits below the last place, within 4 units
  const uint64_t m = (mulhi_est(M << 9, Y) + (64 - 4)) >> 7;
  // sqrt(M 2^52) > m + 1/2 when M 2^52 >= m (m + 1) + 1 (an integer, and never m (m + 1) + 1/4)
  const uint64_t mant = round_up(m, (M << 52) - m * (m + 1) - 1);
  return from_bits(zero ? ux : ((uint64_t)((ex + 1021u - (odd ? 1u : 0u)) >> 1) << 52) + mant);
}

// The hardware operations for the operands outside the fast domain, behind a call that the compiler cannot
// evaluate speculatively next to the integer path.
#ifdef __CUDA_ARCH__
__device__ __noinline__ double div_slow(double a, double b) { return a / b; }
__device__ __noinline__ double sqrt_slow(double x) { return sqrt(x); }
#else
inline double div_slow(double a, double b) { return a / b; }
inline double sqrt_slow(double x) { return std::sqrt(x); }
#endif

BG_HD double div_rn(double a, double b) {
  bool ok;
  double q = div_core(to_bits(a), to_bits(b), ok);
  if (!ok) q = div_slow(a, b);
  return q;
}
BG_HD double sqrt_rn(double x) {
  bool ok;
  double s = sqrt_core(to_bits(x), ok);
  if (!ok) s = sqrt_slow(x);
  return s;
}

// x * 2^k (k = -1 or 1 in the solvers): a change of the exponent field when x and the product are normal,
// the hardware product otherwise (zero, subnormal, infinite, NaN or out-of-range results).
#ifdef __CUDA_ARCH__
__device__ __noinline__ double mul_slow(double a, double b) { return a * b; }
#else
inline double mul_slow(double a, double b) { return a * b; }
#endif
template <int K>
BG_HD double scale2(double x) {
  const uint64_t u = to_bits(x);
  const int e = (int)((u >> 52) & 0x7FFu);
  double r = from_bits(u + (uint64_t)((int64_t)K << 52));
  if (!(e >= 1 && e <= 2046 && e + K >= 1 && e + K <= 2046)) r = mul_slow(x, K > 0 ? double(1 << K) : 1.0 / double(1 << -K));
  return r;
}

// x + 0.0: x itself, except -0.0, which becomes +0.0 (x finite)
BG_HD double plus_zero(double x) {
  const uint64_t u = to_bits(x);
  return from_bits(u == (uint64_t(1) << 63) ? 0 : u);
}

}  // namespace ipipe
}  // namespace bogus_gpu
