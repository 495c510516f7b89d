// fp64_div.cuh -- correctly rounded division by a divisor known in advance.
//
// The grid kernels divide many numerators by the same mesh spacing, and are bound by the FP64
// pipe.  div_by forms the quotient on the integer pipe: the significand of a times R, the
// first 64 bits of the divisor's reciprocal (formed on the host), is the quotient's
// significand with 10 or 11 bits to spare, at most 4 units of its 64th bit low.  Rounding
// it to 53 bits gives RN(a/b) unless the spare bits lie within those 4 units below one half (a
// quotient of two doubles is never half-way between two doubles): one quotient in 300, for
// which, and for operands outside the range, div_by_fp64 runs.  About 35 integer
// instructions, 14 cycles per warp and SM, in place of 4 to 5 FP64 ones, 90.
//
// div_by_fp64 (also used where the divisor is formed on the device): with y = RN(1/b), an
// IEEE division, a / b comes from one multiply and four fused multiply-adds:
//   q0 = RN(a y)                 within 1.5 ulp of a/b (y is within half an ulp of 1/b);
//   q1 = RN(q0 + RN(a - b q0) y) within half an ulp plus a tiny term: faithful;
//   q2 = RN(q1 + (a - b q1) y)   the remainder is exact for a faithful q1, and the
//                                result is RN(a/b) by Markstein's theorem (P. Markstein,
//                                IBM J. Res. Develop. 34(1):111-119, 1990; also
//                                Muller et al., Handbook of Floating-Point Arithmetic,
//                                section on Newton-Raphson based division).
// The theorem holds without underflow or overflow; the fast form is used for
// 2^-500 <= |a| <= 2^500 and a divisor in [2^-400, 2^400] (so every intermediate is a
// normal number), and the plain division otherwise (zero, subnormal, huge, Inf, NaN).
// The second correction is mostly a no-op: q1 already is RN(a/b) whenever the remainder
// r1 = a - b q1 (exact, q1 being faithful) is below half an ulp of q1 times |b|, that is
// |r1| < |b| 2^(e(q1) - 53), the bound of the rounding interval around a q1 that is not a
// power of two.  That test runs on the integer pipe (b's significand with the exponent
// e(b) + e(q1) - 53, compared with |r1| as bit patterns), so the common case costs one
// multiply and three fused multiply-adds; ties, powers of two, and thresholds outside
// the normal range take the full second correction.
// Both checked bit for bit against CUDA's division by mdz_rheo_div_selftest.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

#include "fp64_bits.cuh"
#include "fx64.cuh"

namespace mdz {

// a divisor b, its rounded reciprocal, whether the fast form may be used with it, and
// the biased exponent and significand field of |b| (for the remainder test)
struct Divisor {
  double b, y;
  int fast, eb;
  unsigned long long bman;
  unsigned long long R;  // floor(2^116 / significand of |b|), at most 2^64 - 1 (0 where formed on the device)
};

// the divisor as the kernels use it
__host__ __device__ inline Divisor make_divisor(double b) {
  Divisor d;
  d.b = b;
  d.y = 1.0 / b;
  const double m = b < 0 ? -b : b;
  d.fast = (m >= 0x1p-400 && m <= 0x1p400) ? 1 : 0;
  unsigned long long bits;
#if defined(__CUDA_ARCH__)
  bits = fp64_bits(m);
#else
  memcpy(&bits, &m, sizeof(bits));
#endif
  d.eb = (int)((bits >> 52) & 0x7ffu);
  d.bman = bits & 0xfffffffffffffull;
#if defined(__CUDA_ARCH__)
  d.R = 0;
#else
  const unsigned __int128 r = ((unsigned __int128)1 << 116) / (d.bman | 0x10000000000000ull);
  d.R = (r >> 64) ? ~0ull : (unsigned long long)r;
#endif
  return d;
}

// the second correction, out of line: taken where the remainder test cannot decide
static __device__ __noinline__ double div_by_correct(double r1, double y, double q1) { return __fma_rn(r1, y, q1); }

__device__ __forceinline__ double div_by_fp64(double a, const Divisor &d) {
  if (d.fast && fp64_exponent(a) - (1023u - 500u) <= 1000u) {
    const double q0 = __dmul_rn(a, d.y);
    const double q1 = __fma_rn(__fma_rn(-q0, d.b, a), d.y, q0);
    const double r1 = __fma_rn(-q1, d.b, a);
    unsigned lo, hi;
    fp64_words(q1, lo, hi);
    const int te = d.eb + (int)((hi >> 20) & 0x7ffu) - 1023 - 53;  // exponent of |b| ulp(q1) / 2
    const bool pow2 = ((hi & 0xfffffu) | lo) == 0u;
    if (!pow2 && te > 0 && te < 0x7ff &&
        (fp64_bits(r1) & kFp64AbsMask) < (((unsigned long long)te << 52) | d.bman))
      return q1;
    return div_by_correct(r1, d.y, q1);
  }
  return a / d.b;
}

static __device__ __noinline__ double div_by_rare(double a, double b, double y, int fast, int eb,
                                                  unsigned long long bman) {
  const Divisor d = {b, y, fast, eb, bman, 0};
  return div_by_fp64(a, d);
}

// the significand of |a / b| as a 64-bit number in (2^62, 2^64), at most 4 units low
__device__ __forceinline__ uint64_t div_significand(uint64_t abits, const Divisor &d) {
  return fx_mul64hi(fx_significand(abits) << 11, d.R);
}

// ZEROS: numerators are often zero (differences of a uniform field), and answered here.  Only
// where they are: the test costs the marker update, whose numerators are not, 0.5 %.
template <bool ZEROS = false>
__device__ __forceinline__ double div_by(double a, const Divisor &d) {
  const uint64_t ab = fx_bits(a);
  const uint32_t E = (fx_hi(ab) >> 20) & 0x7ffu;
  if (d.fast && E - (1023u - 500u) <= 1000u) {
    const uint64_t P = div_significand(ab, d);
    const int c = (int)(fx_hi(P) >> 31), sh = 10 + c;  // c: the quotient of the significands is at least 1
    const uint32_t half = 512u << c, low = fx_lo(P) & (2u * half - 1u);
    if (half - 1u - low >= 4u) {
      const uint64_t r = (P >> sh) + (low >= half ? 1 : 0);
      const uint64_t q = r + ((uint64_t)(uint32_t)((int)E - d.eb + 1021 + c) << 52);
      return fx_double(q | ((ab ^ fx_bits(d.b)) & 0x8000000000000000ull));
    }
  }
  if (ZEROS && d.fast && (ab << 1) == 0) return fx_double((ab ^ fx_bits(d.b)) & 0x8000000000000000ull);
  return div_by_rare(a, d.b, d.y, d.fast, d.eb, d.bman);
}

// a / s, correctly rounded, for s within 32 units of 2^-53 of 1 (a sum of weights), on the
// integer pipe: with s = 1 - k 2^-53 and ma the significand of a, the quotient's significand is
//     ma + (T + c) 2^-53,   T = ma k,  c = T k 2^-53 (1 + O(2^-48)) >= 0, below 2^11,
// rounded by its fraction.  false, and nothing formed, where the fraction lies within 8 units
// of 2^-53 below one half (c is taken to 4), where the quotient may leave a's binade, for other
// s, and for subnormal, huge or special a.
FX_FN bool div_near_one(double a, double s, double &out) {
  const uint64_t ab = fx_bits(a), sb = fx_bits(s);
  const int64_t up = (int64_t)(sb - 0x3ff0000000000000ull);  // s = 1 + up 2^-52, or 1 + up 2^-53 below 1
  const int64_t k = up > 0 ? -2 * up : -up;
  const uint32_t E = (fx_hi(ab) >> 20) & 0x7ffu;
  const uint64_t ma = fx_significand(ab);
  if ((ab << 1) == 0 && k <= 32 && k >= -32) { out = a; return true; }
  if (k > 32 || k < -32 || E - 23u > 2000u || ma - 0x10000000000040ull > 0xfffffffffff80ull) return false;
  const int64_t T = (int64_t)ma * k;                                  // |T| <= 2^58
  const int64_t U = T + (((T >> 27) * k) >> 26);                      // T + c
  const uint64_t half = 1ull << 52, frac = (uint64_t)U & (2 * half - 1);
  if (half - 1 - frac < 8) return false;
  const uint64_t r = ma + (uint64_t)(U >> 53) + (frac >= half ? 1 : 0);
  out = fx_double((ab & 0xfff0000000000000ull) | (r & 0xfffffffffffffull));
  return true;
}

// 1 / x, correctly rounded: the reciprocal of fx64.cuh, from 3 units of its 64th bit below to
// 2.1 above (60 M divisors, with the hardware's estimate one ulp off either way), rounded
// unless the spare bits lie within 4 units of one half (one in 250; then, and outside
// [2^-1000, 2^1000], the IEEE division).
static __device__ __noinline__ double recip_ieee(double x) { return 1.0 / x; }
__device__ __forceinline__ double recip_rn(double x) {
  const uint64_t b = fx_bits(x);
  const uint32_t E = (fx_hi(b) >> 20) & 0x7ffu;
  if (E - 23u <= 2000u) {
    const uint64_t Y = fx_recip_core(fx_significand(b) << 11);
    const uint32_t low = fx_lo(Y) & 0x7ffu;
    if (low - 1020u >= 8u)
      return fx_double(fx_bits(fx_assemble(Y, -(int)E + 1023 - 64)) | (b & 0x8000000000000000ull));
  }
  return recip_ieee(x);
}

// r / den for a Newton update, where a correctly rounded quotient is not needed (the
// iteration corrects a step's error on the next evaluation): the hardware reciprocal
// estimate (PTX rcp.approx.ftz.f64) refined by one Newton step, y (2 - den y), then
// r y -- three FP64 instructions in place of the general division.  den outside
// [2^-1000, 2^1000] (zero, subnormal, huge, Inf, NaN) takes the IEEE division.
__device__ __forceinline__ double newton_quotient(double r, double den) {
  if (fp64_exponent(den) - 23u > 2000u) return r / den;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
  y = __fma_rn(y, __fma_rn(-den, y, 1.0), y);
  return __dmul_rn(r, y);
}

// r / den within a couple of ulp, for a result that is an output but need not be
// correctly rounded (the parity bar is 1e-12 relative): the same reciprocal estimate
// refined by two Newton steps, y <- y + y (1 - den y), each of which squares the relative
// error of y until the rounding of the last step dominates, then r y -- five FP64
// instructions in place of the general division.  den outside [2^-1000, 2^1000] takes the
// IEEE division.  Checked against IEEE division by mdz_rheo_quotient_selftest.
__device__ __forceinline__ double quotient(double r, double den) {
  if (fp64_exponent(den) - 23u > 2000u) return r / den;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
  y = __fma_rn(y, __fma_rn(-den, y, 1.0), y);
  y = __fma_rn(y, __fma_rn(-den, y, 1.0), y);
  return __dmul_rn(r, y);
}

}  // namespace mdz
