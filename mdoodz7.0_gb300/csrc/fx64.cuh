// fx64.cuh -- exp, log, reciprocal, square root and sine/cosine of doubles in 64-bit fixed
// point, on the integer pipe.
//
// GB300 issues an FP64 instruction once per 64 cycles and scheduler (about 20 cycles per
// warp instruction and SM, measured with all four schedulers busy), while a 32-bit
// multiply-high takes 1.1, a wide multiply 1.4, and a shift, logic operation or addition
// 0.2-0.6 cycles: one FP64 instruction costs as much as 30 to 60 integer ones, and the
// integer ones issue beside it for free (a chain of one DFMA and 18 integer instructions
// runs at the DFMA's own rate).  The functions here therefore take a double apart, work on
// its significand as a 64-bit integer, and put the result together with the exponent, with
// no FP64 instruction at all.  Notation: Qa.b is a fixed-point number with b fraction bits.
//
//   fx_exp    61 integer instructions in place of 10 FP64 ones (fp64_math.cuh's exp)
//   fx_log    about 75 in place of 12
//   fx_recip  about 35 in place of 4 and the hardware estimate
//   fx_sqrt   about 45 in place of CUDA's 8-9
//   fx_sincos about 110 in place of CUDA's 30-40
//   fx_pow    about 170 in place of CUDA's 60 and more
//
// Used throughout the isotropic and anisotropic sweeps they took the 2049 x 2049 sweep from
// 17.22 to 15.58 ms and the anisotropic 1025 x 1025 one from 2.97 to 2.58 ms, with the same
// errors against 64-bit references.
//
// The methods are the classical ones: table-driven reduction and a short polynomial (P. T.
// P. Tang, ACM TOMS 15(2), 1989, and 16(4), 1990) for exp and log; a second-order Newton
// step on a 24-bit estimate for the reciprocal and the reciprocal square root; the addition
// theorems on a table of step 1/256 for sine and cosine.  Every intermediate carries 56 or
// more bits behind the result's leading one, so the results are within 0.7 ulp (exp
// and log: 0.8) of the exact values; arguments outside the ranges stated at each function take
// CUDA's own function, special values included.
//
// The code compiles for the host too (the CPU test runs it there); only the starting
// estimates differ (CUDA's approximate reciprocal against a division).
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define FX_FN __host__ __device__ __forceinline__
#define FX_DEV __device__ __forceinline__
#else
#include <math.h>
#define FX_FN static inline
#define FX_DEV static inline
#endif

#include "fx64_tables.inc"

namespace mdz {

#ifdef __CUDACC__
// read through the read-only cache, like the tables of fp64_math.cuh
__device__ const unsigned long long g_fx_exp2[256] = MDZ_FX_EXP2_TABLE;  // 2^(j/256), Q2.62
__device__ const unsigned long long g_fx_logc[256] = MDZ_FX_LOGC_TABLE;  // -log(c_j), Q0.64
__device__ const unsigned int g_fx_c[256] = MDZ_FX_C_TABLE;              // c_j, Q16: 1 / (1 + (j + 1/2) / 256)
__device__ const ulonglong2 g_fx_sincos[384] = MDZ_FX_SINCOS_TABLE;      // (sin, cos)(j/256), Q0.63
#endif
static const unsigned long long h_fx_exp2[256] = MDZ_FX_EXP2_TABLE;
static const unsigned long long h_fx_logc[256] = MDZ_FX_LOGC_TABLE;
static const unsigned int h_fx_c[256] = MDZ_FX_C_TABLE;
struct FxPair { unsigned long long x, y; };
static const FxPair h_fx_sincos[384] = MDZ_FX_SINCOS_TABLE;

#if defined(__CUDA_ARCH__)
#define FX_TAB(name, i) __ldg(&g_fx_##name[i])
#else
#define FX_TAB(name, i) (h_fx_##name[i])
#endif

// CUDA's functions for the arguments outside the fast ranges, out of line: inlined, the
// compiler runs their first FP64 instructions ahead of the branch that selects them.
#if defined(__CUDACC__)
static __device__ __noinline__ double fx_exp_rare(double x) { return exp(x); }
static __device__ __noinline__ double fx_log_rare(double x) { return log(x); }
static __device__ __noinline__ double fx_recip_rare(double x) { return 1.0 / x; }
static __device__ __noinline__ double fx_sqrt_rare(double x) { return sqrt(x); }
static __device__ __noinline__ double fx_pow_rare(double x, double y) { return pow(x, y); }
static __device__ __noinline__ double2 fx_sincos_rare(double x) {
  double2 r;
  sincos(x, &r.x, &r.y);
  return r;
}
#endif
#if defined(__CUDA_ARCH__)
#define FX_RARE(f, plain, x) fx_##f##_rare(x)
#define FX_RARE2(f, plain, x, y) fx_##f##_rare(x, y)
#else
#define FX_RARE(f, plain, x) (plain)
#define FX_RARE2(f, plain, x, y) (plain)
#endif

// ---- 32- and 64-bit pieces -----------------------------------------------------------------
FX_FN uint32_t fx_umulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
FX_FN int32_t fx_mulhi(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
FX_FN uint32_t fx_hi(uint64_t x) { return (uint32_t)(x >> 32); }
FX_FN uint32_t fx_lo(uint64_t x) { return (uint32_t)x; }
// floor(a b / 2^64) less at most 2: the product of the low words is left out
FX_FN uint64_t fx_mul64hi(uint64_t a, uint64_t b) {
  return (uint64_t)fx_hi(a) * fx_hi(b) + fx_umulhi(fx_hi(a), fx_lo(b)) + fx_umulhi(fx_lo(a), fx_hi(b));
}
FX_FN int fx_clz(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
// the leading 32 bits of (hi:lo) << s, 0 <= s < 32
FX_FN uint32_t fx_funnel(uint32_t lo, uint32_t hi, int s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
FX_FN uint64_t fx_bits(double x) {
#if defined(__CUDA_ARCH__)
  uint32_t lo, hi;  // opaque, so that tests on the bits stay on the integer pipe (fp64_bits.cuh)
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
  return ((uint64_t)hi << 32) | lo;
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
FX_FN double fx_double(uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
// 53-bit significand with its hidden bit
FX_FN uint64_t fx_significand(uint64_t b) { return (b & 0xfffffffffffffull) | 0x10000000000000ull; }

// V 2^e as a double, rounded to nearest, for V with its top bit set and a result in the
// normal range
FX_FN double fx_assemble(uint64_t V, int e) {
  // (V + half) >> 11 is the significand with its hidden bit, which adds 1 to the exponent
  // field; a carry out of V + half (V close to 2^64) would be lost, so half is added after
  // the shift
  const uint64_t r = (V >> 11) + ((V >> 10) & 1);
  return fx_double(r + ((uint64_t)(uint32_t)(e + 63 + 1022) << 52));
}

// V 2^e for any V != 0
FX_FN double fx_normalise(uint64_t V, int e) {
  if (fx_hi(V) == 0) { V <<= 32; e -= 32; }
  const int s = fx_clz(fx_hi(V));
  const uint64_t N = ((uint64_t)fx_funnel(fx_lo(V), fx_hi(V), s) << 32) | (uint64_t)(fx_lo(V) << s);
  return fx_assemble(N, e - s);
}

// ---- product -------------------------------------------------------------------------------
// a b rounded to nearest even, the bits of the FP64 multiplication, on the integer pipe (about
// 35 instructions, 16 cycles per warp and SM against 20 of a DMUL): for kernels that the FP64
// pipe binds while the integer one idles, as a second multiplier beside it.  Operands and
// products outside the normal range take the FP64 one.
#if defined(__CUDACC__)
static __device__ __noinline__ double fx_mul_rare(double a, double b) { return __dmul_rn(a, b); }
#else
static inline double fx_mul_rare(double a, double b) { return a * b; }
#endif
FX_DEV double fx_mul_rn(double a, double b) {
  const uint64_t ab = fx_bits(a), bb = fx_bits(b);
  const uint32_t ea = (fx_hi(ab) >> 20) & 0x7ffu, eb = (fx_hi(bb) >> 20) & 0x7ffu;
  const uint32_t e = ea + eb;
  // both normal and finite, and the product's exponent e - 1023 (+ 1) in [1, 2045]
  if (ea - 1u >= 0x7feu || eb - 1u >= 0x7feu || e - 1025u >= 2043u) {
    // a zero times a finite number is the common case here
    if (((ab << 1) == 0 && eb != 0x7ffu) || ((bb << 1) == 0 && ea != 0x7ffu)) return fx_double((ab ^ bb) & 0x8000000000000000ull);
    return fx_mul_rare(a, b);
  }
  const uint64_t x = fx_significand(ab) << 11, y = fx_significand(bb) << 11;
  const uint64_t t0 = (uint64_t)fx_lo(x) * fx_lo(y);
  const uint64_t t1 = (uint64_t)fx_hi(x) * fx_lo(y) + fx_hi(t0);
  const uint64_t t2 = (uint64_t)fx_lo(x) * fx_hi(y) + fx_lo(t1);
  uint64_t h = (uint64_t)fx_hi(x) * fx_hi(y) + fx_hi(t1) + fx_hi(t2);  // x y 2^-64
  h |= ((fx_lo(t2) | fx_lo(t0)) != 0u) ? 1u : 0u;                      // what is below it, as a sticky bit
  const int c = (int)(fx_hi(h) >> 31), sh = 10 + c;
  const uint64_t r = (h + (((uint64_t)512u << c) - 1u) + ((h >> sh) & 1u)) >> sh;
  const uint64_t q = r + ((uint64_t)(e - 1024u + (uint32_t)c) << 52);
  return fx_double(q | ((ab ^ bb) & 0x8000000000000000ull));
}

// ---- exp -----------------------------------------------------------------------------------
// x in fixed point with F fraction bits, rounded to nearest, for |x| < 2^(63 - F); bits b of x
template <int F>
FX_FN int64_t fx_fixed(uint64_t b) {
  const int E = (int)(fx_hi(b) >> 20) & 0x7ff;
  const int sh = 1085 - F - E > 63 ? 63 : 1085 - F - E;
  const uint64_t m = ((fx_significand(b) << 10) + ((1ull << sh) >> 1)) >> sh;
  return (int64_t)b < 0 ? -(int64_t)m : (int64_t)m;
}

// exp(X) for |X| < 500, given floor(X) in Q9.22 and the fraction of X in Q0.64: the value is
// M 2^(m - 62), M in [2^62, 2^63 (1 + 2^-9))
FX_FN uint64_t fx_exp_parts(int32_t top, uint64_t fraction, int &m) {
  // X = (256 m + j) ln2/256 + r with 0 <= r < (1 + 2^-10) ln2/256: the quotient from the
  // high word, biased down by 2^-11 so that r is never negative
  const int k = (fx_mulhi(top, 774541002) - 1) >> 11;
  const uint64_t R = fraction - ((uint64_t)(int64_t)k * 0xb17217f7d1cf7aull +
                                            (uint64_t)(int64_t)fx_mulhi(k, -1412832332));  // Q0.64, modulo 1
  const uint64_t T = FX_TAB(exp2, k & 255);
  m = k >> 8;
  // exp(r) - 1 = r + r^2/2 + r^3 (1/6 + r/24 + r^2/120) + O(r^6/720), r < 2^-8.5
  const uint32_t rh = (uint32_t)(R >> 24), rl = (uint32_t)R << 8;  // r = rh 2^-40 + rl 2^-72
  const uint64_t sq = (uint64_t)rh * rh + ((uint64_t)fx_umulhi(rh, rl) << 1);  // r^2, Q.80
  const uint32_t q = fx_hi(sq);                                    // Q.48
  const uint32_t w = 2863311531u + fx_umulhi(rh, 2796203u) + fx_umulhi(q, 2185u);  // Q.34
  const uint64_t p = R + (sq >> 17) + (((uint64_t)fx_umulhi(q, rh) * w) >> 26);
  return T + fx_mul64hi(T, p);
}

// exp(X) for X in Q9.54
FX_FN uint64_t fx_exp_core(int64_t X, int &m) { return fx_exp_parts((int32_t)(X >> 32), (uint64_t)X << 10, m); }

// M 2^(m - 62) of fx_exp_core as a double
FX_FN double fx_exp_double(uint64_t M, int m) {
  const int c = (int)(fx_hi(M) >> 31);  // 1 where M >= 2^63
  const uint64_t r = (M + ((uint64_t)0x200u << c)) >> (10 + c);
  return fx_double(r + ((uint64_t)(uint32_t)(m + 1022 + c) << 52));
}

// |x| < 500; CUDA's exp elsewhere
FX_FN double fx_exp(double x) {
  const uint64_t b = fx_bits(x);
  if ((fx_hi(b) & 0x7fffffffu) >= 0x407f4000u) return FX_RARE(exp, exp(x), x);
  int m;
  const uint64_t M = fx_exp_core(fx_fixed<54>(b), m);
  return fx_exp_double(M, m);
}

// ---- log -----------------------------------------------------------------------------------
// log1p(z) - z for Z = z in Q0.64 (signed), |z| < 2^-8.97
FX_FN int64_t fx_log1p_tail(int64_t Z) {
  const int32_t zh = (int32_t)(Z >> 25);                 // Q.39, |.| < 2^30.1
  const uint32_t zl = (uint32_t)Z << 7;                  // z = zh 2^-39 + zl 2^-71
  const int64_t sq = (int64_t)zh * zh;                   // Q.78
  const int32_t q = (int32_t)(sq >> 30);                 // Q.48
  const int32_t c = (int32_t)(((int64_t)q * zh) >> 30);  // z^3, Q.57
  // 1/3 - z/4 + z^2/5 - z^3/6 in Q.32, Horner in v = 2^8 z = zh 2^-31 (each level's
  // coefficient doubled, as the high word of the product halves it)
  int32_t w = 52429 + fx_mulhi(zh, -341);
  w = -8388608 + fx_mulhi(zh, w);
  w = 1431655765 + fx_mulhi(zh, w);
  // z^2/2 with the product of the two parts of z, zh zl 2^-46 in Q.64 (31 bits of zl, so
  // that the product is a signed one)
  const int64_t cross = ((int64_t)zh * (int32_t)(zl >> 1)) >> 45;
  return (((int64_t)c * w) >> 25) - (sq >> 15) - cross;
}

// log of the significand m53 (53 bits with its hidden bit, value m53 2^-52 in [1, 2)), Q0.64
// as an unsigned number in [0, ln2)
FX_FN uint64_t fx_log_significand(uint64_t m53) {
  const int j = (int)(m53 >> 44) & 255;
  const uint64_t mx = m53 << 11;  // Q1.63
  const uint32_t c = FX_TAB(c, j);
  // z = mx c - 1 in Q0.64 (the product is Q.79; the leading 1 leaves by the modulus)
  const uint64_t Z = (((uint64_t)fx_hi(mx) * c) << 17) + (((uint64_t)fx_lo(mx) * c) >> 15);
  return FX_TAB(logc, j) + Z + (uint64_t)fx_log1p_tail((int64_t)Z);
}

// |m ln2 + F 2^-64| as V 2^e with V's top bit set, and its sign; false where the magnitude is
// below least 2^-32
FX_FN bool fx_log_parts(int m, uint64_t F, uint32_t least, uint64_t &V, int &exponent, bool &neg) {
  // m ln2 + F = m - m (1 - ln2) + F; 1 - ln2 = 0x4e8de808 2e308654 2^-64
  const int64_t p0 = (int64_t)m * 0x2e308654;
  const int64_t p1 = (int64_t)m * 0x4e8de808 + (p0 >> 32);
  const uint64_t sub = ((uint64_t)p1 << 32) | (uint64_t)fx_lo((uint64_t)p0);
  uint64_t f = F - sub;
  int32_t H = m - (int32_t)(p1 >> 32) - (F < sub ? 1 : 0);
  neg = H < 0;
  if (neg) { f = ~f; H = ~H; }  // one unit of 2^-64 off the negation
  uint32_t w2 = (uint32_t)H, w1 = fx_hi(f), w0 = fx_lo(f);
  int e = -32;  // w2:w1 is the value in units of 2^-32
  if (w2 == 0) {
    if (w1 < least) return false;  // the leading bits have cancelled
    w2 = w1; w1 = w0; w0 = 0; e -= 32;
  }
  const int s = fx_clz(w2);
  V = ((uint64_t)fx_funnel(w1, w2, s) << 32) | fx_funnel(w0, w1, s);
  exponent = e - s;
  return true;
}

// m ln2 + F 2^-64 as a double; false as above
FX_FN bool fx_log_of(int m, uint64_t F, uint32_t least, double &out) {
  uint64_t V;
  int e;
  bool neg;
  if (!fx_log_parts(m, F, least, V, e, neg)) return false;
  const double r = fx_assemble(V, e);
  out = neg ? -r : r;
  return true;
}

// positive normal x with |log x| >= 2^-3; CUDA's log elsewhere
FX_FN double fx_log(double x) {
  const uint64_t b = fx_bits(x);
  const uint32_t hi = fx_hi(b);
  if (hi < 0x00100000u || hi >= 0x7ff00000u) return FX_RARE(log, log(x), x);
  double r;
  if (!fx_log_of((int)(hi >> 20) - 1023, fx_log_significand(fx_significand(b)), 0x20000000u, r)) return FX_RARE(log, log(x), x);
  return r;
}

// k ln 2 rounded to nearest, for 0 < |k| <= 1100 (checked for every such k: the bits of
// fma(k, ln2_hi, k ln2_lo)), and 0
FX_FN double fx_k_ln2(int k) {
  double r = 0.0;
  if (k != 0) fx_log_of(k, 0, 0, r);
  return r;
}

// ---- power ---------------------------------------------------------------------------------
// x^y for positive normal x with |log x| >= 2^-3, 2^-60 <= |y| < 1 and |y log x| < 64, as
// exp(y log x) with 64 bits of the logarithm and of the product kept (0.8 ulp); CUDA's pow
// elsewhere.
FX_FN double fx_pow(double x, double y) {
  const uint64_t xb = fx_bits(x), yb = fx_bits(y);
  const uint32_t hi = fx_hi(xb);
  const int ey = (int)((fx_hi(yb) >> 20) & 0x7ffu) - 1023;
  uint64_t V;
  int e;
  bool neg;
  if (hi < 0x00100000u || hi >= 0x7ff00000u || ey < -60 || ey > -1 ||
      !fx_log_parts((int)(hi >> 20) - 1023, fx_log_significand(fx_significand(xb)), 0x20000000u, V, e, neg))
    return FX_RARE2(pow, pow(x, y), x, y);
  // |y log x| = P 2^(sh - 64) (sh: -61 to 10), as a whole part and a fraction in Q0.64
  const uint64_t P = fx_mul64hi(V, fx_significand(yb) << 11);
  const int sh = e + ey + 65;
  const uint64_t whole = sh > 0 ? P >> (64 - sh) : 0;
  if (whole >= 64u) return FX_RARE2(pow, pow(x, y), x, y);
  uint64_t fraction = sh > 0 ? P << sh : P >> -sh;
  int32_t top = (int32_t)(((uint32_t)whole << 22) | (uint32_t)(fraction >> 42));
  if (neg != ((int64_t)yb < 0)) {
    top = ~top + ((fraction << 22) == 0 ? 1 : 0);  // floor of the negation
    fraction = 0 - fraction;
  }
  int m;
  const uint64_t M = fx_exp_parts(top, fraction, m);
  return fx_exp_double(M, m);
}

// ---- reciprocal ----------------------------------------------------------------------------
FX_FN float fx_rcp_estimate(float d) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return y;
#else
  return 1.0f / d;
#endif
}
FX_FN float fx_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}
FX_FN uint32_t fx_float_bits(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  uint32_t b;
  memcpy(&b, &f, 4);
  return b;
#endif
}

// 2^127 / D in (2^63, 2^64), for D in [2^63, 2^64): the estimate y of 1/d, d = D 2^-63, and
// y (1 + e + e^2) with e = 1 - d y (|e| < 2^-22, so the error e^3 is below 2^-66).  At most
// 2^64 - 1 (d = 1).
FX_FN uint64_t fx_recip_core(uint64_t D) {
  const float y0 = fx_rcp_estimate(fx_float(0x3f800000u | (uint32_t)((D >> 40) & 0x7fffff)));
  // y in Q.32: (0.5, 1], the significand of y0 left-aligned, 2^32 - 256 for y0 = 1 and above
  const uint32_t yb = fx_float_bits(y0);
  const uint32_t y = yb >= 0x3f800000u ? 0xffffff00u : (0x80000000u | (yb << 8));
  // d y in Q1.63 close to 2^63: e as a signed Q.63 number
  const uint64_t dy = (uint64_t)fx_hi(D) * y + fx_umulhi(fx_lo(D), y);
  const int64_t e = (int64_t)(0x8000000000000000ull - dy);
  const int32_t e32 = (int32_t)(e >> 16);               // Q.47, |.| < 2^26
  const int64_t t = e + (((int64_t)e32 * e32) >> 31);    // e + e^2, Q.63
  // y t in Q.64: y (Q.32) times the two words of t (Q.63)
  const int64_t corr = 2 * ((int64_t)(int32_t)(t >> 32) * (int64_t)y) + (int64_t)(((uint64_t)fx_lo((uint64_t)t) * y) >> 31);
  return ((uint64_t)y << 32) + (uint64_t)corr;
}

// 1 / x for 2^-1000 <= |x| <= 2^1000; IEEE division elsewhere
FX_FN double fx_recip(double x) {
  const uint64_t b = fx_bits(x);
  const uint32_t E = (fx_hi(b) >> 20) & 0x7ffu;
  if (E - 23u > 2000u) return FX_RARE(recip, 1.0 / x, x);
  const uint64_t Y = fx_recip_core(fx_significand(b) << 11);
  const double r = fx_assemble(Y, -(int)E + 1023 - 64);
  return fx_double(fx_bits(r) | (b & 0x8000000000000000ull));
}

// ---- square root ---------------------------------------------------------------------------
FX_FN float fx_rsqrt_estimate(float d) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return y;
#else
  return 1.0f / sqrtf(d);
#endif
}

// sqrt(x) for 2^-1000 <= x <= 2^1000; CUDA's sqrt elsewhere.  With d = the significand
// scaled by the parity of the exponent into [1, 4) and y the estimate of 1/sqrt(d):
// sqrt(d) = d y / sqrt(1 - e), e = 1 - d y^2, |e| < 2^-21, = d y (1 + e/2 + 3/8 e^2 + O(e^3)).
FX_FN double fx_sqrt(double x) {
  const uint64_t b = fx_bits(x);
  const uint32_t E = fx_hi(b) >> 20;
  if (E - 23u > 2000u) return FX_RARE(sqrt, sqrt(x), x);
  const int odd = (int)((E & 1u) ^ 1u);  // unbiased exponent E - 1023 is odd where E is even
  const uint64_t D = fx_significand(b) << (9 + odd);  // Q2.62... d = D 2^-61 in [1, 4)
  const float df = fx_float(((127u + (uint32_t)odd) << 23) | (uint32_t)((b >> 29) & 0x7fffff));
  const uint32_t yb = fx_float_bits(fx_rsqrt_estimate(df));  // in [0.5, 1]
  const uint32_t y = yb >= 0x3f800000u ? 0xffffff00u : (((yb & 0x7fffffu) | 0x800000u) << 8) >> (126 - (yb >> 23));  // Q.32
  // s = d y in Q2.61, below 2: 62 bits
  const uint64_t s = (uint64_t)fx_hi(D) * y + fx_umulhi(fx_lo(D), y);
  // s y = d y^2 in Q.61, close to 1
  const uint64_t sy = (uint64_t)fx_hi(s) * y + fx_umulhi(fx_lo(s), y);
  const int64_t e = (int64_t)(0x2000000000000000ull - sy);  // Q.61, |e| < 2^41
  const int32_t e32 = (int32_t)(e >> 14);                    // Q.47
  const int64_t e2 = ((int64_t)e32 * e32) >> 33;             // Q.61
  const int64_t t = (e >> 1) + ((3 * e2) >> 3);              // Q.61
  // s t in Q.61: s in [2^61, 2^62) (31 bits of it are enough), |t| < 2^41 in Q.61
  const int32_t sh = (int32_t)(s >> 32);                     // Q.29, < 2^30
  const int64_t corr = 8 * ((int64_t)(int32_t)(t >> 32) * sh) + (int64_t)(((uint64_t)fx_lo((uint64_t)t) * (uint32_t)sh) >> 29) +
                       (((int64_t)(int32_t)(t >> 11) * (int32_t)(fx_lo(s) >> 1)) >> 49);
  const uint64_t S = s + (uint64_t)corr;
  return fx_normalise(S, -61 + (((int)E - 1023 - odd) >> 1));
}

// ---- sine and cosine -----------------------------------------------------------------------
// (sin x, cos x) for 2^-4 <= |x| < 1.5, and x = 0; CUDA's sincos elsewhere
FX_FN void fx_sincos(double x, double *sn, double *cs) {
  const uint64_t b = fx_bits(x);
  const uint32_t ahi = fx_hi(b) & 0x7fffffffu;
  if (ahi - 0x3fb00000u >= 0x00480000u) {
    if ((ahi | fx_lo(b)) == 0u) { *sn = x; *cs = 1.0; return; }
#if defined(__CUDA_ARCH__)
    const double2 r = fx_sincos_rare(x);
    *sn = r.x; *cs = r.y;
#else
    *sn = sin(x); *cs = cos(x);
#endif
    return;
  }
  // |x| in Q1.63 (exact): x = j/256 + r, 0 <= r < 2^-8
  const uint64_t X = (fx_significand(b) << 11) >> (1023 - (int)(ahi >> 20));
  const int j = (int)(X >> 55);
  const uint64_t r = X & 0x7fffffffffffffull;             // Q.63
  const uint32_t rh = (uint32_t)(r >> 23), rl = (uint32_t)r << 9;  // r = rh 2^-40 + rl 2^-72
  const uint64_t sq = (uint64_t)rh * rh + ((uint64_t)fx_umulhi(rh, rl) << 1);  // r^2, Q.80
  const uint32_t q = fx_hi(sq);                           // Q.48
  // sin r = r - r^3 (1/6 - r^2/120), 1 - cos r = r^2/2 - r^4 (1/24 - r^2/720), in Q.63
  const uint32_t w3 = 2863311531u - fx_umulhi(q, 2185u);  // Q.34
  const uint32_t w4 = 178956971u - fx_umulhi(q, 91u);     // Q.32
  const uint64_t cu = (uint64_t)q * rh + fx_umulhi(q, rl);  // r^3, Q.88
  const uint64_t sr = r - (((uint64_t)fx_hi(cu) * w3 + fx_umulhi(fx_lo(cu), w3)) >> 27);
  const uint64_t vr = (sq >> 18) - (((uint64_t)fx_umulhi(q, q) * w4) >> 33);
#if defined(__CUDA_ARCH__)
  const ulonglong2 t = __ldg(&g_fx_sincos[j]);
#else
  const FxPair t = h_fx_sincos[j];
#endif
  // sin(a + r) = S - S (1 - cos r) + C sin r, cos(a + r) = C - C (1 - cos r) - S sin r
  const uint64_t S = t.x + fx_mul64hi(t.y, sr << 1) - fx_mul64hi(t.x, vr << 1);
  const uint64_t C = t.y - fx_mul64hi(t.x, sr << 1) - fx_mul64hi(t.y, vr << 1);
  *sn = fx_double(fx_bits(fx_normalise(S, -63)) | (b & 0x8000000000000000ull));
  *cs = fx_normalise(C, -63);
}

}  // namespace mdz
