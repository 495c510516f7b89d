// ve_fx.cuh -- the visco-elastic local solve in 64-bit fixed point.
//
// The root s of  r(s) = 1 - a s - sum_k exp(n_k ln s + c_k)  (the local residual over Eii in
// the unknown s = eta / eta_n, rheo_device.cuh) from an FP32 point s0 within about 1e-6 of
// it: one evaluation of r at s0, a Halley step q, the residual of s0 (1 + q) from the law
// terms carried by exp(n_k log1p(q)), and a last Newton step from it.  Every quantity is
// O(1), so it is a Q2.62 number, and its products run on the integer pipe; the quotients of
// the two steps are FP32, whose rounding the next residual sees.  The carried residual is
// good to 2^-58 and its root to about as much, below the rounding of the double that eta is
// returned in; the reference stops at |r| < 1e-13.
//
// Before, the same start was moved by a Halley step in double-float (FP32 pairs) and then
// confirmed by one FP64 evaluation of r, a logarithm, an exponential per law and the
// residual: about 36 FP64 instructions, 20 cycles each, and as many FP32 ones as this takes
// integer ones.  The 2049 x 2049 sweep went from 15.58 to 9.97 ms and the anisotropic
// 1025 x 1025 one from 2.58 to 1.63 ms; no local solve of either declines.
//
// The fast form declines (returns false, nothing written) where a number would leave its
// format: a point that the FP32 steps did not settle, terms well above 1, s0 outside [2^-4, 2),
// exponents n_k of 128 and more, |c_k| of 150 and more.  The caller then takes the FP64 iteration.
#pragma once
#include "fx64.cuh"

namespace mdz {

// (E F) / 2^62 for E in [0, 2^63), F signed below 2^50 in magnitude; up to 8 units off
FX_FN int64_t fx_mulq62(uint64_t E, int64_t F) {
  const int32_t eh = (int32_t)fx_hi(E), fh = (int32_t)(F >> 32);
  const uint32_t fl = fx_lo((uint64_t)F);
  return 4 * ((int64_t)eh * fh) + (int64_t)(((uint64_t)(uint32_t)eh * fl) >> 30) +
         (((int64_t)(int32_t)(fx_lo(E) >> 1) * fh) >> 29);
}

FX_FN float fx_float_of(int64_t R) {
  return fmaf((float)(int32_t)(R >> 32), 4294967296.0f, (float)fx_lo((uint64_t)R));
}

// n L in Q9.54 for n = N in Q7.56 and L in Q4.60 (signed), |n L| < 512
FX_FN int64_t fx_mul_nl(int64_t N, int64_t L) {
  const int32_t nh = (int32_t)(N >> 32), lh = (int32_t)(L >> 32);
  const uint32_t nl = fx_lo((uint64_t)N), ll = fx_lo((uint64_t)L);
  // the middle products with 4 more bits, so that their sum is rounded once
  const int64_t mid = (int64_t)((uint64_t)(uint32_t)nh * ll >> 26) + (((int64_t)lh * (int32_t)(nl >> 1)) >> 25) +
                      (int64_t)(fx_umulhi(nl, ll) >> 26);
  return 4 * ((int64_t)nh * lh) + ((mid + 8) >> 4);
}

// n d in Q9.54 for n = N in Q7.56 and d = L in Q9.54 (signed), |n d| < 512
FX_FN int64_t fx_mul_nd(int64_t N, int64_t L) {
  const int32_t nh = (int32_t)(N >> 32), lh = (int32_t)(L >> 32);
  const uint32_t nl = fx_lo((uint64_t)N), ll = fx_lo((uint64_t)L);
  const int64_t mid = (int64_t)((uint64_t)(uint32_t)nh * ll >> 20) + (((int64_t)lh * (int32_t)(nl >> 1)) >> 19) +
                      (int64_t)(fx_umulhi(nl, ll) >> 20);
  return (int64_t)((uint64_t)((int64_t)nh * lh) << 8) + ((mid + 8) >> 4);
}

// n L in Q.62 for n = N in Q7.56 and L in Q.62 with |L| < 2^50 (signed)
FX_FN int64_t fx_mul_ntiny(int64_t N, int64_t L) {
  const int32_t nh = (int32_t)(N >> 32), lh = (int32_t)(L >> 32);
  const uint32_t nl = fx_lo((uint64_t)N), ll = fx_lo((uint64_t)L);
  return 256 * ((int64_t)nh * lh) + (int64_t)(((uint64_t)(uint32_t)nh * ll) >> 24) +
         (((int64_t)lh * (int32_t)(nl >> 1)) >> 23) + (int64_t)(fx_umulhi(nl, ll) >> 24);
}

FX_FN int32_t fx_rint(float x) {
#if defined(__CUDA_ARCH__)
  return __float2int_rn(x);
#else
  return !(x > -2147483648.0f) ? INT32_MIN : (x < 2147483648.0f ? (int32_t)lrintf(x) : INT32_MAX);
#endif
}

// a shift count held to [0, 63]; one below 0 is of a number that has left its format, which
// the caller's checks see
FX_FN int fx_shift(int sh) { return (unsigned)sh > 63u ? 63 : sh; }
// R - E modulo 2^64: sums of Q2.62 numbers that have left their format wrap
FX_FN int64_t fx_sub(int64_t R, uint64_t E) { return (int64_t)((uint64_t)R - E); }

// Bounds on the residual's terms: a s below 1.05 (in Q2.30), each law's argument below 0.05
// (in Q9.22), so each law's term below 1.052.  At the root every term is at most 1.  Within the
// bounds r is above -3.21, so where the sum wraps, modulo 4, it lands above 0.79: never near 0.
constexpr uint32_t kVeMaxLinear = 1127428915u;
constexpr int32_t kVeMaxArgument = 209715;

struct VeFxRoot {
  uint64_t S;          // s, Q2.62
  uint64_t M[3];       // law terms exp(n_k ln s + c_k) = M 2^(m - 62)
  int m[3];
};

// nl: bit k set: law k is non-linear and active.  a: the linear coefficient; N, C: exponent
// (Q7.56) and argument at s = 1 (Q9.54, below 150 in magnitude) of each law, nf the exponents
// in FP32; s0 the FP32 point.
FX_FN bool ve_root_fx(int nl, double a, const int64_t *N, const int64_t *C, const float *nf, float s0, VeFxRoot &o) {
  const uint32_t sb = fx_float_bits(s0);
  const int e0 = (int)(sb >> 23) - 127;  // s0 > 0
  if (e0 > 0 || e0 < -4) return false;
  const uint32_t m24 = (sb & 0x7fffffu) | 0x800000u;
  bool ok = true;
  // a s0: the significand of a times that of s0, shifted to Q2.62
  const uint64_t ab = fx_bits(a);
  const int ea = (int)(fx_hi(ab) >> 20) - 1023;  // a >= 0
  const int shift = -(ea + e0);
  if (shift < 0) return false;  // a s0 >= 2, Inf or NaN
  const uint64_t am = fx_significand(ab) << 11;
  const uint64_t A0 = ((uint64_t)fx_hi(am) * (m24 << 8) + fx_umulhi(fx_lo(am), m24 << 8)) >> (shift > 63 ? 63 : shift);
  ok = ok && fx_hi(A0) < kVeMaxLinear;
  int64_t R = fx_sub(0x4000000000000000ll, A0);
  float D = (float)fx_hi(A0) * 9.31322575e-10f, Q = 0.0f;  // 2^-30
  if (nl) {
    // ln s0 in Q4.60
    const int64_t L = (int64_t)(fx_log_significand((uint64_t)m24 << 29) >> 4) + (int64_t)e0 * 0xb17217f7d1cf79all;
#pragma unroll
    for (int k = 0; k < 3; k++)
      if (nl >> k & 1) {
        const int64_t X = fx_mul_nl(N[k], L) + C[k];
        ok = ok && (int32_t)(X >> 32) < kVeMaxArgument;  // (and above -505)
        o.M[k] = fx_exp_core(X, o.m[k]);
        const int sh = -o.m[k];
        const uint64_t E = o.M[k] >> fx_shift(sh);
        R = fx_sub(R, E);
        const float ne = nf[k] * ((float)fx_hi(E) * 9.31322575e-10f);
        D += ne;
        Q = fmaf(ne, nf[k] - 1.0f, Q);
      }
  }
  // Halley: q - q^2 Q / (2 D) with q = r / D
  const float iD = fx_rcp_estimate(D);
  float q = (fx_float_of(R) * 2.16840434e-19f) * iD;  // 2^-62
  q = fmaf(-0.5f * q * q, Q * iD, q);
  ok = ok && fabsf(q) < 6.0e-5f;
  const int32_t qi = fx_rint(q * 17592186044416.0f);  // Q.44, below 2^30; exact from here on
  const int64_t sq = (int64_t)qi * qi;                        // Q.88
  const int64_t q62 = (int64_t)qi * 262144;
  // log1p(q) = q - q^2/2 + q^3/3
  const int64_t lam = q62 - (sq >> 27) + ((((sq >> 44) * (int64_t)qi) >> 26) * 21845 >> 16);
  const uint64_t S0 = (uint64_t)m24 << (39 + e0);
  const uint64_t S1 = S0 + (uint64_t)fx_mulq62(S0, q62);
  R = fx_sub(fx_sub(0x4000000000000000ll, A0), (uint64_t)fx_mulq62(A0, q62));
  if (nl) {
#pragma unroll
    for (int k = 0; k < 3; k++)
      if (nl >> k & 1) {
        // exp(n log1p(q)) - 1 = t + t^2/2 + t^3/6, |t| < 2^-14
        const int64_t t = fx_mul_ntiny(N[k], lam);
        const int32_t ts = (int32_t)(t >> 17);  // Q.45
        ok = ok && (int32_t)(t >> 48) >= -1 && (int32_t)(t >> 48) < 1;
        const int64_t t2 = (int64_t)ts * ts;    // Q.90
        const int64_t f = t + (t2 >> 29) + ((((t2 >> 45) * (int64_t)ts) >> 28) * 10923 >> 16);
        o.M[k] += (uint64_t)fx_mulq62(o.M[k] >> 1, 2 * f);
        const int sh = -o.m[k];
        R = fx_sub(R, o.M[k] >> fx_shift(sh));
      }
  }
  ok = ok && R < (1ll << 27) && R > -(1ll << 27);
  // the last step, in units of 2^-62, with D at the new point: D + q (D + Q)
  const float q2 = (float)(int32_t)R * fmaf(-q * iD, fmaf(Q, iD, 1.0f), iD);
  o.S = S1 + (uint64_t)(((int64_t)(int32_t)fx_hi(S1) * fx_rint(q2)) >> 30);
#pragma unroll
  for (int k = 0; k < 3; k++)
    if (nl >> k & 1) o.M[k] += (uint64_t)(((int64_t)(int32_t)(fx_hi(o.M[k]) >> 1) * fx_rint(nf[k] * q2 * 0.015625f)) >> 23);
  return ok;
}

// The residual r(sv) in Q2.62, for a double sv in [2^-4, 2); nl, a, N, C as above.  false
// where a number leaves its format.
FX_FN bool ve_residual_fx(int nl, double a, const int64_t *N, const int64_t *C, double sv, int64_t &R) {
  const uint64_t sb = fx_bits(sv), ab = fx_bits(a);
  const int e0 = (int)(fx_hi(sb) >> 20) - 1023, ea = (int)(fx_hi(ab) >> 20) - 1023;  // sv > 0, a >= 0
  const int shift = -(ea + e0);
  if (e0 > 0 || e0 < -4 || shift < 0) return false;
  const uint64_t m53 = fx_significand(sb);
  const uint64_t A0 = fx_mul64hi(fx_significand(ab) << 11, m53 << 11) >> (shift > 63 ? 63 : shift);
  bool ok = fx_hi(A0) < kVeMaxLinear;
  R = fx_sub(0x4000000000000000ll, A0);
  if (nl) {
    const int64_t L = (int64_t)(fx_log_significand(m53) >> 4) + (int64_t)e0 * 0xb17217f7d1cf79all;
#pragma unroll
    for (int k = 0; k < 3; k++)
      if (nl >> k & 1) {
        const int64_t X = fx_mul_nl(N[k], L) + C[k];
        ok = ok && (int32_t)(X >> 32) < kVeMaxArgument;
        int m;
        const uint64_t M = fx_exp_core(X, m);
        R = fx_sub(R, M >> fx_shift(-m));
      }
  }
  return ok;
}

}  // namespace mdz
