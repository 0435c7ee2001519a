// exact64.cuh -- correctly rounded FP64 division and square root without FP64 instructions, for the
// separately rounded (reference-exact) kernels.
//
// The quotient (root) of the 53-bit significands is estimated in a pair of FP32 values, about 46 bits,
// and becomes an integer; its exact remainder, which fits 64 bits, corrects it and then decides the
// rounding.  No estimate enters the result: the last comparison is exact, and a quotient or root of
// 53-bit numbers is never a tie.  About 70 integer and FP32 instructions against eight to ten FP64
// instructions, each of which keeps a sub-partition's FP64 path busy for 65 cycles.  With halvings,
// comparisons and HLLD's masks off the FP64 pipe too, the three flux kernels of a 64x96x48 stage step
// went from 1.47 to 0.71 ms and a fused step of 100x62x90 from 4.75 to 2.99 ms, bit for bit the same (0.78
// and 3.40 with a branch in every division; 2.2 ms on the form's 256-thread kernel).
#pragma once

#include "fp32pair.cuh"

namespace mhdgb {

// A pair near 1..2 as an integer in units of 2^-52.
MHDGB_HD long long pair_to_units(float h, float l) {
  const unsigned u = f_bits(h);
  const unsigned long long m = (u & 0x007FFFFFu) | 0x00800000u;
  return (long long)(m << ((u >> 23) - 98u)) + 2 * (long long)f_to_i(f_mul(l, 0x1p51f));
}
// The significand of a normal double as a float pair in [1, 2) (truncated to 24 bits, then the rest).
MHDGB_HD Pair significand_pair(unsigned hi, unsigned lo) {
  return Pair{f_from((f_shl(hi, lo, 3) & 0x007FFFFFu) | 0x3F800000u), f_mul(i_to_f((int)(lo & 0x1FFFFFFFu)), 0x1p-52f)};
}

// a / b, rounded to nearest even, without a branch; ok becomes false for subnormal, infinite and NaN
// operands, zero divisors and results near the ends of the exponent range (the result is then
// meaningless).  Several of these overlap where a branch in each would run them one after the other.
MHDGB_HD double div_core(double a, double b, bool& ok) {
  const unsigned ha = d_hi(a), la = d_lo(a), hb = d_hi(b), lb = d_lo(b);
  const int ea = (int)((ha >> 20) & 0x7FFu), eb = (int)((hb >> 20) & 0x7FFu), er = ea - eb + 1023;
  const bool zero = ((ha << 1) | la) == 0u;
  ok = ok && (unsigned)(eb - 1) < 2046u && (zero || ((unsigned)(ea - 1) < 2046u && (unsigned)(er - 2) < 2044u));
  const unsigned long long B = ((unsigned long long)((hb & 0xFFFFFu) | 0x100000u) << 32) | lb;
  const unsigned ma = ha & 0xFFFFFu, mb = hb & 0xFFFFFu;
  const bool s = ma < mb || (ma == mb && la < lb);  // significand quotient below 1: scale a by 2
  const float two = s ? 2.0f : 1.0f;
  const Pair x0 = significand_pair(ha, la), y = significand_pair(hb, lb);
  const float xh = f_mul(x0.h, two), xl = f_mul(x0.l, two);
  const float r0 = f_rcp_seed(y.h), r = f_fma(r0, f_fma(-y.h, r0, 1.0f), r0);
  const float q = f_mul(xh, r);
  const float ql = f_mul(r, f_fma(-q, y.l, f_add(f_fma(-q, y.h, xh), xl)));
  long long Q = pair_to_units(q, ql);
  long long R = (long long)(((unsigned long long)la << (s ? 53 : 52)) - B * (unsigned long long)Q);  // A 2^(52+s) - B Q
  const int n = f_to_i(f_mul(i_to_f((int)(R >> 32)), f_mul(r, 0x1p-20f)));
  Q += n;
  R -= (long long)n * (long long)B;
  Q += (2 * R > (long long)B ? 1 : 0) - (2 * R < -(long long)B ? 1 : 0);
  const unsigned long long bits =
      (unsigned long long)Q + ((unsigned long long)(unsigned)(er - 1 - (s ? 1 : 0)) << 52);
  const unsigned sign = (ha ^ hb) & 0x80000000u;
  return d_from(zero ? sign : (unsigned)(bits >> 32) | sign, zero ? 0u : (unsigned)bits);
}

// sqrt(x), rounded to nearest even, as div_core; zero, subnormal, negative, infinite and NaN arguments are
// left to the caller.
MHDGB_HD double sqrt_core(double x, bool& ok) {
  const unsigned hx = d_hi(x), lx = d_lo(x);
  ok = ok && hx - 0x00100000u < 0x7FE00000u;
  const int e = (int)(hx >> 20) - 1023, p = e & 1;
  const Pair m = significand_pair(hx, lx);
  const float two = p ? 2.0f : 1.0f;
  float y;
  const Pair g = p_sqrt(Pair{f_mul(m.h, two), f_mul(m.l, two)}, &y);
  long long Q = pair_to_units(g.h, g.l);
  long long R = (long long)(((unsigned long long)lx << (52 + p)) - (unsigned long long)Q * (unsigned long long)Q);
  const int n = f_to_i(f_mul(i_to_f((int)(R >> 32)), f_mul(y, 0x1p-21f)));
  R -= (long long)n * (2 * Q + n);
  Q += n;
  Q += (R > Q ? 1 : 0) - (R <= -Q ? 1 : 0);
  const unsigned long long bits = (unsigned long long)Q + ((unsigned long long)(unsigned)((e - p) / 2 + 1022) << 52);
  return d_from((unsigned)(bits >> 32), (unsigned)bits);
}

// The instruction sequences, out of line, for what the cores leave.
inline __host__ __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }
inline __host__ __device__ __noinline__ double sqrt_ieee(double x) { return sqrt(x); }

MHDGB_HD double div_rn(double a, double b) {
  bool ok = true;
  const double q = div_core(a, b, ok);
  return ok ? q : div_ieee(a, b);
}
MHDGB_HD double sqrt_rn(double x) {
  bool ok = true;
  const double q = sqrt_core(x, ok);
  return ok ? q : sqrt_ieee(x);
}
// N divisions with one test for all.
template <int N>
MHDGB_HD void div_many(const double (&a)[N], const double (&b)[N], double (&q)[N]) {
  unsigned left = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    bool ok = true;
    q[i] = div_core(a[i], b[i], ok);
    left |= ok ? 0u : 1u << i;
  }
  if (left) {
#pragma unroll
    for (int i = 0; i < N; i++)
      if ((left >> i) & 1u) q[i] = div_ieee(a[i], b[i]);
  }
}

}  // namespace mhdgb
