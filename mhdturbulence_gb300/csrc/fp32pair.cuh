// fp32pair.cuh -- arithmetic on unevaluated sums of two FP32 values (48 significant bits), for the
// parts of the FP64 form that need fewer than 53 bits.
//
// GB300 issues one FP64 warp instruction per SM in about 19 cycles (measured, 16.5 per ns over 152
// SMs); in that time the four sub-partitions issue up to 76 FP32 or integer instructions, of which
// the FP64 form used a tenth.  A pair sum takes 8 FP32 instructions and a pair product 4, so moving
// an operation off the FP64 pipe pays five to ten times over.
//
// The algorithms are the published error-free transformations (Knuth's TwoSum, Dekker's Fast2Sum,
// the FMA product of Ogita, Rump and Oishi) and Newton corrections of the hardware's approximate
// reciprocal and reciprocal square root.  Every operation is rounded to nearest and explicit (no
// contraction), hence odd in its arguments: mirror-image inputs give mirror-image results.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#define MHDGB_HD __host__ __device__ __forceinline__

namespace mhdgb {

// ---- explicitly rounded FP32 operations (host versions for checks on the CPU) -----------------
#ifdef __CUDA_ARCH__
MHDGB_HD float f_add(float a, float b) { return __fadd_rn(a, b); }
MHDGB_HD float f_sub(float a, float b) { return __fsub_rn(a, b); }
MHDGB_HD float f_mul(float a, float b) { return __fmul_rn(a, b); }
MHDGB_HD float f_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
MHDGB_HD float f_rcp_seed(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
MHDGB_HD float f_rsqrt_seed(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
MHDGB_HD unsigned f_bits(float x) { return __float_as_uint(x); }
MHDGB_HD float f_from(unsigned u) { return __uint_as_float(u); }
MHDGB_HD unsigned d_hi(double d) { return (unsigned)__double2hiint(d); }
MHDGB_HD unsigned d_lo(double d) { return (unsigned)__double2loint(d); }
MHDGB_HD double d_from(unsigned hi, unsigned lo) { return __hiloint2double((int)hi, (int)lo); }
MHDGB_HD float i_to_f(int m) { return __int2float_rn(m); }
MHDGB_HD int f_to_i(float x) { return __float2int_rn(x); }
MHDGB_HD int i_clz(unsigned x) { return __clz((int)x); }
MHDGB_HD unsigned f_shl(unsigned hi, unsigned lo, unsigned n) { return __funnelshift_l(lo, hi, n); }
#else
MHDGB_HD float f_add(float a, float b) { return a + b; }
MHDGB_HD float f_sub(float a, float b) { return a - b; }
MHDGB_HD float f_mul(float a, float b) { return a * b; }
MHDGB_HD float f_fma(float a, float b, float c) { return fmaf(a, b, c); }
MHDGB_HD float f_rcp_seed(float x) { return 1.0f / x; }
MHDGB_HD float f_rsqrt_seed(float x) { return 1.0f / sqrtf(x); }
MHDGB_HD unsigned f_bits(float x) { unsigned u; memcpy(&u, &x, 4); return u; }
MHDGB_HD float f_from(unsigned u) { float x; memcpy(&x, &u, 4); return x; }
MHDGB_HD unsigned d_hi(double d) { unsigned long long u; memcpy(&u, &d, 8); return (unsigned)(u >> 32); }
MHDGB_HD unsigned d_lo(double d) { unsigned long long u; memcpy(&u, &d, 8); return (unsigned)u; }
MHDGB_HD double d_from(unsigned hi, unsigned lo) {
  const unsigned long long u = ((unsigned long long)hi << 32) | lo;
  double d;
  memcpy(&d, &u, 8);
  return d;
}
MHDGB_HD float i_to_f(int m) { return (float)m; }
MHDGB_HD int f_to_i(float x) { return (int)nearbyintf(x); }
MHDGB_HD int i_clz(unsigned x) { return __builtin_clz(x); }
MHDGB_HD unsigned f_shl(unsigned hi, unsigned lo, unsigned n) { return n ? (hi << n) | (lo >> (32 - n)) : hi; }
#endif

// h + l.  The operations leave their results unnormalised: l stays around 2^-23 of the largest term
// that went into h, but h is not the pair rounded to FP32.  h is then ready one instruction after its
// operands' h, and the low parts trail behind off the critical path (renormalising after every
// operation made each wait for the previous one's low part).  Dropped products of low parts are below
// 2^-46 of the terms.  p_norm() restores |l| <= ulp(h)/2 where terms cancelled and the result is
// divided by, squared or rooted.
struct Pair {
  float h, l;
};

MHDGB_HD Pair p_make(float h, float l = 0.0f) { return Pair{h, l}; }
MHDGB_HD Pair p_neg(Pair a) { return Pair{-a.h, -a.l}; }
MHDGB_HD Pair p_neg_if(Pair a, bool n) {
  const unsigned s = n ? 0x80000000u : 0u;
  return Pair{f_from(f_bits(a.h) ^ s), f_from(f_bits(a.l) ^ s)};
}
MHDGB_HD Pair p_sel(bool c, Pair a, Pair b) { return Pair{c ? a.h : b.h, c ? a.l : b.l}; }
MHDGB_HD Pair p_scale(Pair a, float s) { return Pair{f_mul(a.h, s), f_mul(a.l, s)}; }  // s a power of two
MHDGB_HD Pair p_norm(Pair a) {  // |h| >= |l|
  const float s = f_add(a.h, a.l);
  return Pair{s, f_sub(a.l, f_sub(s, a.h))};
}
// a + b
MHDGB_HD Pair p_add(Pair a, Pair b) {
  const float s = f_add(a.h, b.h), v = f_sub(s, a.h);
  const float e = f_add(f_sub(a.h, f_sub(s, v)), f_sub(b.h, v));
  return Pair{s, f_add(e, f_add(a.l, b.l))};
}
MHDGB_HD Pair p_sub(Pair a, Pair b) { return p_add(a, p_neg(b)); }
MHDGB_HD Pair p_mul(Pair a, Pair b) {
  const float p = f_mul(a.h, b.h);
  return Pair{p, f_fma(a.l, b.h, f_fma(a.h, b.l, f_fma(a.h, b.h, -p)))};
}
MHDGB_HD Pair p_sqr(Pair a) {
  const float p = f_mul(a.h, a.h);
  return Pair{p, f_fma(f_add(a.h, a.h), a.l, f_fma(a.h, a.h, -p))};
}
// a * b + c
MHDGB_HD Pair p_fma(Pair a, Pair b, Pair c) { return p_add(p_mul(a, b), c); }
// 1 / b from a seed y: an FP32 reciprocal of h first, then its error against the pair to second order.
MHDGB_HD Pair p_rcp_from(Pair b, float y) {
  const float r = f_fma(y, f_fma(-b.h, y, 1.0f), y);
  const float e = f_fma(-b.l, r, f_fma(-b.h, r, 1.0f));
  return Pair{r, f_mul(r, f_fma(e, e, e))};
}
MHDGB_HD Pair p_rcp(Pair b) { return p_rcp_from(b, f_rcp_seed(b.h)); }
// sqrt(a) for a >= 0: an FP32 root g and reciprocal root from the seed, then g + (a - g^2) / (2 g)
// (error about 2^-47); *y_out receives the reciprocal root.
MHDGB_HD Pair p_sqrt(Pair a, float* y_out = nullptr) {
  const float y0 = f_rsqrt_seed(a.h), g0 = f_mul(a.h, y0);
  const float g = f_fma(f_mul(0.5f, y0), f_fma(-g0, g0, a.h), g0);
  const float y = f_fma(y0, f_fma(-g, y0, 1.0f), y0);
  const float d = f_add(f_fma(-g, g, a.h), a.l);
  if (y_out) *y_out = y;
  const bool z = !(a.h > 0.0f);
  return Pair{z ? 0.0f : g, z ? 0.0f : f_mul(f_mul(0.5f, y), d)};
}
MHDGB_HD bool p_less(Pair a, Pair b) { return f_add(f_sub(a.h, b.h), f_sub(a.l, b.l)) < 0.0f; }
MHDGB_HD Pair p_max(Pair a, Pair b) { return p_sel(p_less(a, b), b, a); }
MHDGB_HD Pair p_min(Pair a, Pair b) { return p_sel(p_less(b, a), b, a); }

MHDGB_HD unsigned u_max(unsigned a, unsigned b) { return a > b ? a : b; }
MHDGB_HD unsigned u_min(unsigned a, unsigned b) { return a < b ? a : b; }

// ---- conversions, on the integer pipe (the hardware's conversions issue on the FP64 pipe) -------

// The FP32 value nearest d (ties away from zero), |d| in [2^-126, 2^127): the exponent is rebiased by
// 896 = 3 * 256 + 128, which in the eight bits that the shift leaves of it is one bit flip.
MHDGB_HD float d_round_f(unsigned hi, unsigned lo) {
  const unsigned x = f_shl(hi, lo, 3) + ((lo >> 28) & 1u);
  return f_from(((x ^ 0x40000000u) & 0x7FFFFFFFu) | (hi & 0x80000000u));
}
// d as a pair (error below 2^-49 |d|) for |d| in [2^-102, 2^127).
MHDGB_HD Pair p_narrow_nz(double d) {
  const unsigned hi = d_hi(d), lo = d_lo(d);
  const float h = d_round_f(hi, lo);
  // the 29 bits below, as a signed remainder, in units of 2^(E - 52)
  return Pair{h, f_mul(f_mul(i_to_f((int)(lo << 3)), 0x1p-32f), f_from((f_shl(hi, lo, 3) & 0x7F800000u ^ 0x40000000u) +
                                                                      (hi & 0x80000000u) - (23u << 23)))};
}
// The same for |d| < 2^127: the low part ends at 2^-102, magnitudes below 2^-126 become 0.
MHDGB_HD Pair p_narrow(double d) {
  const unsigned hi = d_hi(d), lo = d_lo(d);
  const bool z = (hi << 1) < ((1023u - 126u) << 21);
  const unsigned e = u_max(f_shl(hi, lo, 3) & 0x7F800000u ^ 0x40000000u, 23u << 23) - (23u << 23);
  const float l = f_mul(f_mul(i_to_f((int)(lo << 3)), 0x1p-32f), f_from(e | (hi & 0x80000000u)));
  return Pair{z ? 0.0f : d_round_f(hi, lo), z ? 0.0f : l};
}
// x / 2 rounded to nearest even, for any x, on the integer pipe.  A front that decays into a uniform
// background cell by cell passes through the subnormal numbers, so no magnitude is left out.
MHDGB_HD double d_half(double x) {
  const unsigned hi = d_hi(x), lo = d_lo(x), e = hi & 0x7FF00000u;
  // exponent field 0 or 1: the magnitude is a whole number of the smallest subnormal
  const unsigned sl = (hi << 31) | (lo >> 1), l = sl + ((lo & 3u) == 3u ? 1u : 0u);
  const unsigned h = ((hi & 0x7FFFFFFFu) >> 1) + (l < sl ? 1u : 0u) + (hi & 0x80000000u);
  const bool tiny = e < (2u << 20), keep = e == 0x7FF00000u;  // infinities and NaN stay
  return d_from(tiny ? h : (keep ? hi : hi - (1u << 20)), tiny ? l : lo);
}
// h + l as a double (within an ulp), on the integer pipe, for a normalised pair; ex is added to the
// result's high word (a power of two, given as its exponent << 20).  h = 0 gives 0.
MHDGB_HD double p_join(Pair a, unsigned ex = 0u) {
  const unsigned u = f_bits(a.h);
  const unsigned m = (u & 0x007FFFFFu) | 0x00800000u;
  // l in units of 2^(E - 51), counted along h's sign
  // (below 2^-76 the unit stays put, and l is rounded to 24 bits below h)
  int li = f_to_i(f_mul(a.l, f_from((305u << 23) - u_max(u & 0x7F800000u, 51u << 23))));
  li = (int)u < 0 ? -li : li;
  const unsigned lo = (m << 28) + (unsigned)li;
  const unsigned hi = (m >> 4) + (unsigned)(li >> 31) + (lo < (unsigned)li ? 1u : 0u);
  const int sh = i_clz(hi) - 11;  // 1, or 0 or 2 where l carried h across a power of two
  const unsigned e = ((u & 0x7F800000u) >> 3) + ex + (896u << 20) - ((unsigned)sh << 20);
  const double r = d_from((f_shl(hi, lo, sh) + e) | (u & 0x80000000u), lo << sh);
  return (u & 0x7FFFFFFFu) < 0x00800000u ? 0.0 : r;
}

}  // namespace mhdgb
