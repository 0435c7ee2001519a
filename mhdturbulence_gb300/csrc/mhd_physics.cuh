// mhd_physics.cuh -- per-face physics of the ideal-MHD step, as device functions templated on the
// arithmetic type R (double for the FP64 form, float for the mixed form's reconstruction and
// Riemann solve).
//
// Every expression keeps the operation order of the reference's src_cpp_kokkos_host/mhd.cpp
// (left-to-right evaluation of the C++ source).  Compiled with -fmad=false the FP64 instantiation
// therefore reproduces the reference's separately rounded results bit for bit; compiled with FMA
// contraction it differs from them in the last bits only.  The two builds live in different
// translation units; MHDGB_VNS names the namespace of the current one so that their instantiations
// never merge at link time.
#pragma once

#include "mhd_defs.cuh"

#ifndef MHDGB_VNS
#error "define MHDGB_VNS (v_exact or v_fast) before including mhd_physics.cuh"
#endif
#ifndef MHDGB_FAST
#error "define MHDGB_FAST (0: the reference's expressions, 1: shortened arithmetic) before including"
#endif

#include <type_traits>

#include "common.cuh"
#include "exact64.cuh"
#include "face_split.cuh"

namespace mhdgb {
namespace MHDGB_VNS {

// kFast selects, for the FMA-contracted builds, algebraically identical but shorter forms of a few
// expressions (each marked below) and the division of fdiv(); the bit-exact build keeps the
// reference's expressions and IEEE division.
constexpr bool kFast = MHDGB_FAST != 0;

// Comparisons of doubles on the integer pipe.  GB300 issues FP64 compares and min/max on the FP64
// pipe, which bounds the FP64 form; the integer pipe is nearly idle.  For non-NaN arguments these
// give the results of the FP64 comparisons (min/max order -0 below +0, which only changes the sign of
// a zero).
__device__ __forceinline__ bool pos_nonzero(double x) {  // x > 0
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7FF0000000000000LL;
}
__device__ __forceinline__ bool abs_less(double x, double lim) {  // |x| < lim, for a finite lim > 0
  return (__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFLL) < __double_as_longlong(lim);
}
__device__ __forceinline__ long long order_key(double x) {  // monotone in x
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL);
}
__device__ __forceinline__ double imin(double a, double b) { return order_key(b) < order_key(a) ? b : a; }
__device__ __forceinline__ double imax(double a, double b) { return order_key(a) < order_key(b) ? b : a; }

// x with its sign flipped when neg (a bit operation on the integer pipe, not an FP64 instruction).
__device__ __forceinline__ double negate_if(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}

// FP32 counterparts for the mixed form's solver (FP32 compares are cheap; these keep one code path).
__device__ __forceinline__ float negate_if(float x, bool neg) {
  return __int_as_float(__float_as_int(x) ^ (neg ? (int)0x80000000 : 0));
}
__device__ __forceinline__ bool abs_less(float x, float lim) { return fabsf(x) < lim; }
__device__ __forceinline__ float imin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float imax(float a, float b) { return (a < b) ? b : a; }

// The MUFU approximate reciprocal of an FP32 value (flushes denormals).
__device__ __forceinline__ float rcp_approx_f32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Separately rounded multiply, add and subtract (never contracted into an FMA).
__device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double rn_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rn_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rn_sub(float a, float b) { return __fsub_rn(a, b); }

// Narrowing and widening for FP32 seeds only.  The callers have checked that the argument is a
// finite normal number well inside the float range, and a seed needs no rounding (the Newton steps
// that follow remove its error), so the narrowing truncates the mantissa (error < 2^-23) and the
// widening skips the zero and denormal cases: a few integer operations each, off the FP64 pipe.
__device__ __forceinline__ float seed_narrow(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  return __uint_as_float((hi & 0x80000000u) | (((hi & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lo >> 29));
}
__device__ __forceinline__ double seed_widen(float f) {
  const unsigned u = __float_as_uint(f);
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(u << 29));
}

// FP64 reciprocal from an FP32 seed (integer-pipe narrowing, the MUFU approximate reciprocal) and two
// Newton-Raphson steps r <- r + r(1 - b r): the error of the seed (~2^-22) squares at each step,
// so the result is within about one ulp of 1/b.
__device__ __forceinline__ double rcp_newton(double b) {
  float sf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(sf) : "f"(seed_narrow(b)));
  double r = seed_widen(sf);
  r = fma(r, fma(-b, r, 1.0), r);
  r = fma(r, fma(-b, r, 1.0), r);
  return r;
}

// FP64 square root by Goldschmidt's iteration from an FP32 reciprocal-square-root seed y (MUFU,
// error ~2^-22): g = x y ~ sqrt(x) and h = y/2 ~ 1/(2 sqrt(x)) are refined together by
// r = 1/2 - g h, g += g r, h += h r (error ~2^-44), then one Newton correction of g with the
// residual x - g^2 (formed by an FMA): g += h (x - g^2).  Seven FP64 operations against nine for
// the IEEE routine; arguments outside [2^-120, 2^120] (zero, denormals, negatives, inf, NaN) take
// the IEEE square root.  Given inv, *inv receives 1/sqrt(x) from a second correction of h.
__device__ __forceinline__ bool sqrt_seed_range(double x) {
  const unsigned e = (unsigned)__double2hiint(x) >> 20;  // the sign bit makes negatives fail
  return e >= 1023u - 120u && e <= 1023u + 120u;
}
__device__ __forceinline__ double sqrt_goldschmidt(double x, double* inv = nullptr) {
  float yf;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(seed_narrow(x)));
  const double y = seed_widen(yf);
  double g = x * y, h = 0.5 * y;
  const double r = fma(-g, h, 0.5);
  g = fma(g, r, g);
  h = fma(h, r, h);
  const double d = fma(-g, g, x);
  if (inv) {
    const double r2 = fma(-g, h, 0.5);
    const double hh = fma(h, r2, h);
    *inv = hh + hh;
  }
  return fma(d, h, g);
}

// sqrt: correctly rounded in the exact build, off the FP64 pipe (sqrt_rn); the build's sqrt in FP32;
// sqrt_goldschmidt in the FP64 fast build.
template <class R>
__device__ __forceinline__ R fsqrt(R x) {
  if constexpr (kFast && std::is_same<R, double>::value) {
    return sqrt_seed_range(x) ? sqrt_goldschmidt(x) : sqrt(x);
  } else if constexpr (std::is_same<R, double>::value) {
    return sqrt_rn(x);
  } else {
    return sqrt(x);
  }
}

// sqrt of quantities that only estimate wave speeds (sound and fast speeds, the dt and c_h
// candidates).  FP64 fast build: the FP32 root g0 = x y (y the MUFU reciprocal square root of the
// narrowed x, error ~2^-22) and one Newton correction g0 + (x - g0^2) y / 2, whose residual is
// formed exactly by an FP64 FMA and scaled in FP32 (relative error ~2^-43, two FP64 operations).
// Arguments outside [2^-80, 2^100] (below it a residual that still matters, down to 2x * 2^-43,
// could underflow FP32), zero, negatives, inf and NaN take the IEEE square root.  sqrt otherwise.
template <class R>
__device__ __forceinline__ R fsqrt_est(R x) {
  if constexpr (kFast && std::is_same<R, double>::value) {
    const unsigned e = (unsigned)__double2hiint(x) >> 20;  // the sign bit makes negatives fail
    if (e - (1023u - 80u) > 180u) return sqrt(x);
    const float xf = seed_narrow(x);
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(xf));
    const float g0 = xf * yf;
    const double g0d = seed_widen(g0);
    const double d = fma(-g0d, g0d, x);
    return g0d + f2d_exact(d2f_rne(d) * (0.5f * yf));
  } else {
    return fsqrt(x);
  }
}

// a / b: correctly rounded in the exact build, off the FP64 pipe (div_rn); a * rcp_newton(b) in the FP64 fast build (within ~1.5
// ulp), with IEEE division where |b| is outside the FP32 seed's range; in the FP32 (mixed) build a
// times the MUFU reciprocal (within ~2 ulp, like the build's approximate division, with fewer
// instructions).
template <class R>
__device__ __forceinline__ R fdiv(R a, R b) {
  if constexpr (kFast && std::is_same<R, double>::value) {
    const unsigned e = ((unsigned)__double2hiint(b) >> 20) & 0x7FFu;
    if (e < 1023u - 120u || e > 1023u + 120u) return a / b;
    return a * rcp_newton(b);
  } else if constexpr (kFast && std::is_same<R, float>::value) {
    return a * rcp_approx_f32(b);
  } else {
    return div_rn(a, b);
  }
}

// a / b for quantities that only limit or estimate (slopes, wave-speed estimates, the dt and c_h
// candidates): in the FP64 fast build one Newton step from the FP32 seed (relative error ~2^-44;
// these values reach the state only as a small relative perturbation of a small quantity, ~1e-15
// after a step); fdiv otherwise.
template <class R>
__device__ __forceinline__ R fdiv_est(R a, R b) {
  if constexpr (kFast && std::is_same<R, double>::value) {
    const unsigned e = ((unsigned)__double2hiint(b) >> 20) & 0x7FFu;
    if (e < 1023u - 120u || e > 1023u + 120u) return a / b;
    float sf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(sf) : "f"(seed_narrow(b)));
    const double r = seed_widen(sf);
    return a * fma(r, fma(-b, r, 1.0), r);
  } else {
    return fdiv(a, b);
  }
}

// x / 2, and min / max with the reference's std::min / std::max results, for the exact build on the
// integer pipe.
template <class R>
__device__ __forceinline__ R half_of(R x) {
  if constexpr (!kFast && std::is_same<R, double>::value) {
    const unsigned hi = d_hi(x), lo = d_lo(x), e = (hi >> 20) & 0x7FFu;
    if (e - 2u < 2045u) return d_from(hi - (1u << 20), lo);
    if (((hi << 1) | lo) == 0u) return x;
  }
  return R(0.5) * x;
}
template <class R>
__device__ __forceinline__ bool less_than(R a, R b) {
  if constexpr (!kFast && std::is_same<R, double>::value) {  // a < b: zeros of either sign equal, NaN never less
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    constexpr long long mag = 0x7FFFFFFFFFFFFFFFLL, inf = 0x7FF0000000000000LL;
    return order_key(a) < order_key(b) && ((x | y) & mag) != 0 && (x & mag) <= inf && (y & mag) <= inf;
  } else {
    return a < b;
  }
}
template <class R> __device__ __forceinline__ R xmin(R a, R b) { return less_than(b, a) ? b : a; }
template <class R> __device__ __forceinline__ R xmax(R a, R b) { return less_than(a, b) ? b : a; }

// 2p / s at the accuracy of fdiv_est, with the factor 2 taken into the FP32 seed (exact there):
// y0 = 2 r0 and one Newton step y1 = y0 + r0 (2 - s y0) = 2 r0 (2 - s r0).  One FP64 operation fewer
// than fdiv_est(p + p, s).
__device__ __forceinline__ double twice_div_est(double p, double s) {
  const unsigned e = ((unsigned)__double2hiint(s) >> 20) & 0x7FFu;
  if (e < 1023u - 120u || e > 1023u + 120u) return (p + p) / s;
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(seed_narrow(s)));
  const double h = seed_widen(r0), y0 = seed_widen(2.0f * r0);
  return p * fma(h, fma(-s, y0, 2.0), y0);
}

// 2 a b rounded as (2 a) b, from p = a b > 0: twice p unless p is subnormal or twice it overflows.
__device__ __forceinline__ double twice_product(double p, double a, double b) {
  const unsigned e = (unsigned)__double2hiint(p) >> 20;
  return e - 1u < 2045u ? d_from(d_hi(p) + (1u << 20), d_lo(p)) : 2.0 * a * b;
}
// van_leer_general: the FP64 fast build's expression for the arguments van_leer_split leaves, out of line.
__device__ __noinline__ double van_leer_general(double dsvp, double dsvm) {
  const double p = dsvp * dsvm;
  return pos_nonzero(p) ? twice_div_est(p, dsvp + dsvm) : 0.0;
}
// vanLeer, src_cpp_kokkos_host/mhd.cpp:89-95.  The limited slope of a cell c is
// van_leer(P[c+1]-P[c], P[c]-P[c-1]); the reference evaluates the same expression for the left
// state of face c+1/2 and the right state of face c-1/2 (mhd.cpp:1134-1154), so one evaluation
// per cell and direction gives both.
template <class R>
__device__ __forceinline__ R van_leer(R dsvp, R dsvm) {
  if constexpr (kFast) {  // one product for the test and the numerator: p + p == (2 dsvp) dsvm exactly
    [[maybe_unused]] const R p = dsvp * dsvm;
    if constexpr (std::is_same<R, double>::value) {
      bool ok = true;
      const double s = van_leer_split(dsvp, dsvm, ok);
      return ok ? s : van_leer_general(dsvp, dsvm);
    } else {  // FP32: (p + p) times the MUFU reciprocal, the form the paired evaluation repeats
      return (p > R(0)) ? (p + p) * rcp_approx_f32(dsvp + dsvm) : R(0);
    }
  } else {
    const R p = dsvp * dsvm;
    return pos_nonzero(p) ? fdiv(twice_product(p, dsvp, dsvm), dsvp + dsvm) : R(0);
  }
}

// N slopes of a thread, van_leer(dp[n], dm[n]); in the FP64 fast build they overlap, and those the
// split leaves are replaced afterwards.
template <class R, int N>
__device__ __forceinline__ void van_leer_batch(const R (&dp)[N], const R (&dm)[N], R (&s)[N]) {
  if constexpr (kFast && std::is_same<R, double>::value) {
    unsigned left = 0;
#pragma unroll
    for (int n = 0; n < N; n++) {
      bool ok = true;
      s[n] = van_leer_split(dp[n], dm[n], ok);
      left |= ok ? 0u : 1u << n;
    }
    if (left) {
#pragma unroll
      for (int n = 0; n < N; n++)
        if ((left >> n) & 1u) s[n] = van_leer_general(dp[n], dm[n]);
    }
  } else if constexpr (std::is_same<R, double>::value) {  // the exact build: van_leer's steps, one test for all
    double num[N], den[N];
    bool on[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
      const double p = dp[n] * dm[n];
      on[n] = pos_nonzero(p);
      num[n] = twice_product(p, dp[n], dm[n]);
      den[n] = dp[n] + dm[n];
      if (!on[n]) {  // 0 / 1
        num[n] = 0.0;
        den[n] = 1.0;
      }
    }
    div_many<N>(num, den, s);
  } else {
#pragma unroll
    for (int n = 0; n < N; n++) s[n] = van_leer<R>(dp[n], dm[n]);
  }
}

// The slopes of two adjacent cells at once, from the stencil s0 s1 s2 s3 of a face: the left
// cell's van_leer(s2-s1, s1-s0) and the right cell's van_leer(s3-s2, s2-s1), with packed FP32
// instructions (two lanes per instruction); each lane rounds as the scalar van_leer<float> does,
// so the results are the same bit for bit.  Returns the face's states (s1 + sl/2, s2 - sr/2).
__device__ __forceinline__ float2 van_leer_states_pair(float s0, float s1, float s2, float s3) {
  const float2 lo = make_float2(s0, s1), mid = make_float2(s1, s2);
  const float2 dm = __ffma2_rn(lo, make_float2(-1.0f, -1.0f), mid);  // (s1 - s0, s2 - s1), exact as a subtraction
  const float2 dp = make_float2(dm.y, s3 - s2);                      // (s2 - s1, s3 - s2)
  const float2 p = __fmul2_rn(dp, dm);
  const float2 sum = __fadd2_rn(dp, dm);
  const float2 pp = __fadd2_rn(p, p);
  const float2 q = __fmul2_rn(pp, make_float2(rcp_approx_f32(sum.x), rcp_approx_f32(sum.y)));
  const float2 sl = make_float2(p.x > 0.0f ? q.x : 0.0f, p.y > 0.0f ? q.y : 0.0f);
  return __ffma2_rn(sl, make_float2(0.5f, -0.5f), mid);
}

// Rotation maps of Prim2Cons1/2/3, mhd.cpp:1078-1118.
template <int DIR> struct Dir;
template <> struct Dir<1> {
  static constexpr int muv1 = muvu, muv2 = muvv, muv3 = muvw, mub1 = mubu, mub2 = mubv, mub3 = mubw;
  static constexpr int mfv1 = mfvu, mfv2 = mfvv, mfv3 = mfvw;
  static constexpr int nved = nve1, nbmd = nbm1, nvef = nve2, nbmf = nbm2, nveb = nve3, nbmb = nbm3;
  // output slots, mhd.cpp:1225-1240
  static constexpr int orv1 = mrvu, orv2 = mrvv, orv3 = mrvw, glm = mbm1;
  static constexpr int ob_a = mbm2, sb_a = mubv, ob_b = mbm3, sb_b = mubw;
};
template <> struct Dir<2> {
  static constexpr int muv1 = muvw, muv2 = muvu, muv3 = muvv, mub1 = mubw, mub2 = mubu, mub3 = mubv;
  static constexpr int mfv1 = mfvw, mfv2 = mfvu, mfv3 = mfvv;
  static constexpr int nved = nve2, nbmd = nbm2, nvef = nve3, nbmf = nbm3, nveb = nve1, nbmb = nbm1;
  // mhd.cpp:1306-1321
  static constexpr int orv1 = mrvw, orv2 = mrvu, orv3 = mrvv, glm = mbm2;
  static constexpr int ob_a = mbm1, sb_a = mubw, ob_b = mbm3, sb_b = mubv;
};
template <> struct Dir<3> {
  static constexpr int muv1 = muvv, muv2 = muvw, muv3 = muvu, mub1 = mubv, mub2 = mubw, mub3 = mubu;
  static constexpr int mfv1 = mfvv, mfv2 = mfvw, mfv3 = mfvu;
  static constexpr int nved = nve3, nbmd = nbm3, nvef = nve1, nbmf = nbm1, nveb = nve2, nbmb = nbm2;
  // mhd.cpp:1391-1406
  static constexpr int orv1 = mrvv, orv2 = mrvw, orv3 = mrvu, glm = mbm3;
  static constexpr int ob_a = mbm1, sb_a = mubv, ob_b = mbm2, sb_b = mubw;
};

// Dir<0>: the face's primitives arrive rotated already (normal, first and second tangential
// components in the slots of x, y, z, as Dir<1> reads them), for the fused step's direction-generic
// face list.  rot = 0, 1, 2 for x, y, z faces; the one place it enters the FP64 arithmetic is the
// sums over the three components, which keep the unrotated x, y, z order (sum_sq3), so an FP64
// Dir<0> flux is bit for bit the Dir<1/2/3> flux of the same face.  The FP32 solver sums in the
// rotated order (no selects; every FP32 kernel uses the same order, so they agree bit for bit).
template <> struct Dir<0> : Dir<1> {};

// Unrotated component (0, 1, 2 = x, y, z) held in rotated slot 0, 1, 2 of a face with rotation rot.
__device__ __forceinline__ int unrot_comp(int slot, int rot) { return slot + rot < 3 ? slot + rot : slot + rot - 3; }

// P[b]^2 + P[b+1]^2 + P[b+2]^2 over unrotated components x, y, z in that order.
template <int DIR, class R>
__device__ __forceinline__ R sum_sq3(const R (&P)[NPRIM], int b, int rot) {
  if constexpr (DIR != 0 || std::is_same<R, float>::value) {
    return P[b] * P[b] + P[b + 1] * P[b + 1] + P[b + 2] * P[b + 2];
  } else {
    const R r0 = P[b], r1 = P[b + 1], r2 = P[b + 2];
    const R x = rot == 0 ? r0 : (rot == 1 ? r2 : r1);
    const R y = rot == 0 ? r1 : (rot == 1 ? r0 : r2);
    const R z = rot == 0 ? r2 : (rot == 1 ? r1 : r0);
    return x * x + y * y + z * z;
  }
}

// Prim2ConsD, mhd.cpp:997-1076 (note the energy flux term bsq*B_d of mhd.cpp:1049-1050).
template <class R, int DIR>
__device__ __forceinline__ void prim2cons(const R (&Prim)[NPRIM], R (&Cons)[NVEC], bool left, int rot = 0) {
  using D = Dir<DIR>;
  const R rho = Prim[nden];
  const R rhoinv = fdiv_est(R(1), rho);  // only in the fast-speed estimate below
  const R vsq = sum_sq3<DIR>(Prim, nve1, rot);
  const R bsq = sum_sq3<DIR>(Prim, nbm1, rot);
  Cons[mudn] = rho;
  Cons[D::muv1] = rho * Prim[nve1];
  Cons[D::muv2] = rho * Prim[nve2];
  Cons[D::muv3] = rho * Prim[nve3];
  Cons[muet] = rho * Prim[nene] + half_of(rho) * vsq + half_of(bsq);
  Cons[D::mub1] = Prim[nbm1];
  Cons[D::mub2] = Prim[nbm2];
  Cons[D::mub3] = Prim[nbm3];
  Cons[mubp] = Prim[nbps];
  Cons[must] = rho * Prim[nst];
  const R ptl = Prim[npre] + half_of(bsq);
  Cons[mfdn] = rho * Prim[D::nved];
  Cons[D::mfv1] = rho * Prim[nve1] * Prim[D::nved] - Prim[nbm1] * Prim[D::nbmd];
  Cons[D::mfv2] = rho * Prim[nve2] * Prim[D::nved] - Prim[nbm2] * Prim[D::nbmd];
  Cons[D::mfv3] = rho * Prim[nve3] * Prim[D::nved] - Prim[nbm3] * Prim[D::nbmd];
  Cons[mfet] = (Cons[muet] + ptl) * Prim[D::nved] - bsq * Prim[D::nbmd];
  Cons[mfvu] += ptl;
  Cons[mfbu] = R(0);
  Cons[mfbv] = Prim[D::nbmf] * Prim[D::nved] - Prim[D::nvef] * Prim[D::nbmd];
  if constexpr (kFast && std::is_same<R, float>::value) {
    // Which product is rounded before the other is fused in: left to the compiler, it changed with code far
    // from here, and the mixed form's HLLE and HLLC results with it.
    const R a = Prim[D::nbmb], b = Prim[D::nved], c = Prim[D::nveb], d = Prim[D::nbmd];
    Cons[mfbw] = left ? __fmaf_rn(a, b, -__fmul_rn(c, d)) : __fmaf_rn(-c, d, __fmul_rn(a, b));
  } else {
    Cons[mfbw] = Prim[D::nbmb] * Prim[D::nved] - Prim[D::nveb] * Prim[D::nbmd];
  }
  Cons[mfbp] = R(0);
  Cons[mfst] = rho * Prim[nst] * Prim[D::nved];
  const R css = Prim[ncsp] * Prim[ncsp];
  const R cts = css + bsq * rhoinv;
  Cons[mcsp] = fsqrt_est(half_of(cts + fsqrt_est(cts * cts - R(4) * css * Prim[D::nbmd] * Prim[D::nbmd] * rhoinv)));
  Cons[mvel] = Prim[D::nved];
  Cons[mpre] = ptl;
}

// Prim2ConsD split in two for the FP64 branch-form HLLD, which needs the physical flux of the
// upwind side only: the state part (conserved variables, fast speed, normal velocity, total
// pressure) for both sides, then the flux part for the chosen side, with prim2cons's expressions.
template <class R, int DIR>
__device__ __forceinline__ void prim2cons_state(const R (&Prim)[NPRIM], R (&Cons)[NVEC], int rot = 0) {
  using D = Dir<DIR>;
  const R rho = Prim[nden];
  const R rhoinv = fdiv_est(R(1), rho);
  const R vsq = sum_sq3<DIR>(Prim, nve1, rot);
  const R bsq = sum_sq3<DIR>(Prim, nbm1, rot);
  Cons[mudn] = rho;
  Cons[D::muv1] = rho * Prim[nve1];
  Cons[D::muv2] = rho * Prim[nve2];
  Cons[D::muv3] = rho * Prim[nve3];
  Cons[muet] = rho * Prim[nene] + half_of(rho) * vsq + half_of(bsq);
  Cons[D::mub1] = Prim[nbm1];
  Cons[D::mub2] = Prim[nbm2];
  Cons[D::mub3] = Prim[nbm3];
  Cons[mubp] = Prim[nbps];
  Cons[must] = rho * Prim[nst];
  const R css = Prim[ncsp] * Prim[ncsp];
  const R cts = css + bsq * rhoinv;
  Cons[mcsp] = fsqrt_est(half_of(cts + fsqrt_est(cts * cts - R(4) * css * Prim[D::nbmd] * Prim[D::nbmd] * rhoinv)));
  Cons[mvel] = Prim[D::nved];
  Cons[mpre] = Prim[npre] + half_of(bsq);
}
// The left (x) and right (y) lanes of packed state pairs, indexed like a state vector.
struct PairLo {
  const float2* c;
  __device__ __forceinline__ float operator[](int q) const { return c[q].x; }
};
struct PairHi {
  const float2* c;
  __device__ __forceinline__ float operator[](int q) const { return c[q].y; }
};

// prim2cons_state of a face's two states at once (FP32, rotated frame as Dir<0>): P[n] holds the
// left and right primitive, C[q] receives the two state vectors, with packed FP32 instructions (two
// lanes per instruction) and a fixed order of operations; the sums over the components are in the
// rotated order, as sum_sq3 forms them in FP32.
__device__ __forceinline__ void prim2cons_state_pair(const float2 (&P)[NPRIM], float2 (&C)[NVEC], int) {
  const float2 half = make_float2(0.5f, 0.5f);
  auto sq3 = [&](int b) {  // P[b]^2 + P[b+1]^2 + P[b+2]^2
    return __ffma2_rn(P[b + 2], P[b + 2], __ffma2_rn(P[b + 1], P[b + 1], __fmul2_rn(P[b], P[b])));
  };
  const float2 rho = P[nden];
  const float2 rinv = make_float2(rcp_approx_f32(rho.x), rcp_approx_f32(rho.y));
  const float2 vsq = sq3(nve1), bsq = sq3(nbm1);
  C[mudn] = rho;
  C[muvu] = __fmul2_rn(rho, P[nve1]);
  C[muvv] = __fmul2_rn(rho, P[nve2]);
  C[muvw] = __fmul2_rn(rho, P[nve3]);
  C[muet] = __ffma2_rn(half, bsq, __ffma2_rn(__fmul2_rn(half, rho), vsq, __fmul2_rn(rho, P[nene])));
  C[mubu] = P[nbm1];
  C[mubv] = P[nbm2];
  C[mubw] = P[nbm3];
  C[mubp] = P[nbps];
  C[must] = __fmul2_rn(rho, P[nst]);
  const float2 css = __fmul2_rn(P[ncsp], P[ncsp]);
  const float2 cts = __ffma2_rn(bsq, rinv, css);
  const float2 ca = __fmul2_rn(__fmul2_rn(P[nbm1], P[nbm1]), rinv);  // normal-field Alfven speed squared
  const float2 disc = __ffma2_rn(cts, cts, __fmul2_rn(make_float2(-4.0f, -4.0f), __fmul2_rn(css, ca)));
  const float2 cf2 = __fmul2_rn(half, __fadd2_rn(cts, make_float2(sqrtf(disc.x), sqrtf(disc.y))));
  C[mcsp] = make_float2(sqrtf(cf2.x), sqrtf(cf2.y));
  C[mvel] = P[nve1];
  C[mpre] = __ffma2_rn(half, bsq, P[npre]);
}

// The flux slots (mfdn .. mfst) of Cons from the primitive state and Cons[muet], Cons[mpre].
template <class R, int DIR>
__device__ __forceinline__ void prim2cons_flux(const R (&Prim)[NPRIM], R (&Cons)[NVEC], int rot = 0) {
  using D = Dir<DIR>;
  const R rho = Prim[nden];
  const R bsq = sum_sq3<DIR>(Prim, nbm1, rot);
  const R ptl = Cons[mpre];
  Cons[mfdn] = rho * Prim[D::nved];
  Cons[D::mfv1] = rho * Prim[nve1] * Prim[D::nved] - Prim[nbm1] * Prim[D::nbmd];
  Cons[D::mfv2] = rho * Prim[nve2] * Prim[D::nved] - Prim[nbm2] * Prim[D::nbmd];
  Cons[D::mfv3] = rho * Prim[nve3] * Prim[D::nved] - Prim[nbm3] * Prim[D::nbmd];
  Cons[mfet] = (Cons[muet] + ptl) * Prim[D::nved] - bsq * Prim[D::nbmd];
  Cons[mfvu] += ptl;
  Cons[mfbu] = R(0);
  Cons[mfbv] = Prim[D::nbmf] * Prim[D::nved] - Prim[D::nvef] * Prim[D::nbmd];
  Cons[mfbw] = Prim[D::nbmb] * Prim[D::nved] - Prim[D::nveb] * Prim[D::nbmd];
  Cons[mfbp] = R(0);
  Cons[mfst] = rho * Prim[nst] * Prim[D::nved];
}

// HLLD, mhd.cpp:97-417, for the exact build: the reference's expressions, operation by operation, with
// its 0/1 masks (maxs1 / mins1 of mhd.cpp:272-275, 306-308, 343-346, 384-386) taken as selections, which
// leaves every finite result the same (a product with a mask and the sum with the masked-out zero are
// exact), and the flux formed for the upwind side only (prim2cons_flux fills its flux slots).  Divisions,
// roots, comparisons and halvings run off the FP64 pipe, which bounds this build.  Writes the 10
// rotated fluxes (slot mubp is left undefined: the GLM pair replaces it).
template <int DIR>
__device__ __forceinline__ void hlld(const double (&leftst)[NVEC], const double (&rigtst)[NVEC],
                                     const double (&Pl)[NPRIM], const double (&Pr)[NPRIM], double (&nflux)[NCONS],
                                     int rot = 0) {
  using R = double;
  const R eps = 1.0e-30;
  R v6[6];
  {
    const R num[6] = {leftst[muvu], leftst[muvv], leftst[muvw], rigtst[muvu], rigtst[muvv], rigtst[muvw]};
    const R den[6] = {leftst[mudn], leftst[mudn], leftst[mudn], rigtst[mudn], rigtst[mudn], rigtst[mudn]};
    div_many<6>(num, den, v6);
  }
  const R vxl = v6[0], vyl = v6[1], vzl = v6[2], vxr = v6[3], vyr = v6[4], vzr = v6[5];
  const R ptl = leftst[mpre], ptr = rigtst[mpre];
  // Step 1 (mhd.cpp:212-216)
  const R cfast = xmax(leftst[mcsp], rigtst[mcsp]);
  const R sl = xmin(vxl, vxr) - cfast, sr = xmax(vxl, vxr) + cfast;
  // Step 4 (mhd.cpp:248-258)
  const R sdl = xmin(-1e-20, sl - vxl), sdr = xmax(1e-20, sr - vxr);
  const R rosdl = leftst[mudn] * sdl, rosdr = rigtst[mudn] * sdr;
  const R tden = fdiv(1.0, rosdr - rosdl);
  const R sm = (rosdr * vxr - rosdl * vxl - ptr + ptl) * tden;
  const R sdml = xmin(-1e-20, sl - sm), sdmr = xmax(1e-20, sr - sm);
  // Step 5 (mhd.cpp:264)
  const R ptst = (rosdr * ptl - rosdl * ptr + rosdl * rosdr * (vxr - vxl)) * tden;
  const R bxs = half_of(leftst[mubu] + rigtst[mubu]);
  const R bxsq = bxs * bxs;
  const bool left = !signbit(sm);
  // star states of the upwind side (u) and the other (o), Steps 5A and 5B (mhd.cpp:269-333)
  struct Star {
    R ro, vx, vy, vz, by, bz, isdm;
    bool nondeg;
  };
  auto star = [&](R ro, R vx, R vy, R vz, R by, R bz, R sd, R rosd, R sdm, R f, R isdm, R itf) {
    Star t;
    t.isdm = isdm;
    t.nondeg = !abs_less(f, eps);
    const R t1 = bxs * (sd - sdm) * itf, t2 = (rosd * sd - bxsq) * itf;
    t.ro = t.nondeg ? rosd * t.isdm : ro;
    t.vx = t.nondeg ? sm : vx;
    t.vy = t.nondeg ? vy - by * t1 : vy;
    t.vz = t.nondeg ? vz - bz * t1 : vz;
    t.by = t.nondeg ? by * t2 : by;
    t.bz = t.nondeg ? bz * t2 : bz;
    return t;
  };
  auto sel = [left](R a, R b) { return left ? a : b; };
  R cst[NVEC], pup[NPRIM];  // the upwind side's vectors
#pragma unroll
  for (int q = 0; q < NVEC; q++) cst[q] = sel(leftst[q], rigtst[q]);
#pragma unroll
  for (int n = 0; n < NPRIM; n++) pup[n] = sel(Pl[n], Pr[n]);
  const R ro = cst[mudn], by = cst[mubv], bz = cst[mubw], ee = cst[muet], pt = cst[mpre];
  const R vx = sel(vxl, vxr), vy = sel(vyl, vyr), vz = sel(vzl, vzr), sd = sel(sdl, sdr);
  const R fl = rosdl * sdml - bxsq, fr = rosdr * sdmr - bxsq;
  R inv4[4];  // a degenerate side's 1 / f is not used
  {
    const R one[4] = {1.0, 1.0, 1.0, 1.0};
    const R den[4] = {sdml, sdmr, abs_less(fl, eps) ? 1.0 : fl, abs_less(fr, eps) ? 1.0 : fr};
    div_many<4>(one, den, inv4);
  }
  const Star u = star(ro, vx, vy, vz, by, bz, sd, sel(rosdl, rosdr), sel(sdml, sdmr), sel(fl, fr),
                      sel(inv4[0], inv4[1]), sel(inv4[2], inv4[3]));
  const Star o = star(sel(rigtst[mudn], leftst[mudn]), sel(vxr, vxl), sel(vyr, vyl), sel(vzr, vzl),
                      sel(rigtst[mubv], leftst[mubv]), sel(rigtst[mubw], leftst[mubw]), sel(sdr, sdl),
                      sel(rosdr, rosdl), sel(sdmr, sdml), sel(fr, fl), sel(inv4[1], inv4[0]), sel(inv4[3], inv4[2]));
  const R rost = u.ro, rxst = rost * u.vx, ryst = rost * u.vy, rzst = rost * u.vz;
  const R vdbst = u.vx * bxs + u.vy * u.by + u.vz * u.bz;
  R eest = ee;
  if (u.nondeg) {  // the reference sums the two sides' numerators in different orders (mhd.cpp:297-300, 329-333)
    const R a = sd * ee - pt * vx + ptst * sm, b = bxs * (vx * bxs + vy * by + vz * bz - vdbst);
    eest = left ? (a + b) * u.isdm : a * u.isdm + b * u.isdm;
  }
  // Step 5C (mhd.cpp:338-377) and the Alfven speed of Step 6 (mhd.cpp:381-383)
  R rydst = ryst, rzdst = rzst, bydst = u.by, bzdst = u.bz, eedst = eest, sst = 0.0;
  if (!abs_less(bxs, eps)) {
    bool ok = true;
    R sq = sqrt_core(rost, ok), sqo = sqrt_core(o.ro, ok);
    if (!ok) {
      sq = sqrt_ieee(rost);
      sqo = sqrt_ieee(o.ro);
    }
    const R ql = sel(sq, sqo), qr = sel(sqo, sq);
    const R vylst = sel(u.vy, o.vy), vyrst = sel(o.vy, u.vy), vzlst = sel(u.vz, o.vz), vzrst = sel(o.vz, u.vz);
    const R bylst = sel(u.by, o.by), byrst = sel(o.by, u.by), bzlst = sel(u.bz, o.bz), bzrst = sel(o.bz, u.bz);
    const bool neg = signbit(bxs);
    R is[2];
    {
      const R num[2] = {1.0, fabs(bxs)}, den[2] = {ql + qr, sq};
      div_many<2>(num, den, is);
    }
    const R inv = is[0];
    const R vydst = inv * (ql * vylst + qr * vyrst + negate_if(byrst - bylst, neg));
    const R vzdst = inv * (ql * vzlst + qr * vzrst + negate_if(bzrst - bzlst, neg));
    const R sqq = negate_if(ql, neg) * qr;
    bydst = inv * (ql * byrst + qr * bylst + sqq * (vyrst - vylst));
    bzdst = inv * (ql * bzrst + qr * bzlst + sqq * (vzrst - vzlst));
    rydst = rost * vydst;
    rzdst = rost * vzdst;
    const R vdb = sm * bxs + vydst * bydst + vzdst * bzdst;
    const R de = negate_if(sq, neg) * (vdbst - vdb);
    eedst = left ? eest - de : eest + de;
    sst = left ? sm - is[1] : sm + is[1];
  }
  // Step 6 (mhd.cpp:384-415)
  const R ms = left ? xmin(sl, 0.0) : xmax(sr, 0.0), msst = left ? xmin(sst, 0.0) : xmax(sst, 0.0);
  prim2cons_flux<R, DIR>(pup, cst, rot);
  nflux[mden] = cst[mfdn] + (rost - ro) * ms;
  nflux[meto] = cst[mfet] + (eest - ee) * ms + (eedst - eest) * msst;
  nflux[mrv1] = cst[mfvu] + (rxst - cst[muvu]) * ms;
  nflux[mrv2] = cst[mfvv] + (ryst - cst[muvv]) * ms + (rydst - ryst) * msst;
  nflux[mrv3] = cst[mfvw] + (rzst - cst[muvw]) * ms + (rzdst - rzst) * msst;
  nflux[mbm1] = 0.0;
  nflux[mbm2] = cst[mfbv] + (u.by - by) * ms + (bydst - u.by) * msst;
  nflux[mbm3] = cst[mfbw] + (u.bz - bz) * ms + (bzdst - u.bz) * msst;
  nflux[mst] = cst[mfst] + (fdiv(rost, ro) * cst[must] - cst[must]) * ms;
  nflux[mbps] = 0.0;
}

// HLLD in branch form, for the FMA-contracted builds (FP64 and the mixed form's FP32 solve).  Same
// states and fluxes as hlld(), but the selections the reference performs with 0/1 masks
// (maxs1/mins1 of mhd.cpp:272-275, 306-308, 343-346, 384-386) are branches: the degenerate-field
// forms are taken only when their conditions hold, and only the upwind side's physical flux is
// formed (face_flux() passes states without flux slots; prim2cons_flux() fills the upwind side's).
// Results agree with hlld() to rounding (and in the sign of zero results).
// leftst / rigtst: the two state vectors, as arrays or as PairLo / PairHi views of packed pairs.
template <class R, int DIR, class CL, class CR>
__device__ __forceinline__ void hlld_branch(const CL& leftst, const CR& rigtst, const R (&Pl)[NPRIM],
                                            const R (&Pr)[NPRIM], R (&nflux)[NCONS], int rot = 0) {
  using D = Dir<DIR>;
  const R eps = R(1.0e-30);
  const R rol = leftst[mudn], eel = leftst[muet];
  const R vxl = Pl[D::nved], vyl = Pl[D::nvef], vzl = Pl[D::nveb];
  const R byl = leftst[mubv], bzl = leftst[mubw], ptl = leftst[mpre];
  const R ror = rigtst[mudn], eer = rigtst[muet];
  const R vxr = Pr[D::nved], vyr = Pr[D::nvef], vzr = Pr[D::nveb];
  const R byr = rigtst[mubv], bzr = rigtst[mubw], ptr = rigtst[mpre];
  const R cfl = leftst[mcsp], cfr = rigtst[mcsp];
  // min/max and the eps tests below are integer-pipe comparisons (imin, imax, abs_less)
  const R cmax = imax(cfl, cfr);
  const R sl = imin(vxl, vxr) - cmax;
  const R sr = imax(vxl, vxr) + cmax;
  const R sdl = imin(R(-1e-20), sl - vxl);
  const R sdr = imax(R(1e-20), sr - vxr);
  const R rosdl = rol * sdl;
  const R rosdr = ror * sdr;
  const R tden = fdiv(R(1), rosdr - rosdl);
  // The contact speed decides the upwind side, and the reference's fluxes differ on the two sides of
  // S_M = 0 when B_n != 0 (e.g. the energy flux at a reflecting wall, whose two states are mirror
  // images).  There the reference's separately rounded products cancel to exactly +0 and it takes
  // the left side; an FMA-contracted numerator would leave the rounding error of one product, of
  // either sign.  So the numerator is formed from separately rounded products, as the reference does.
  const R sm = rn_mul(rn_add(rn_add(rn_sub(rn_mul(rosdr, vxr), rn_mul(rosdl, vxl)), -ptr), ptl), tden);
  const R ptst = (rosdr * ptl - rosdl * ptr + rosdl * rosdr * (vxr - vxl)) * tden;
  const R bxs = R(0.5) * (leftst[mubu] + rigtst[mubu]);
  const R bxsq = bxs * bxs;
  const bool left = !signbit(sm);  // copysign(1, sm) > 0, mhd.cpp:384
  // The left side's clamps min(-1e-20, x) and min(x, 0) are the right side's max(1e-20, -x) and
  // max(-x, 0) negated: each selection is one max on the chosen side with sign flips (bit
  // operations) instead of both arms.
  auto side_max = [&](R floor_, R x, bool neg) { return negate_if(imax(floor_, negate_if(x, neg)), neg); };
  // upwind side only: s = side speed, sd = s - v, sdm = s - sm, ro/e/v/b of that side
  const R s_ = left ? sl : sr;
  const R sd = left ? sdl : sdr;
  const R rosd = left ? rosdl : rosdr;
  const R sdm = side_max(R(1e-20), s_ - sm, left);
  const R ro = left ? rol : ror, ee = left ? eel : eer, pt = left ? ptl : ptr;
  const R vx = left ? vxl : vxr, vy = left ? vyl : vyr, vz = left ? vzl : vzr;
  const R by = left ? byl : byr, bz = left ? bzl : bzr;
  const R sc = left ? Pl[nst] : Pr[nst];
  // star state of the upwind side (Step 5A/5B); one reciprocal of sdm * T gives 1/sdm and 1/T
  R rost = ro, vxst = vx, vyst = vy, vzst = vz, byst = by, bzst = bz;
  const R temp_fst = rosd * sdm - bxsq;
  // Degenerate star states (rho (S - v)(S - S_M) = B_x^2, e.g. field-aligned flow with c_f = v_A):
  // the reference switches to v* = v, B* = B below |T| < 1e-30, which FP64 rounding noise (~1e-16)
  // never reaches.  In FP32, T and the numerators it divides are rounding noise (~1e-7 of p_T*)
  // near degeneracy, so the FP32 solver treats |T| < 1e-6 p_T* (about eight FP32 ulps of the star
  // total pressure) as degenerate.  Above that the FP32 star state still follows FP64's: on the
  // low-beta KH layer (B_x = 1, p = 0.1) thresholds from 3e-7 to 3e-6 give the same state, while
  // 1e-5 and above switch faces the FP64 solver resolves, and its absolute 1e-30 fails in FP32.
  const R deg = std::is_same<R, float>::value ? imax(eps, R(1e-6) * fabs(ptst)) : eps;
  const bool nondeg = !abs_less(temp_fst, deg);
  R isdm = R(0);
  if (nondeg) {
    const R rr = fdiv(R(1), sdm * temp_fst);
    isdm = temp_fst * rr;
    const R itf = sdm * rr;
    const R t1 = bxs * (sd - sdm) * itf;
    rost = rosd * isdm;
    vxst = sm;
    vyst = vy - by * t1;
    vzst = vz - bz * t1;
    const R t2 = (rosd * sd - bxsq) * itf;
    byst = by * t2;
    bzst = bz * t2;
  }
  const R vdbst = vxst * bxs + vyst * byst + vzst * bzst;
  const R eest = nondeg ? (sd * ee - pt * vx + ptst * sm + bxs * (vx * bxs + vy * by + vz * bz - vdbst)) * isdm : ee;
  // Alfven (double-star) correction of the tangential states and energy (Step 5C), needs both
  // star states: the other side's star state is formed the same way.
  const R so_sd = left ? sdr : sdl;
  const R so_rosd = left ? rosdr : rosdl;
  const R so_sdm = side_max(R(1e-20), (left ? sr : sl) - sm, !left);
  const R so_ro = left ? ror : rol;
  const R so_vy = left ? vyr : vyl, so_vz = left ? vzr : vzl, so_by = left ? byr : byl, so_bz = left ? bzr : bzl;
  R so_rost = so_ro, so_vyst = so_vy, so_vzst = so_vz, so_byst = so_by, so_bzst = so_bz;
  const R so_tf = so_rosd * so_sdm - bxsq;
  if (!abs_less(so_tf, deg)) {
    const R rr = fdiv(R(1), so_sdm * so_tf);
    const R itf = so_sdm * rr;
    const R t1 = bxs * (so_sd - so_sdm) * itf;
    so_rost = so_rosd * (so_tf * rr);
    so_vyst = so_vy - so_by * t1;
    so_vzst = so_vz - so_bz * t1;
    const R t2 = (so_rosd * so_sd - bxsq) * itf;
    so_byst = so_by * t2;
    so_bzst = so_bz * t2;
  }
  const R abbx = fabs(bxs);
  const bool bneg = signbit(bxs);  // signbx = copysign(1, bxs) < 0
  R vydst = vyst, vzdst = vzst, bydst = byst, bzdst = bzst, eedst = eest, sst = R(0);
  if (!abs_less(bxs, eps)) {
    // sqrt of the upwind star density and its reciprocal from one Goldschmidt iteration
    R sq, isq;
    if constexpr (std::is_same<R, double>::value) {
      if (sqrt_seed_range(rost)) {
        sq = sqrt_goldschmidt(rost, &isq);
      } else {
        sq = sqrt(rost);
        isq = R(1) / sq;
      }
    } else {
      sq = sqrt(rost);
      isq = R(1) / sq;
    }
    const R so_sq = fsqrt(so_rost);
    // (sqrtrol, sqrtror) ordered as in the reference
    const R sql = left ? sq : so_sq, sqr = left ? so_sq : sq;
    const R invsumro = fdiv(R(1), sql + sqr);
    const R vyl_st = left ? vyst : so_vyst, vyr_st = left ? so_vyst : vyst;
    const R vzl_st = left ? vzst : so_vzst, vzr_st = left ? so_vzst : vzst;
    const R byl_st = left ? byst : so_byst, byr_st = left ? so_byst : byst;
    const R bzl_st = left ? bzst : so_bzst, bzr_st = left ? so_bzst : bzst;
    vydst = invsumro * (sql * vyl_st + sqr * vyr_st + negate_if(byr_st - byl_st, bneg));
    vzdst = invsumro * (sql * vzl_st + sqr * vzr_st + negate_if(bzr_st - bzl_st, bneg));
    const R sgq = negate_if(sql * sqr, bneg);  // signbx * sqrtrol * sqrtror
    bydst = invsumro * (sql * byr_st + sqr * byl_st + sgq * (vyr_st - vyl_st));
    bzdst = invsumro * (sql * bzr_st + sqr * bzl_st + sgq * (vzr_st - vzl_st));
    const R tdd = sm * bxs + vydst * bydst + vzdst * bzdst;
    // left: eest - sq signbx (vdbst - tdd); right: eest + sq signbx (vdbst - tdd)
    eedst = eest + negate_if(sq * (vdbst - tdd), bneg != left);
    // left: sm - |bx|/sq; right: sm + |bx|/sq
    sst = sm + negate_if(abbx * isq, left);
  }
  // Step 6: flux of the upwind side (ms = min(s, 0) on the left, max(s, 0) on the right)
  const R ms = side_max(R(0), s_, left);
  const R msst = side_max(R(0), sst, left);
  // physical flux of the upwind side only (its state part is already in leftst / rigtst)
  R cst[NVEC];
#pragma unroll
  for (int q = 0; q < NVEC; q++) cst[q] = left ? leftst[q] : rigtst[q];
  R pup[NPRIM];
#pragma unroll
  for (int n = 0; n < NPRIM; n++) pup[n] = left ? Pl[n] : Pr[n];
  prim2cons_flux<R, DIR>(pup, cst, rot);
  const R rx = cst[muvu], ry = cst[muvv], rz = cst[muvw];
  nflux[mden] = cst[mfdn] + (rost - ro) * ms;
  nflux[meto] = cst[mfet] + (eest - ee) * ms + (eedst - eest) * msst;
  nflux[mrv1] = cst[mfvu] + (rost * vxst - rx) * ms;
  const R ryst = rost * vyst, rzst = rost * vzst;
  nflux[mrv2] = cst[mfvv] + (ryst - ry) * ms + (rost * vydst - ryst) * msst;
  nflux[mrv3] = cst[mfvw] + (rzst - rz) * ms + (rost * vzdst - rzst) * msst;
  nflux[mbm1] = R(0);
  nflux[mbm2] = cst[mfbv] + (byst - by) * ms + (bydst - byst) * msst;
  nflux[mbm3] = cst[mfbw] + (bzst - bz) * ms + (bzdst - bzst) * msst;
  nflux[mst] = cst[mfst] + (rost * sc - cst[must]) * ms;
  nflux[mbps] = R(0);
}

// HLLE of the Fortran variant (src_f90_acc_device/mhd.f90:877-907), on the same rotated state/flux
// vectors as hlld(): one intermediate state between the fastest left- and right-going signals
// sl = min(0, min(vl,vr) - max(cfl,cfr)), sr = max(0, max(vl,vr) + max(cfl,cfr)).
template <class R, int DIR>
__device__ __forceinline__ void hlle(const R (&leftst)[NVEC], const R (&rigtst)[NVEC], R (&nflux)[NCONS]) {
  const R csl = leftst[mcsp], csr = rigtst[mcsp];
  const R vl = leftst[mvel], vr = rigtst[mvel];
  R sl = xmin(vl, vr) - xmax(csl, csr);
  sl = xmin(R(0), sl);
  R sr = xmax(vl, vr) + xmax(csl, csr);
  sr = xmax(R(0), sr);
  if constexpr (kFast) {
    const R inv = fdiv(R(1), sr - sl);
#pragma unroll
    for (int m = 0; m < NCONS; m++)
      nflux[m] = (sr * leftst[NCONS + m] - sl * rigtst[NCONS + m] + sl * sr * (rigtst[m] - leftst[m])) * inv;
  } else {
#pragma unroll
    for (int m = 0; m < NCONS; m++)
      nflux[m] = fdiv(sr * leftst[NCONS + m] - sl * rigtst[NCONS + m] + sl * sr * (rigtst[m] - leftst[m]), sr - sl);
  }
}

// HLLC of the Fortran variant (src_f90_acc_device/mhd.f90:909-1141; Toro, Spruce & Speares): the
// contact speed sm and total pressure ptst of eqs. 45 and 49, star states with the transverse field
// scaled by rho*/rho, and the upwind side's flux chosen by the sign of sm.  The Fortran routine
// reads a passive-scalar star state it never sets; here it is scaled by rho*/rho like the field.
template <class R, int DIR>
__device__ __forceinline__ void hllc(const R (&leftst)[NVEC], const R (&rigtst)[NVEC], const R (&Pl)[NPRIM],
                                     const R (&Pr)[NPRIM], R (&nflux)[NCONS]) {
  using D = Dir<DIR>;
  const R rol = leftst[mudn], eel = leftst[muet];
  const R rxl = leftst[muvu], ryl = leftst[muvv], rzl = leftst[muvw];
  const R ror = rigtst[mudn], eer = rigtst[muet];
  const R rxr = rigtst[muvu], ryr = rigtst[muvv], rzr = rigtst[muvw];
  R vxl, vyl, vzl, vxr, vyr, vzr;
  if constexpr (kFast) {  // the reconstructed velocities these momenta were formed from
    vxl = Pl[D::nved]; vyl = Pl[D::nvef]; vzl = Pl[D::nveb];
    vxr = Pr[D::nved]; vyr = Pr[D::nvef]; vzr = Pr[D::nveb];
  } else {
    vxl = fdiv(leftst[muvu], rol); vyl = fdiv(leftst[muvv], rol); vzl = fdiv(leftst[muvw], rol);
    vxr = fdiv(rigtst[muvu], ror); vyr = fdiv(rigtst[muvv], ror); vzr = fdiv(rigtst[muvw], ror);
  }
  const R scl = leftst[must], scr = rigtst[must];
  const R byl = leftst[mubv], bzl = leftst[mubw], byr = rigtst[mubv], bzr = rigtst[mubw];
  const R ptl = leftst[mpre], ptr = rigtst[mpre];
  const R cfl = leftst[mcsp], cfr = rigtst[mcsp];
  const R sl = xmin(vxl, vxr) - xmax(cfl, cfr);
  const R sr = xmax(vxl, vxr) + xmax(cfl, cfr);
  const R sdl = sl - vxl, sdr = sr - vxr;
  const R rosdl = rol * sdl, rosdr = ror * sdr;
  const R temp = fdiv(R(1), rosdr - rosdl);
  // separately rounded, so mirror-image states give exactly +0 as in the reference (see hlld_branch)
  const R sm = rn_mul(rn_add(rn_add(rn_sub(rn_mul(rosdr, vxr), rn_mul(rosdl, vxl)), -ptr), ptl), temp);
  const R sdml = sl - sm, isdml = fdiv(R(1), sdml);
  const R sdmr = sr - sm, isdmr = fdiv(R(1), sdmr);
  const R ptst = (rosdr * ptl - rosdl * ptr + rosdl * rosdr * (vxr - vxl)) * temp;
  const R rolst = rol * sdl * isdml;
  const R rxlst = rolst * sm, rylst = rolst * vyl, rzlst = rolst * vzl;
  const R bylst = rolst / rol * byl, bzlst = rolst / rol * bzl, sclst = rolst / rol * scl;
  const R eelst = (sdl * eel - ptl * vxl + ptst * sm) * isdml;
  const R rorst = rosdr * isdmr;
  const R rxrst = rorst * sm, ryrst = rorst * vyr, rzrst = rorst * vzr;
  const R byrst = rorst / ror * byr, bzrst = rorst / ror * bzr, scrst = rorst / ror * scr;
  const R eerst = (sdr * eer - ptr * vxr + ptst * sm) * isdmr;
  const R sign1 = copysign(R(1), sm);
  const R maxs1 = xmax(R(0), sign1), mins1 = -xmin(R(0), sign1);
  const R msl = xmin(sl, R(0)), msr = xmax(sr, R(0));
  nflux[mden] = (leftst[mfdn] + msl * (rolst - rol)) * maxs1 + (rigtst[mfdn] + msr * (rorst - ror)) * mins1;
  nflux[meto] = (leftst[mfet] + msl * (eelst - eel)) * maxs1 + (rigtst[mfet] + msr * (eerst - eer)) * mins1;
  nflux[mrvu] = (leftst[mfvu] + msl * (rxlst - rxl)) * maxs1 + (rigtst[mfvu] + msr * (rxrst - rxr)) * mins1;
  nflux[mrvv] = (leftst[mfvv] + msl * (rylst - ryl)) * maxs1 + (rigtst[mfvv] + msr * (ryrst - ryr)) * mins1;
  nflux[mrvw] = (leftst[mfvw] + msl * (rzlst - rzl)) * maxs1 + (rigtst[mfvw] + msr * (rzrst - rzr)) * mins1;
  nflux[mbmu] = R(0);
  nflux[mbmv] = (leftst[mfbv] + msl * (bylst - byl)) * maxs1 + (rigtst[mfbv] + msr * (byrst - byr)) * mins1;
  nflux[mbmw] = (leftst[mfbw] + msl * (bzlst - bzl)) * maxs1 + (rigtst[mfbw] + msr * (bzrst - bzr)) * mins1;
  nflux[mbps] = R(0);
  nflux[mst] = (leftst[mfst] + msl * (sclst - scl)) * maxs1 + (rigtst[mfst] + msr * (scrst - scr)) * mins1;
}

// Face flux from the reconstructed left/right primitive states: Prim2Cons of both sides, the Riemann
// solver (HLLD as in the C++ path by default; HLLE or HLLC, the Fortran variant's alternatives),
// then the rotation back to (rho, m1, m2, m3, E, B1, B2, B3, psi, X) order with the GLM pair for
// the normal field and psi (mhd.cpp:1223-1240 and equivalents).
// riemann selects the solver (RIEMANN_HLLD / _HLLE / _HLLC); it is the same for a whole launch.
// GLM constants of a step (c_h, 0.5 / c_h, c_h^2), formed once rather than per face.
template <class R> struct GlmConst {
  R chg, hoc, chg2;
};
template <class R>
__device__ __forceinline__ GlmConst<R> glm_const(R chg) {
  return GlmConst<R>{chg, fdiv(R(0.5), chg), chg * chg};
}
// DIR = 0: rotated primitives (see Dir<0>) and F in the rotated order of Dir<1> (normal, first and
// second tangential momentum and field fluxes); the caller puts them back in their slots.
template <class R, int DIR>
__device__ __forceinline__ void face_flux(const R (&Pl)[NPRIM], const R (&Pr)[NPRIM], const GlmConst<R>& g,
                                          R (&F)[NCONS], int riemann = RIEMANN_HLLD, int rot = 0) {
  const R chg = g.chg;
  using D = Dir<DIR>;
  R Cl[NVEC], Cr[NVEC], nf[NCONS];
  constexpr bool branch_hlld = kFast;
  if constexpr (branch_hlld && std::is_same<R, float>::value && DIR == 0) {
    if (riemann == RIEMANN_HLLD) {  // FP32: both sides' states in packed pairs, read in place by HLLD
      float2 P2[NPRIM], C2[NVEC];
#pragma unroll
      for (int n = 0; n < NPRIM; n++) P2[n] = make_float2(Pl[n], Pr[n]);
      prim2cons_state_pair(P2, C2, rot);
      hlld_branch<R, DIR>(PairLo{C2}, PairHi{C2}, Pl, Pr, nf, rot);
      F[mden] = nf[mden];
      F[mrv1] = nf[D::orv1];
      F[mrv2] = nf[D::orv2];
      F[mrv3] = nf[D::orv3];
      F[meto] = nf[meto];
      F[D::ob_a] = nf[D::sb_a];
      F[D::ob_b] = nf[D::sb_b];
      const R bpl = C2[mubp].x, bpr = C2[mubp].y, bul = C2[mubu].x, bur = C2[mubu].y;
      F[D::glm] = R(0.5) * (bpl + bpr) - R(0.5) * chg * (bur - bul);
      F[mbps] = (R(0.5) * (bul + bur) - fdiv(R(0.5), chg) * (bpr - bpl)) * chg * chg;
      F[mst] = nf[mst];
      return;
    }
  }
  if (riemann == RIEMANN_HLLD) {  // the upwind flux is formed inside hlld_branch / hlld
    prim2cons_state<R, DIR>(Pl, Cl, rot);
    prim2cons_state<R, DIR>(Pr, Cr, rot);
  } else {
    prim2cons<R, DIR>(Pl, Cl, true, rot);
    prim2cons<R, DIR>(Pr, Cr, false, rot);
  }
  if (riemann == RIEMANN_HLLE) {
    hlle<R, DIR>(Cl, Cr, nf);
  } else if (riemann == RIEMANN_HLLC) {
    hllc<R, DIR>(Cl, Cr, Pl, Pr, nf);
  } else {
    if constexpr (branch_hlld) hlld_branch<R, DIR>(Cl, Cr, Pl, Pr, nf, rot);
    else hlld<DIR>(Cl, Cr, Pl, Pr, nf, rot);
  }
  F[mden] = nf[mden];
  F[mrv1] = nf[D::orv1];
  F[mrv2] = nf[D::orv2];
  F[mrv3] = nf[D::orv3];
  F[meto] = nf[meto];
  // HLLD output slots for the two tangential fields (numflux[mbmv]/[mbmw] = slots 6/7)
  F[D::ob_a] = nf[D::sb_a];
  F[D::ob_b] = nf[D::sb_b];
  F[D::glm] = half_of(Cl[mubp] + Cr[mubp]) - R(0.5) * chg * (Cr[mubu] - Cl[mubu]);
  if constexpr (kFast && std::is_same<R, double>::value) {  // hoisted 0.5/c_h and c_h^2
    F[mbps] = (R(0.5) * (Cl[mubu] + Cr[mubu]) - g.hoc * (Cr[mubp] - Cl[mubp])) * g.chg2;
  } else if constexpr (kFast) {  // FP32: recomputed per face (cheap, and two fewer live registers)
    F[mbps] = (R(0.5) * (Cl[mubu] + Cr[mubu]) - fdiv(R(0.5), chg) * (Cr[mubp] - Cl[mubp])) * chg * chg;
  } else {  // the reference's order: ((...) * chg) * chg
    F[mbps] = (half_of(Cl[mubu] + Cr[mubu]) - g.hoc * (Cr[mubp] - Cl[mubp])) * chg * chg;
  }
  F[mst] = nf[mst];
}

// Left state of face c+1/2 and right state of face c-1/2 from cell value p and limited slope s
// (mhd.cpp:1139 and 1153).
template <class R> __device__ __forceinline__ R left_state(R p, R s) { return p + half_of(s); }
template <class R> __device__ __forceinline__ R right_state(R p, R s) { return p - half_of(s); }

// UpdatePrimitvP for one cell, mhd.cpp:1483-1506.  u: 10 conserved values -> p: 12 primitives.
template <class R>
__device__ __forceinline__ void cons2prim(const R (&u)[NCONS], R gam, R (&p)[NPRIM]) {
  const R rho = u[mden];
  const R rhoinv = fdiv(R(1), rho);
  p[nden] = rho;
  p[nve1] = u[mrv1] * rhoinv;
  p[nve2] = u[mrv2] * rhoinv;
  p[nve3] = u[mrv3] * rhoinv;
  const R m2 = u[mrv1] * u[mrv1] + u[mrv2] * u[mrv2] + u[mrv3] * u[mrv3];
  const R b2 = u[mbm1] * u[mbm1] + u[mbm2] * u[mbm2] + u[mbm3] * u[mbm3];
  if constexpr (kFast) {  // (E - m^2 / (2 rho) - B^2 / 2) / rho in two FMAs
    p[nene] = fma(R(-0.5) * rhoinv, m2, fma(R(-0.5), b2, u[meto])) * rhoinv;
  } else {
    const R ekin = half_of(m2) * rhoinv, emag = half_of(b2);
    p[nene] = fdiv(u[meto] - ekin - emag, u[mden]);
  }
  p[npre] = p[nene] * p[nden] * (gam - R(1));
  p[ncsp] = fsqrt_est(p[nene] * gam * (gam - R(1)));  // the sound speed only enters wave-speed estimates
  p[nbm1] = u[mbm1];
  p[nbm2] = u[mbm2];
  p[nbm3] = u[mbm3];
  p[nbps] = u[mbps];
  p[nst] = u[mst] * rhoinv;
}

// Per-cell CFL time (ControlTimestep, mhd.cpp:1542-1550): min over d of dx_d/(|v_d| + ctot).
template <class R>
__device__ __forceinline__ R cell_dt(const R (&p)[NPRIM], R dx, R dy, R dz) {
  const R ctot = fsqrt_est(p[ncsp] * p[ncsp] + fdiv_est(p[nbm1] * p[nbm1] + p[nbm2] * p[nbm2] + p[nbm3] * p[nbm3], p[nden]));
  R dt = fdiv_est(dx, fabs(p[nve1]) + ctot);
  const R b = fdiv_est(dy, fabs(p[nve2]) + ctot);
  const R c = fdiv_est(dz, fabs(p[nve3]) + ctot);
  if constexpr (kFast && std::is_same<R, double>::value) return imin(imin(dt, b), c);  // integer pipe
  return xmin(xmin(dt, b), c);
}

// Per-cell maximum signal speed (EvaluateCh, mhd.cpp:1589-1601).
template <class R>
__device__ __forceinline__ R cell_ch(const R (&p)[NPRIM]) {
  const R css = p[ncsp] * p[ncsp];
  const R ri = kFast ? fdiv_est(R(1), p[nden]) : R(0);  // fast form: one reciprocal of rho
  const R ca1 = kFast ? p[nbm1] * p[nbm1] * ri : fdiv(p[nbm1] * p[nbm1], p[nden]);
  const R ca2 = kFast ? p[nbm2] * p[nbm2] * ri : fdiv(p[nbm2] * p[nbm2], p[nden]);
  const R ca3 = kFast ? p[nbm3] * p[nbm3] * ri : fdiv(p[nbm3] * p[nbm3], p[nden]);
  const R cts = css + ca1 + ca2 + ca3;
  const R cm1 = fsqrt_est(half_of(cts + fsqrt_est(cts * cts - R(4) * css * ca1)));
  const R ch1 = (fabs(p[nve1]) + cm1);
  const R cm2 = fsqrt_est(half_of(cts + fsqrt_est(cts * cts - R(4) * css * ca2)));
  const R ch2 = (fabs(p[nve2]) + cm2);
  const R cm3 = fsqrt_est(half_of(cts + fsqrt_est(cts * cts - R(4) * css * ca3)));
  const R ch3 = (fabs(p[nve3]) + cm3);
  R m = ch1;
  if constexpr (kFast && std::is_same<R, double>::value) return imax(imax(m, ch2), ch3);  // integer pipe
  return xmax(xmax(m, ch2), ch3);
}

}  // namespace MHDGB_VNS
}  // namespace mhdgb
