// face_split.cuh -- the FP64 form's face flux with its work split by the accuracy each part needs.
//
// The flux through a face is the upwind side's physical flux plus corrections (star and double-star
// states minus the upwind state, times wave speeds) that are proportional to the jump across the
// face.  The physical flux, the jumps and the GLM pair are FP64.  The corrections need less: they
// are products with wave speeds that an estimate of the fast speed sets, which the FP64 form takes at
// about 2^-43, so they are formed from pairs of FP32 values (fp32pair.cuh, about 2^-46) on pipes that
// are otherwise idle.  Each is written in the small quantities that drive it (the contact speed
// relative to the side, the jumps), never as a difference of two nearly equal states, so its
// relative accuracy carries over to the flux however small the jump is; strong jumps take the general FP64
// flux (kJump):
//
//   w  = max(c_f) + max(0, v_l - v_r)        the outer waves run at v_l - w and v_r + w
//   d  = S_M - v                             from the jumps of v and of the total pressure
//   rho* - rho = rho d / (S - S_M),  m_n* - m_n = (rho* - rho) S
//   v_t* - v_t = -B_n B_t d / T,     B_t* - B_t = rho (S - v) B_t d / T,  T = rho (S-v)(S-S_M) - B_n^2
//   E* - E     = [d (E + p_T + rho (S-v) S_M) + B_n (v.B - v*.B*)] / (S - S_M)
//   v_t** - v_t* = (sqrt(rho_o*) J_v + h J_B) / (sqrt(rho*) + sqrt(rho_o*)),  B_t** - B_t* = h sqrt(rho*) (v_t** - v_t*)
//
// with _o the other side, J the star states' jump from this side to the other and h = +-1 the sign of
// B_n as seen from this side.  These are the reference's HLLD states (mhd.cpp:97-417) rearranged.
//
// What bounds it: a warp's FP64 instruction keeps its sub-partition's FP64 path busy for 65 cycles
// (19 per instruction and SM with all four in use), so a face costs about 67 x 76 cycles of that
// path and, beside it, 2200 other instructions.  Hence nothing here that the pairs can hold is FP64, the
// corrections enter as the innermost addend of the flux's last FMAs, and there are no branches before
// the end, so that one face's conversions, pair chains and FP64 instructions overlap.
//
// Measured on the FP64 fused step (KH 150^3 / 256^3): 2.68 / 2.57 -> 1.09 / 1.02 ns per cell and step,
// FP64-pipe instructions 1350 -> 393 per cell, with the limited slopes and the dt / c_h candidates below
// in pairs too (1.27 / 1.21 with renormalised pairs, branches and two subtractions per slope; 1.08 / 1.01 without
// kJump's bounds and with the contact's and the Alfven waves' speeds from unnormalised differences).
// Against the step in 64 bits the error over the Kelvin-Helmholtz, turbulence and smooth states at CFL
// 0.05 and 0.3 is 0.41 to 1.02 times that of the FP64 expressions it replaced (geometric mean 0.79).
#pragma once

#include "fp32pair.cuh"
#include "mhd_defs.cuh"

namespace mhdgb {

// Bounds within which the pairs neither overflow nor lose their low parts: density and sound speed
// in [2^-20, 2^20], velocities and fields below 2^20, the larger tangential field component zero or
// above 2^-83 (pressure and energy follow from density and sound speed; a NaN in them is one in the
// sound speed).  Other faces take the general FP64 flux.
constexpr unsigned kSplitMax = (1023u + 20u) << 20, kSplitMin = (1023u - 20u) << 20, kSplitTinyB = (1023u - 83u) << 20;

// Jumps beyond which the general flux is the more accurate one.  A correction's error is 2^-46 of the wave speed
// times the jump that drives it; the FP64 expressions' are a few 2^-53 of the fluxes' own terms, and 2^-43 (their
// estimate of the fast speed) of what the outer waves carry with S_M.  So the bounds, in units of w:
//   S_M relative to the sides, unless S_M itself is above 1/8 (a moving shock, not a wall),
//   the rotations' velocity jump, times S_M or |B_n| / sqrt(rho*) where these are below 1/4 (without B_n a shear is
//   no rotation's jump),
//   and each field component's part of the magnetic pressure's jump, of rho w^2: the gas pressure may balance it.
// No outer wave comes near the contact then.  Against extended precision the mean error of the flux components
// from given face states is at most 1.15 times the FP64 expressions' (0.2 to 0.9 times for jumps up to 0.1; 1.2 times
// where both only round FP64's last bit) over random states with jumps of 1e-6 to 1, pressure-balanced sheets, shears,
// low beta (1e-3), density ratios up to 2^16, stationary Alfven waves and walls with a normal velocity; from cell
// values, with the slopes' errors in it, 0.1 to 1.05 times.  Without the bounds it is up to 2.7 times for jumps of order
// one, 17 times for strong stationary rotations and 8 to 16 times at walls, whose mass flux is the difference of two
// such terms; from cell values the walls alone are worse than FP64 was.  A warp with such a face forms both fluxes: a
// 24x40x20 state whose walls start with a normal velocity takes 161 us a call instead of 124 (224 with FP64
// expressions alone), decaying turbulence of 128^3 at Mach 0.6 after 200 steps 1.14 ns a cell instead of 1.06 (2.62).
constexpr float kJump = 0.04f;

MHDGB_HD unsigned d_mag(double d) { return d_hi(d) & 0x7FFFFFFFu; }

// Whether the states of a face lie within the bounds.
MHDGB_HD bool face_in_range(const double (&Pl)[NPRIM], const double (&Pr)[NPRIM]) {
  unsigned mb = 0;
#pragma unroll
  for (int n = nbm2; n <= nbm3; n++) mb = u_max(mb, u_max(d_mag(Pl[n]), d_mag(Pr[n])));
  unsigned mx = mb;
  const int q[] = {nve1, nve2, nve3, nbm1, nden, ncsp};
#pragma unroll
  for (int n = 0; n < 6; n++) mx = u_max(mx, u_max(d_mag(Pl[q[n]]), d_mag(Pr[q[n]])));
  // signed comparison: a negative value fails
  const int mn = (int)kSplitMin;
  const bool pos = (int)d_hi(Pl[nden]) >= mn && (int)d_hi(Pr[nden]) >= mn && (int)d_hi(Pl[ncsp]) >= mn &&
                   (int)d_hi(Pr[ncsp]) >= mn;
  return mx < kSplitMax && mb - 1u >= kSplitTinyB - 1u && pos;  // (mb = 0 passes)
}

// Flux through a face from its reconstructed states (rotated: normal component first), HLLD or, with
// hllc, HLLC; returns false where the split does not apply (F is then meaningless).  hchg = c_h / 2, chg2 =
// c_h^2 (the GLM pair, mhd.cpp:1234-1237).  The energy and the scalar are wanted on the upwind side only:
// up(n, left) gives them (their slots of Pl and Pr are not read).
template <class UP>
MHDGB_HD bool face_flux_split(const double (&Pl)[NPRIM], const double (&Pr)[NPRIM], const UP& up, double hchg,
                              double chg2, double (&F)[NCONS], bool hllc) {
  // (checked at the end: a branch here would keep the loads and conversions below from overlapping)
  bool ok = face_in_range(Pl, Pr);
  const Pair rl = p_narrow_nz(Pl[nden]), rr = p_narrow_nz(Pr[nden]);
  const Pair bxl = p_narrow(Pl[nbm1]), bxr = p_narrow(Pr[nbm1]);
  const Pair byl = p_narrow(Pl[nbm2]), byr = p_narrow(Pr[nbm2]);
  const Pair bzl = p_narrow(Pl[nbm3]), bzr = p_narrow(Pr[nbm3]);
  const Pair vxl = p_narrow(Pl[nve1]), vxr = p_narrow(Pr[nve1]);
  const Pair dvx = p_narrow(Pr[nve1] - Pl[nve1]);
  const Pair dby = p_narrow(Pr[nbm2] - Pl[nbm2]), dbz = p_narrow(Pr[nbm3] - Pl[nbm3]);
  const double jb = Pr[nbm1] - Pl[nbm1], hb = d_half(Pl[nbm1] + Pr[nbm1]);
  // (B_n from the FP64 mean: a sum of the sides' pairs may cancel, and its h then has neither sign nor size)
  const Pair dbx = p_narrow(jb), bx = p_narrow(hb), bxs = p_scale(bx, 2.0f);

  // fast speeds: c_f^2 = (a + b + sqrt((a-b)^2 + t (t + 2(a+b)))) / 2 with a = c_s^2, b = B_n^2/rho,
  // t = B_t^2/rho (the discriminant as a sum of squares, without cancellation)
  const Pair bt2l = p_add(p_sqr(byl), p_sqr(bzl)), bt2r = p_add(p_sqr(byr), p_sqr(bzr));
  auto fast2 = [](Pair rho, Pair cs, Pair bn, Pair bt2) {  // c_f^2
    const Pair ri = p_rcp(rho), a = p_sqr(cs), b = p_mul(p_sqr(bn), ri), t = p_mul(bt2, ri);
    const Pair s = p_add(a, b), d = p_norm(p_sub(a, b));
    const Pair disc = p_fma(t, p_add(t, p_scale(s, 2.0f)), p_sqr(d));
    return p_scale(p_add(p_add(s, t), p_sqrt(disc)), 0.5f);
  };
  const Pair cm = p_sqrt(p_max(fast2(rl, p_narrow_nz(Pl[ncsp]), bxl, bt2l), fast2(rr, p_narrow_nz(Pr[ncsp]), bxr, bt2r)));
  const Pair w = p_norm(dvx.h < 0.0f ? p_sub(cm, dvx) : cm);

  // contact speed, and relative to the sides (the results that the largest corrections are proportional
  // to are normalised: that takes a quarter off the error of the mass and energy fluxes)
  float jump_b;
  Pair dp = p_narrow(Pr[npre] - Pl[npre]);
  {
    const Pair b1 = p_mul(dbx, bxs), b2 = p_mul(dby, p_add(byl, byr)), b3 = p_mul(dbz, p_add(bzl, bzr));
    dp = p_add(dp, p_scale(p_add(b3, p_add(b2, b1)), 0.5f));
    jump_b = fmaxf(fabsf(b1.h), fmaxf(fabsf(b2.h), fabsf(b3.h)));
  }
  const Pair ir = p_rcp(p_add(rl, rr)), dpw = p_mul(dp, p_rcp(w));
  // mirror-image states (a reflecting wall) give exactly zero here, and the left side is taken, as
  // in the reference (its fluxes on the two sides of S_M = 0 differ when B_n != 0)
  const Pair sm = p_mul(p_sub(p_fma(rr, vxr, p_mul(rl, vxl)), dpw), ir);
  const bool left = !(f_add(sm.h, sm.l) < 0.0f);
  const Pair dl = p_norm(p_mul(p_norm(p_sub(p_mul(rr, dvx), dpw)), ir));
  // (dr formed as dl is, not as dl - dvx: with the right side much the denser that difference cancels, and
  // mirror-image states would not give mirror-image fluxes)
  const Pair dr = p_norm(p_mul(p_norm(p_neg(p_add(p_mul(rl, dvx), dpw))), ir));

  // upwind side; signs as seen from it (x_: times +1 on the left, -1 on the right)
  const double rho = left ? Pl[nden] : Pr[nden], vx = left ? Pl[nve1] : Pr[nve1], vy = left ? Pl[nve2] : Pr[nve2],
               vz = left ? Pl[nve3] : Pr[nve3], bxu = left ? Pl[nbm1] : Pr[nbm1], by = left ? Pl[nbm2] : Pr[nbm2],
               bz = left ? Pl[nbm3] : Pr[nbm3];
  const double bsq = fma(bz, bz, fma(by, by, bxu * bxu)), vsq = fma(vz, vz, fma(vy, vy, vx * vx));
  const double pu = left ? Pl[npre] : Pr[npre], pt = fma(0.5, bsq, pu), m = rho * vx;
  const double ep = fma(rho, fma(0.5, vsq, up(nene, left)), pu + bsq);  // E + p_T

  const Pair ru = p_sel(left, rl, rr), ro = p_sel(left, rr, rl);
  const Pair byu = p_sel(left, byl, byr), bzu = p_sel(left, bzl, bzr);
  const Pair vyu = p_narrow(vy), vzu = p_narrow(vz);
  const Pair tau = p_neg_if(p_sel(left, dl, dr), !left);
  const Pair wm = p_norm(p_add(w, tau));
  const Pair sms = p_neg_if(sm, !left), vs = p_neg_if(p_sel(left, vxl, vxr), !left), bs = p_neg_if(bx, !left);
  const Pair tauo = p_neg_if(p_sel(left, dr, dl), left);
  const Pair wmo = p_norm(p_add(w, tauo));
  const float d = fmaxf(fabsf(dl.h), fabsf(dr.h));
  ok = ok && (d < kJump * w.h || (fabsf(sm.h) > 0.125f * w.h && d < 0.5f * w.h)) &&
       jump_b < 0.5f * kJump * f_add(rl.h, rr.h) * w.h * w.h;

  const Pair iwm = p_rcp(wm);
  // T = N + rho w tau with N = rho w^2 - B_n^2 in FP64: near B_t = 0 the fast speed is close to the
  // Alfven speed and N cancels, and a star state needs T and N as consistent as FP64 makes them
  // (an error of w itself only moves the outer wave)
  const double wd = p_join(w), w2 = wd * wd, bb = hb * hb;
  const Pair rw = p_mul(ru, w);
  const Pair ti = p_norm(p_mul(tau, iwm));
  Pair r1 = p_norm(p_mul(ru, ti));        // rho - rho*
  Pair f = p_make(0.0f), g, g1;   // v_t* = v_t + f B_t, B_t* = g1 B_t = B_t + g B_t
  bool nondeg = true;
  if (hllc) {
    g = p_neg(ti);
    g1 = p_add(g, p_make(1.0f));
  } else {
    const Pair N = p_narrow(fma(rho, w2, -bb)), rt = p_mul(rw, tau), T = p_norm(p_add(N, rt));
    nondeg = !(fabsf(T.h) < 1.0e-30f);
    const Pair x = nondeg ? p_rcp(T) : p_make(0.0f);
    f = p_neg(p_mul(p_mul(bs, tau), x));
    g = p_neg(p_mul(rt, x));
    g1 = nondeg ? p_mul(N, x) : p_make(1.0f);
    if (!nondeg) r1 = p_make(0.0f);
  }
  const Pair rst = p_norm(p_sub(ru, r1));
  const Pair fby = p_mul(f, byu), fbz = p_mul(f, bzu), gby = p_mul(g, byu), gbz = p_mul(g, bzu);
  // energy: E* - E = -(tau (E + p_T - rho w S_M) - B_n (v*.B* - v.B)) / w_m, signs as seen from the side
  Pair es = p_norm(p_mul(tau, p_norm(p_sub(p_narrow(ep), p_mul(rw, sms)))));
  const Pair byst = p_mul(byu, g1), bzst = p_mul(bzu, g1);
  if (!hllc) {
    Pair q = p_mul(bs, tau);
    q = p_fma(gby, vyu, q);
    q = p_fma(gbz, vzu, q);
    q = p_fma(fby, byst, q);
    q = p_fma(fbz, bzst, q);
    es = p_sub(es, p_mul(bs, q));
    if (!nondeg) es = p_make(0.0f);
  }
  const Pair S = p_norm(p_sub(w, vs));                                             // outer wave's speed away from the side
  const Pair am = p_neg_if(S.h > 0.0f ? S : p_make(0.0f), !left);
  const Pair cr = p_mul(r1, am);                                           // corrections to the fluxes
  Pair ce = p_mul(p_mul(es, iwm), am);
  Pair cy = p_mul(am, fby), cz = p_mul(am, fbz), cby = p_mul(am, gby), cbz = p_mul(am, gbz);
  if (!hllc && !(fabsf(bx.h) < 1.0e-30f)) {
    const Pair r1o = p_mul(ro, p_mul(tauo, p_rcp(wmo)));
    const double rhoo = left ? Pr[nden] : Pl[nden];
    const Pair rto = p_mul(p_mul(ro, w), tauo), To = p_norm(p_add(p_narrow(fma(rhoo, w2, -bb)), rto));
    const bool nondego = !(fabsf(To.h) < 1.0e-30f);
    const Pair xo = nondego ? p_rcp(To) : p_make(0.0f);
    const Pair rsto = nondego ? p_sub(ro, r1o) : ro;
    const Pair fo = p_mul(p_mul(bs, tauo), xo), go = p_neg(p_mul(rto, xo));
    const Pair byo = p_sel(left, byr, byl), bzo = p_sel(left, bzr, bzl);
    float y;
    const Pair q = p_sqrt(rst, &y), qo = p_sqrt(rsto);
    const Pair inv = p_rcp(p_add(q, qo)), iq = p_rcp_from(q, y);
    const bool hn = bs.h < 0.0f;
    const Pair dvy = p_narrow(Pr[nve2] - Pl[nve2]), dvz = p_narrow(Pr[nve3] - Pl[nve3]);
    const Pair jvy = p_sub(p_fma(fo, byo, p_neg_if(dvy, !left)), fby);
    const Pair jvz = p_sub(p_fma(fo, bzo, p_neg_if(dvz, !left)), fbz);
    const Pair jby = p_sub(p_fma(go, byo, p_neg_if(dby, !left)), gby);
    const Pair jbz = p_sub(p_fma(go, bzo, p_neg_if(dbz, !left)), gbz);
    const Pair Dvy = p_mul(p_fma(qo, jvy, p_neg_if(jby, hn)), inv);
    const Pair Dvz = p_mul(p_fma(qo, jvz, p_neg_if(jbz, hn)), inv);
    const Pair hq = p_neg_if(q, hn);
    // E** - E* = h sqrt(rho*) (v**.B** - v*.B*) = h sqrt(rho*) sum Dv (B* + h sqrt(rho*) v**)
    const Pair v2y = p_add(p_add(vyu, fby), Dvy), v2z = p_add(p_add(vzu, fbz), Dvz);
    Pair e2 = p_mul(Dvy, p_fma(hq, v2y, byst));
    e2 = p_fma(Dvz, p_fma(hq, v2z, bzst), e2);
    if (!nondeg) e2 = p_fma(p_sel(left, dl, dr), bx, e2);
    const Pair ab = f_bits(bx.h) >> 31 ? p_neg(bx) : bx;
    const Pair S2 = p_norm(p_sub(p_mul(ab, iq), sms));  // normalised: its sign is that of h
    const float dv = fmaxf(fabsf(Dvy.h), fabsf(Dvz.h)), speed = fmaxf(fabsf(sms.h), ab.h * iq.h);
    ok = ok && dv * fminf(w.h, 4.0f * speed) < kJump * w.h * w.h;
    const Pair a2 = p_neg_if(S2.h > 0.0f ? S2 : p_make(0.0f), !left);
    const Pair ahq = p_mul(a2, hq);
    ce = p_sub(ce, p_mul(ahq, e2));
    cy = p_fma(a2, Dvy, cy);
    cz = p_fma(a2, Dvz, cz);
    cby = p_fma(ahq, Dvy, cby);
    cbz = p_fma(ahq, Dvz, cbz);
  }
  const Pair crx = p_neg_if(p_mul(cr, S), left);                           // (rho* - rho) S, S with its sign
  const Pair cry = p_sub(p_mul(cr, vyu), p_mul(rst, cy)), crz = p_sub(p_mul(cr, vzu), p_mul(rst, cz));

  auto wide = [](Pair c) { return p_join(p_norm(c)); };
  const double fr = m + wide(cr);
  F[mden] = fr;
  F[mrv1] = fma(m, vx, fma(-bxu, bxu, pt + wide(crx)));
  F[mrv2] = fma(m, vy, fma(-by, bxu, wide(cry)));
  F[mrv3] = fma(m, vz, fma(-bz, bxu, wide(crz)));
  F[meto] = fma(ep, vx, fma(-bsq, bxu, wide(ce)));
  F[mbm2] = fma(by, vx, fma(-vy, bxu, wide(p_neg(cby))));
  F[mbm3] = fma(bz, vx, fma(-vz, bxu, wide(p_neg(cbz))));
  F[mst] = fr * up(nst, left);  // the scalar is advected with the mass flux
  F[mbm1] = fma(-hchg, jb, d_half(Pl[nbps] + Pr[nbps]));
  F[mbps] = fma(-hchg, Pr[nbps] - Pl[nbps], hb * chg2);
  return ok;
}

// vanLeer (mhd.cpp:89-95), 2 dp dm / (dp + dm) where the differences have the same sign, from FP64
// differences: both are scaled by one power of two and taken as pairs, so the slope has the pairs'
// relative accuracy (about 2^-45) at any magnitude.  Every step is symmetric in dp and dm: the slopes
// of mirror-image cells are exact mirror images.  ok becomes false for infinities, NaN and
// magnitudes below 2^-700, which take the general expression; there is no branch, so that a thread's
// slopes overlap.
MHDGB_HD double van_leer_split(double dp, double dm, bool& ok) {
  const unsigned hp = d_hi(dp), hm = d_hi(dm), ap = hp & 0x7FFFFFFFu, am = hm & 0x7FFFFFFFu;
  const unsigned top = u_max(ap, am);
  constexpr unsigned lo_lim = (1023u - 700u) << 20, hi_lim = 0x7FF00000u;
  const bool zero = (top | d_lo(dp) | d_lo(dm)) == 0u;  // a uniform stretch: common, and exact
  ok = ok && (zero || top - lo_lim < hi_lim - lo_lim);
  const unsigned base = (top & 0x7FF00000u) - (127u << 20);  // the larger one scaled into [1, 2)
  // opposite signs, or the smaller one below 2^-71 of the larger: no slope
  const bool flat = zero || (int)(hp ^ hm) < 0 || (int)(u_min(ap, am) - base) < (56 << 20);
  auto scaled = [base](unsigned a, unsigned lo) {  // as p_narrow_nz
    const unsigned f = f_shl(a - base, lo, 3);
    return Pair{f_from(f + ((lo >> 28) & 1u)), f_mul(i_to_f((int)(lo << 3)), f_from((f & 0x7F800000u) - (55u << 23)))};
  };
  const Pair x = scaled(ap, d_lo(dp)), y = scaled(am, d_lo(dm));
  const Pair sum = p_norm(p_add(x, y));
  const float p = f_mul(x.h, y.h);
  const float pl = f_add(f_fma(x.h, y.h, -p), f_fma(x.l, y.l, f_add(f_mul(x.h, y.l), f_mul(x.l, y.h))));
  const float y0 = f_rcp_seed(sum.h), r = f_fma(y0, f_fma(-sum.h, y0, 1.0f), y0), q = f_mul(p, r);
  const float ql = f_mul(r, f_fma(-q, sum.l, f_add(f_fma(-q, sum.h, p), pl)));
  const double v = p_join(p_norm(Pair{q, ql}), base - (895u << 20));  // twice the quotient, in the original scale
  return flat ? 0.0 : d_from(d_hi(v) | (hp & 0x80000000u), d_lo(v));
}

// The cell's candidates for dt (ControlTimestep, mhd.cpp:1542-1550: min over d of dx_d / (|v_d| + sqrt(
// c_s^2 + B^2/rho))) and c_h (EvaluateCh, mhd.cpp:1589-1601: max over d of |v_d| + c_f,d), which the
// FP64 form takes at about 2^-43; returns false outside the pairs' range (dt, ch meaningless).
MHDGB_HD bool cell_speeds_split(const double (&p)[NPRIM], double dx, double dy, double dz, double& dt, double& ch) {
  unsigned mx = u_max(d_mag(p[nden]), d_mag(p[ncsp]));
#pragma unroll
  for (int n = 0; n < 3; n++) mx = u_max(mx, u_max(d_mag(p[nve1 + n]), d_mag(p[nbm1 + n])));
  const unsigned smx = u_max(d_mag(dx), u_max(d_mag(dy), d_mag(dz))), smn = u_min(d_mag(dx), u_min(d_mag(dy), d_mag(dz)));
  const bool ok = mx < kSplitMax && (int)d_hi(p[nden]) >= (int)kSplitMin && (int)d_hi(p[ncsp]) >= (int)kSplitMin &&
                  smx < kSplitMax && smn >= (1023u - 40u) << 20;
  const Pair ri = p_rcp(p_narrow_nz(p[nden])), a = p_sqr(p_narrow_nz(p[ncsp]));
  const Pair b1 = p_mul(p_sqr(p_narrow(p[nbm1])), ri), b2 = p_mul(p_sqr(p_narrow(p[nbm2])), ri),
             b3 = p_mul(p_sqr(p_narrow(p[nbm3])), ri);
  const Pair b12 = p_add(b1, b2), cts = p_add(p_add(a, b12), b3), ct = p_sqrt(cts);
  auto mag = [](double v) { return p_narrow(d_from(d_mag(v), d_lo(v))); };
  const Pair v1 = mag(p[nve1]), v2 = mag(p[nve2]), v3 = mag(p[nve3]);
  auto time = [ct](double d, Pair v) { return p_mul(p_narrow_nz(d), p_rcp(p_add(v, ct))); };
  const Pair t = p_min(p_min(time(dx, v1), time(dy, v2)), time(dz, v3));
  auto signal = [&](Pair bn, Pair bt, Pair v) {  // |v| + c_f, the discriminant as in face_flux_split
    const Pair s = p_add(a, bn), d = p_norm(p_sub(a, bn));
    const Pair disc = p_fma(bt, p_add(bt, p_scale(s, 2.0f)), p_sqr(d));
    return p_add(v, p_sqrt(p_scale(p_add(cts, p_sqrt(disc)), 0.5f)));
  };
  const Pair c = p_max(p_max(signal(b1, p_add(b2, b3), v1), signal(b2, p_add(b1, b3), v2)), signal(b3, b12, v3));
  dt = p_join(p_norm(t));
  ch = p_join(p_norm(c));
  return ok;
}

}  // namespace mhdgb
