// chasqui_b200 — ideal-MHD Riemann solvers on one face, evaluated entirely in registers.
//
// States are in the face frame: u normal velocity, (v, w) transverse velocities, bn the
// face-normal field, (by, bz) transverse fields; magnetic pressure B^2/2.
//   HLLE  : Einfeldt (1988)                       (src/riemann.hpp:55-68)
//   HLLD  : Miyoshi & Kusano, JCP 208, 315 (2005)  (src/riemann.hpp:96-234)
//   LHLLD : HLLD with the shock-stability / low-dissipation factors and signal speeds of
//           Minoshima & Miyoshi (2021), star fluxes from the star states.
// The left and right halves are exact mirror copies and multi-term sums are grouped in
// mirror-image pairs, as in the reference, so that reflected inputs give bitwise-reflected
// fluxes (the reference's symmetry_test contract). Flux slots follow the reference:
// 0 mass, 1 normal momentum, 2/3 transverse momenta, 4 energy, 5/6 transverse fields.
#pragma once
#include "chq_common.cuh"
#include "chq_quot.cuh"

namespace chq {

enum : int { FD = 0, FMU = 1, FMV = 2, FMW = 3, FEN = 4, FBY = 5, FBZ = 6, NFLX = 7 };

template <class T> struct MState { T d, u, v, w, p, by, bz; };

// fast magnetosonic speed (src/riemann.hpp:19-25)
template <class T> CHQ_HD T fast_speed(const MState<T> &s, T bn, T gamma) {
  const T bsq = bn * bn + s.by * s.by + s.bz * s.bz;
  const T gp = gamma * s.p;
  const T a = (gp + bsq) / s.d;
  const T disc = a * a - divz(T(4) * gp * bn * bn, s.d * s.d);
  return sqrt_(T(0.5) * (a + sqrt_(fmax_(disc, T(0)))));
}

// physical flux, total energy and total pressure of a state (src/riemann.hpp:27-40)
template <class T> CHQ_HD void phys_flux(const MState<T> &s, T bn, T gm1, T &e, T &pt, T f[NFLX]) {
  const T vsq = s.u * s.u + s.v * s.v + s.w * s.w;
  const T bsq = bn * bn + s.by * s.by + s.bz * s.bz;
  e = s.p / gm1 + T(0.5) * (s.d * vsq + bsq);
  pt = s.p + T(0.5) * bsq;
  const T vdotb = s.u * bn + s.v * s.by + s.w * s.bz;
  f[FD] = s.d * s.u;
  f[FMU] = s.d * s.u * s.u + pt - bn * bn;
  f[FMV] = s.d * s.u * s.v - bn * s.by;
  f[FMW] = s.d * s.u * s.w - bn * s.bz;
  f[FEN] = (e + pt) * s.u - bn * vdotb;
  f[FBY] = s.by * s.u - bn * s.v;
  f[FBZ] = s.bz * s.u - bn * s.w;
}

// total energy and total pressure alone (the scalars phys_flux computes first)
template <class T> CHQ_HD void energy_ptot(const MState<T> &s, T bn, T gm1, T &e, T &pt) {
  const T vsq = s.u * s.u + s.v * s.v + s.w * s.w;
  const T bsq = bn * bn + s.by * s.by + s.bz * s.bz;
  e = s.p / gm1 + T(0.5) * (s.d * vsq + bsq);
  pt = s.p + T(0.5) * bsq;
}

// the flux vector of phys_flux from already computed e and pt
template <class T> CHQ_HD void flux_from(const MState<T> &s, T bn, T e, T pt, T f[NFLX]) {
  const T vdotb = s.u * bn + s.v * s.by + s.w * s.bz;
  f[FD] = s.d * s.u;
  f[FMU] = s.d * s.u * s.u + pt - bn * bn;
  f[FMV] = s.d * s.u * s.v - bn * s.by;
  f[FMW] = s.d * s.u * s.w - bn * s.bz;
  f[FEN] = (e + pt) * s.u - bn * vdotb;
  f[FBY] = s.by * s.u - bn * s.v;
  f[FBZ] = s.bz * s.u - bn * s.w;
}

// modified fast speed with the sound speed replaced by |v| (src/riemann.hpp:44-51)
template <class T> CHQ_HD T flow_speed_u(const MState<T> &s, T bn) {
  const T vsq = s.u * s.u + s.v * s.v + s.w * s.w;
  const T casq = divz(bn * bn + s.by * s.by + s.bz * s.bz, s.d);
  const T caxsq = divz(bn * bn, s.d);
  const T a = casq + vsq;
  const T disc = a * a - T(4) * vsq * caxsq;
  return sqrt_(T(0.5) * (a + sqrt_(fmax_(disc, T(0)))));
}

template <class T> CHQ_HD void hlle(const MState<T> &L, const MState<T> &R, T bn, T gamma, T gm1, T f[NFLX]) {
  // speeds first; the flux vectors are built only for the region that is selected
  const T cl = fast_speed(L, bn, gamma), cr = fast_speed(R, bn, gamma);
  const T sl = fmin_(L.u - cl, R.u - cr);
  const T sr = fmax_(L.u + cl, R.u + cr);
  T el, er, ptl, ptr;
  energy_ptot(L, bn, gm1, el, ptl);
  if (sl >= T(0)) {
    flux_from(L, bn, el, ptl, f);
    return;
  }
  energy_ptot(R, bn, gm1, er, ptr);
  if (sr <= T(0)) {
    flux_from(R, bn, er, ptr, f);
    return;
  }
  T fl[NFLX], fr[NFLX];
  flux_from(L, bn, el, ptl, fl);
  flux_from(R, bn, er, ptr, fr);
  const T ul[NFLX] = {L.d, L.d * L.u, L.d * L.v, L.d * L.w, el, L.by, L.bz};
  const T ur[NFLX] = {R.d, R.d * R.u, R.d * R.v, R.d * R.w, er, R.by, R.bz};
  const T inv = T(1) / (sr - sl);
#pragma unroll
  for (int n = 0; n < NFLX; ++n) f[n] = (sr * fl[n] - sl * fr[n] + sl * sr * (ur[n] - ul[n])) * inv;
}

// flux of an intermediate state with intermediate total pressure pts (src/riemann.hpp:81-91)
template <class T>
CHQ_HD void star_flux(T d, T sm, T v, T w, T e, T by, T bz, T bn, T pts, T f[NFLX]) {
  const T vdotb = (sm * bn + v * by) + w * bz;
  f[FD] = d * sm;
  f[FMU] = (d * sm) * sm + (pts - bn * bn);
  f[FMV] = (d * sm) * v - bn * by;
  f[FMW] = (d * sm) * w - bn * bz;
  f[FEN] = (e + pts) * sm - bn * vdotb;
  f[FBY] = by * sm - bn * v;
  f[FBZ] = bz * sm - bn * w;
}

// One side's single-star transverse velocity and field (MK05 eqs. 43-47); the left and
// right calls run the identical expression sequence.
template <class T>
CHQ_HD void star_side(const MState<T> &S, T slm, T sms, T sm, T bn, T bnsq, T &vs, T &ws, T &bys, T &bzs) {
  const T den = (S.d * slm) * sms - bnsq;
  const T scale = fabs_((S.d * slm) * sms) + bnsq;
  if (fabs_(den) <= T(1e-12) * scale + Tiny<T>::v) {
    vs = S.v;
    ws = S.w;
    bys = S.by;
    bzs = S.bz;
  } else {
    const T num_v = divz(bn * (sm - S.u), den);
    vs = S.v - S.by * num_v;
    ws = S.w - S.bz * num_v;
    const T num_b = ((S.d * slm) * slm - bnsq) / den;
    bys = S.by * num_b;
    bzs = S.bz * num_b;
  }
}

// single-star flux of one side: F + S (U* - U) (HLLD) or the star state's own flux (LHLLD)
template <bool LHLLD, class T>
CHQ_HD void side_star_flux(const MState<T> &S, T bn, T e, T pt, T s, T ds, T sm, T vs, T ws, T bys, T bzs, T es,
                           T pts, T f[NFLX]) {
  if constexpr (LHLLD) {
    star_flux(ds, sm, vs, ws, es, bys, bzs, bn, pts, f);
  } else {
    T fs[NFLX];
    flux_from(S, bn, e, pt, fs);
    const T us[NFLX] = {ds, ds * sm, ds * vs, ds * ws, es, bys, bzs};
    const T u[NFLX] = {S.d, S.d * S.u, S.d * S.v, S.d * S.w, e, S.by, S.bz};
#pragma unroll
    for (int n = 0; n < NFLX; ++n) f[n] = fs[n] + s * (us[n] - u[n]);
  }
}

// double-star flux of one side: F* + S* (U** - U*) (HLLD) or the ** state's own flux (LHLLD)
template <bool LHLLD, class T>
CHQ_HD void side_dstar_flux(const MState<T> &S, T bn, T e, T pt, T s, T ds, T sm, T vs, T ws, T bys, T bzs, T es,
                            T pts, T ss, T vss, T wss, T byss, T bzss, T ess, T f[NFLX]) {
  if constexpr (LHLLD) {
    star_flux(ds, sm, vss, wss, ess, byss, bzss, bn, pts, f);
  } else {
    T fs[NFLX];
    side_star_flux<false>(S, bn, e, pt, s, ds, sm, vs, ws, bys, bzs, es, pts, fs);
    const T us[NFLX] = {ds, ds * sm, ds * vs, ds * ws, es, bys, bzs};
    const T uss[NFLX] = {ds, ds * sm, ds * vss, ds * wss, ess, byss, bzss};
#pragma unroll
    for (int n = 0; n < NFLX; ++n) f[n] = fs[n] + ss * (uss[n] - us[n]);
  }
}

// Single-star (single) or double-star flux of the side `left` selects. The operands of the
// two sides are picked value by value, then one evaluation runs with exactly the expression
// sequence of side_star_flux / side_dstar_flux, so the result is bitwise the flux of that
// side. The left side's double-star energy is E*_L - sqrt(D*_L) (v*_L.B*_L - v**.B**) sgn(bn),
// the right side's E*_R + (the mirror term); x - t and x + (-t) are the same IEEE operation.
template <bool LHLLD, class T>
CHQ_HD void side_region_flux(bool left, bool single, const MState<T> &L, const MState<T> &R, T bn, T el, T er, T ptl,
                             T ptr, T sl, T sr, T dls, T drs, T sm, T vls, T vrs, T wls, T wrs, T byls, T byrs, T bzls,
                             T bzrs, T els, T ers, T pts, T sls, T srs, T sqdl, T sqdr, T vdotb_ls, T vdotb_rs, T sg,
                             T vss, T wss, T byss, T bzss, T vdotb_ss, T f[NFLX]) {
  const T ds = left ? dls : drs, vs = left ? vls : vrs, ws = left ? wls : wrs;
  const T bys = left ? byls : byrs, bzs = left ? bzls : bzrs, es = left ? els : ers;
  if constexpr (LHLLD) {
    if (single) {
      star_flux(ds, sm, vs, ws, es, bys, bzs, bn, pts, f);
    } else {
      const T t = (left ? sqdl : sqdr) * (((left ? vdotb_ls : vdotb_rs) - vdotb_ss) * sg);
      const T ess = es + (left ? -t : t);
      star_flux(ds, sm, vss, wss, ess, byss, bzss, bn, pts, f);
    }
  } else {
    const MState<T> S{left ? L.d : R.d, left ? L.u : R.u, left ? L.v : R.v, left ? L.w : R.w,
                      left ? L.p : R.p, left ? L.by : R.by, left ? L.bz : R.bz};
    const T e = left ? el : er, pt = left ? ptl : ptr, s = left ? sl : sr;
    side_star_flux<false>(S, bn, e, pt, s, ds, sm, vs, ws, bys, bzs, es, pts, f);
    if (!single) {
      const T t = (left ? sqdl : sqdr) * (((left ? vdotb_ls : vdotb_rs) - vdotb_ss) * sg);
      const T ess = es + (left ? -t : t);
      const T ss = left ? sls : srs;
      const T us[NFLX] = {ds, ds * sm, ds * vs, ds * ws, es, bys, bzs};
      const T uss[NFLX] = {ds, ds * sm, ds * vss, ds * wss, ess, byss, bzss};
#pragma unroll
      for (int n = 0; n < NFLX; ++n) f[n] = f[n] + ss * (uss[n] - us[n]);
    }
  }
}

template <bool LHLLD, class T>
CHQ_HD void hlld(const MState<T> &L, const MState<T> &R, T bn, T gamma, T gm1, T f[NFLX], T theta, T phi) {
  // speeds and the scalars of both sides first; flux vectors only for the selected region
  T el, er, ptl, ptr;
  energy_ptot(L, bn, gm1, el, ptl);
  energy_ptot(R, bn, gm1, er, ptr);
  const T cl = fast_speed(L, bn, gamma), cr = fast_speed(R, bn, gamma);
  T sl, sr;
  if constexpr (LHLLD) {
    const T cmax = fmax_(cl, cr);
    sl = fmin_(T(0), fmin_(L.u, R.u) - cmax);
    sr = fmax_(T(0), fmax_(L.u, R.u) + cmax);
  } else {
    sl = fmin_(L.u - cl, R.u - cr);
    sr = fmax_(L.u + cl, R.u + cr);
  }
  if (sl >= T(0)) {
    flux_from(L, bn, el, ptl, f);
    return;
  }
  if (sr <= T(0)) {
    flux_from(R, bn, er, ptr, f);
    return;
  }
  const T bnsq = bn * bn;
  const T slml = sl - L.u;
  const T srmr = sr - R.u;
  const T dsl = L.d * slml;
  const T dsr = R.d * srmr;
  const T iden = T(1) / (dsr - dsl);
  // contact speed and star total pressure (MK05 eqs. 38, 41)
  const T sm = ((dsr * R.u - dsl * L.u) + theta * (ptl - ptr)) * iden;
  const T pts = ((dsr * ptl - dsl * ptr) + (phi * ((L.d * R.d) * (srmr * slml))) * (R.u - L.u)) * iden;

  const T slms = sl - sm;
  const T dls = dsl / slms;
  T vls, wls, byls, bzls;
  star_side(L, slml, slms, sm, bn, bnsq, vls, wls, byls, bzls);
  const T vdotb_l = (L.u * bn + L.v * L.by) + L.w * L.bz;
  const T vdotb_ls = (sm * bn + vls * byls) + wls * bzls;
  const T els = (((slml * el - ptl * L.u) + pts * sm) + bn * (vdotb_l - vdotb_ls)) / slms;

  const T srms = sr - sm;
  const T drs = dsr / srms;
  T vrs, wrs, byrs, bzrs;
  star_side(R, srmr, srms, sm, bn, bnsq, vrs, wrs, byrs, bzrs);
  const T vdotb_r = (R.u * bn + R.v * R.by) + R.w * R.bz;
  const T vdotb_rs = (sm * bn + vrs * byrs) + wrs * bzrs;
  const T ers = (((srmr * er - ptr * R.u) + pts * sm) + bn * (vdotb_r - vdotb_rs)) / srms;

  // Alfven waves bounding the double-star region (MK05 eq. 51)
  const T sqdl = sqrt_(dls), sqdr = sqrt_(drs);
  const T abn = fabs_(bn);
  const T sls = sm - divz(abn, sqdl);
  const T srs = sm + divz(abn, sqdr);

  // Region of the face (strict inequalities: with S*_L = S*_R = 0 both sides are averaged):
  //   S*_L > 0           single-star flux of the left side
  //   S*_R < 0           single-star flux of the right side
  //   bn ~ 0             the double-star region collapses onto the contact: single-star flux
  //                      of the side the contact moves away from
  //   otherwise          double-star flux of that side
  // and both sides averaged when the contact speed is exactly zero (or not a number). The
  // side's operands are selected first and its flux is evaluated once, so the lanes of a
  // warp whose contacts move either way run one flux evaluation instead of one per side.
  const T bnsmall = T(1e-12) * (ptl + ptr);
  const bool star_l = sls > T(0);
  const bool star_r = !star_l && (srs < T(0));
  const bool single = star_l || star_r || (bnsq <= bnsmall);
  const bool pos = sm > T(0), neg = sm < T(0);
  const bool both = !star_l && !star_r && !pos && !neg;
  const bool left = star_l || (!star_r && (pos || both));
  // double-star states (MK05 eqs. 59-63)
  T sg = T(0), vss = T(0), wss = T(0), byss = T(0), bzss = T(0), vdotb_ss = T(0);
  if (!single) {
    sg = sgn(bn);
    const T inv = T(1) / (sqdl + sqdr);
    vss = ((sqdl * vls + sqdr * vrs) + (byrs - byls) * sg) * inv;
    wss = ((sqdl * wls + sqdr * wrs) + (bzrs - bzls) * sg) * inv;
    byss = ((sqdl * byrs + sqdr * byls) + (sqdl * sqdr) * ((vrs - vls) * sg)) * inv;
    bzss = ((sqdl * bzrs + sqdr * bzls) + (sqdl * sqdr) * ((wrs - wls) * sg)) * inv;
    vdotb_ss = (sm * bn + vss * byss) + wss * bzss;
  }
  side_region_flux<LHLLD>(left, single, L, R, bn, el, er, ptl, ptr, sl, sr, dls, drs, sm, vls, vrs, wls, wrs, byls,
                          byrs, bzls, bzrs, els, ers, pts, sls, srs, sqdl, sqdr, vdotb_ls, vdotb_rs, sg, vss, wss,
                          byss, bzss, vdotb_ss, f);
  if (both) {
    T fb[NFLX];
    side_region_flux<LHLLD>(false, single, L, R, bn, el, er, ptl, ptr, sl, sr, dls, drs, sm, vls, vrs, wls, wrs,
                            byls, byrs, bzls, bzrs, els, ers, pts, sls, srs, sqdl, sqdr, vdotb_ls, vdotb_rs, sg, vss,
                            wss, byss, bzss, vdotb_ss, fb);
#pragma unroll
    for (int n = 0; n < NFLX; ++n) f[n] = T(0.5) * (f[n] + fb[n]);
  }
}

// ---------------------------------------------------------------------------------------
// The face solver of the flux kernel: hlld with the quotients of chq_quot.cuh. Bound by FP64
// issue, so it evaluates only what the selected side needs: both sides' speeds and star
// states, then the energies and the flux of one side. Every rounded operation has hlld's
// operands, so the fluxes are the same; `ok` turns false when a divisor leaves the range the
// quotients are exact in, or a numerator overflows (vacuum, non-finite states, a degenerate negative star denominator),
// and the caller then evaluates hlld itself.

// fast magnetosonic speed (fast_speed) from bsq = B^2
template <class T> CHQ_D T fast_speed_q(const MState<T> &s, T bn, T bsq, T gamma, bool &ok) {
  const T gp = gamma * s.p;
  const T yd = rcp_n(s.d);
  const T a = quot(gp + bsq, s.d, yd);
  const T dd = s.d * s.d;
  const T disc = fma_(T(-4), quot(gp * bn * bn, dd, yd * yd), a * a);   // the scaling by 4 is exact
  const T root = sqrt_q(disc);
  ok = ok && in_range(s.d) && in_range(a);
  return sqrt_q(T(0.5) * (a + (disc > RootFloor<T>::v ? root : T(0))));
}

// modified fast speed of LHLLD (flow_speed_u)
template <class T> CHQ_D T flow_speed_q(const MState<T> &s, T bn, bool &ok) {
  const T vsq = s.u * s.u + s.v * s.v + s.w * s.w;
  const T yd = rcp_n(s.d);
  const T casq = quot(bn * bn + s.by * s.by + s.bz * s.bz, s.d, yd);
  const T caxsq = quot(bn * bn, s.d, yd);
  const T a = casq + vsq;
  const T disc = a * a - T(4) * vsq * caxsq;
  const T root = sqrt_q(disc);
  const T h = T(0.5) * (a + (disc > RootFloor<T>::v ? root : T(0)));
  const T r = sqrt_q(h);
  ok = ok && a < QuotMax<T>::v;   // (false for a NaN)
  return (h <= RootFloor<T>::v) ? T(0) : r;
}

// single-star transverse velocity and field of one side (star_side); dm = rho (S - u), sms = S - S_M
template <class T>
CHQ_D void star_side_q(const MState<T> &S, T dm, T slm, T sms, T sm, T bn, T bnsq, T &vs, T &ws, T &bys, T &bzs,
                       bool &ok) {
  const T t = dm * sms;
  const T den = t - bnsq;
  // (star_side's tiny addend counts only where the products vanish, out of the quotients' range)
  const bool deg = fabs_(den) <= T(1e-12) * (fabs_(t) + bnsq);
  const T y = rcp_n(den);
  const T nv = quot(bn * (sm - S.u), den, y);
  const T nb = quot(dm * slm - bnsq, den, y);
  vs = deg ? S.v : S.v - S.by * nv;
  ws = deg ? S.w : S.w - S.bz * nv;
  bys = deg ? S.by : S.by * nb;
  bzs = deg ? S.bz : S.bz * nb;
  ok = ok && (deg || in_range(den));
}

// total energy (energy_ptot) with the quotient by gamma - 1 taken from its rounded reciprocal
template <class T> CHQ_D T energy_q(const MState<T> &s, T bsq, T gm1, T rgm1) {
  const T vsq = s.u * s.u + s.v * s.v + s.w * s.w;
  return fma_(T(0.5), s.d * vsq + bsq, quot(s.p, gm1, rgm1));
}

// One side of a star region: the side's state S with its pressure, wave speed s, S - u (slm),
// star density, star transverse state, |S - S_M| (n) and its reciprocal (y), and what its
// double-star state adds (ss: the Alfven speed, sqd: sqrt of the star density).
template <class T> struct StarSide {
  MState<T> S;
  T bsq, pt, s, slm, n, y, ds, vs, ws, bys, bzs, sqd, ss;
};

// single-star (single) or double-star flux of the side
template <bool LHLLD, class T>
CHQ_D void star_region_flux(const StarSide<T> &Q, bool left, bool single, T bn, T gm1, T rgm1, T sm, T pts, T vss, T wss,
                            T byss, T bzss, T f[NFLX]) {
  const MState<T> &S = Q.S;
  const T e = energy_q(S, Q.bsq, gm1, rgm1);
  const T vdotb = (S.u * bn + S.v * S.by) + S.w * S.bz;
  const T vdotb_s = (sm * bn + Q.vs * Q.bys) + Q.ws * Q.bzs;
  const T num = ((Q.slm * e - Q.pt * S.u) + pts * sm) + bn * (vdotb - vdotb_s);
  const T es = quot(left ? -num : num, Q.n, Q.y);
  const T vdotb_ss = (sm * bn + vss * byss) + wss * bzss;
  const T t = Q.sqd * flip_sign(vdotb_s - vdotb_ss, bn);
  const T ess = es + (left ? -t : t);
  if constexpr (LHLLD) {
    star_flux(Q.ds, sm, single ? Q.vs : vss, single ? Q.ws : wss, single ? es : ess, single ? Q.bys : byss,
              single ? Q.bzs : bzss, bn, pts, f);
  } else {
    flux_from(S, bn, e, Q.pt, f);
    const T us[NFLX] = {Q.ds, Q.ds * sm, Q.ds * Q.vs, Q.ds * Q.ws, es, Q.bys, Q.bzs};
    const T u[NFLX] = {S.d, S.d * S.u, S.d * S.v, S.d * S.w, e, S.by, S.bz};
#pragma unroll
    for (int n = 0; n < NFLX; ++n) f[n] = f[n] + Q.s * (us[n] - u[n]);
    if (!single) {
      // the double star keeps the star density and normal momentum: those differences are zero
      const T uss[NFLX] = {Q.ds, Q.ds * sm, Q.ds * vss, Q.ds * wss, ess, byss, bzss};
#pragma unroll
      for (int n = FMV; n < NFLX; ++n) f[n] = f[n] + Q.ss * (uss[n] - us[n]);
    }
  }
}

// cl, cr: the sides' fast speeds; bsql, bsqr: their B^2; rgm1 = RN(1 / gm1)
template <bool LHLLD, class T>
CHQ_D bool hlld_q(const MState<T> &L, const MState<T> &R, T bn, T gm1, T rgm1, T bsql, T bsqr, T cl, T cr, T theta,
                  T phi, T f[NFLX]) {
  const T bnsq = bn * bn;
  const T ptl = fma_(T(0.5), bsql, L.p), ptr = fma_(T(0.5), bsqr, R.p);
  T sl, sr;
  if constexpr (LHLLD) {
    const T cmax = (cl > cr) ? cl : cr;
    const T ul = ((L.u < R.u) ? L.u : R.u) - cmax, ur = ((L.u > R.u) ? L.u : R.u) + cmax;
    sl = (ul < T(0)) ? ul : T(0);
    sr = (ur > T(0)) ? ur : T(0);
  } else {
    const T a = L.u - cl, b = R.u - cr, c = L.u + cl, d = R.u + cr;
    sl = (a < b) ? a : b;
    sr = (c > d) ? c : d;
  }
  if (sl >= T(0) || sr <= T(0)) {
    const bool left = sl >= T(0);
    const MState<T> S{left ? L.d : R.d, left ? L.u : R.u, left ? L.v : R.v, left ? L.w : R.w,
                      left ? L.p : R.p, left ? L.by : R.by, left ? L.bz : R.bz};
    flux_from(S, bn, energy_q(S, left ? bsql : bsqr, gm1, rgm1), left ? ptl : ptr, f);
    return true;
  }
  const T slml = sl - L.u, srmr = sr - R.u;
  const T dsl = L.d * slml, dsr = R.d * srmr;
  const T dds = dsr - dsl;
  const T iden = rcp_rn(dds);
  const T sm = ((dsr * R.u - dsl * L.u) + theta * (ptl - ptr)) * iden;
  const T pts = ((dsr * ptl - dsl * ptr) + (phi * ((L.d * R.d) * (srmr * slml))) * (R.u - L.u)) * iden;
  // left divisors negated (S_M - S_L > 0), which negates the numerators: the same quotients
  const T nl = sm - sl, nr = sr - sm;
  const T yl = rcp_n(nl), yr = rcp_n(nr);
  const T dls = quot(-dsl, nl, yl), drs = quot(dsr, nr, yr);
  bool ok = in_range(dds) && in_range(nl) && in_range(nr) && in_range(dls) && in_range(drs);
  T yql, yqr;
  const T sqdl = sqrt_q(dls, yql), sqdr = sqrt_q(drs, yqr);
  const T abn = fabs_(bn);
  const T sls = sm - quot(abn, sqdl, rcp_root(sqdl, yql));
  const T srs = sm + quot(abn, sqdr, rcp_root(sqdr, yqr));
  // region and side as in hlld
  const bool star_l = sls > T(0);
  const bool star_r = !star_l && (srs < T(0));
  const bool single = star_l || star_r || (bnsq <= T(1e-12) * (ptl + ptr));
  const bool pos = sm > T(0), neg = sm < T(0);
  const bool both = !star_l && !star_r && !pos && !neg;
  const bool left = star_l || (!star_r && (pos || both));
  T vls, wls, byls, bzls, vrs, wrs, byrs, bzrs;
  star_side_q(L, dsl, slml, -nl, sm, bn, bnsq, vls, wls, byls, bzls, ok);
  star_side_q(R, dsr, srmr, nr, sm, bn, bnsq, vrs, wrs, byrs, bzrs, ok);
  T vss = T(0), wss = T(0), byss = T(0), bzss = T(0);
  if (!single) {
    const T inv = rcp_rn(sqdl + sqdr);
    vss = ((sqdl * vls + sqdr * vrs) + flip_sign(byrs - byls, bn)) * inv;
    wss = ((sqdl * wls + sqdr * wrs) + flip_sign(bzrs - bzls, bn)) * inv;
    byss = ((sqdl * byrs + sqdr * byls) + (sqdl * sqdr) * flip_sign(vrs - vls, bn)) * inv;
    bzss = ((sqdl * bzrs + sqdr * bzls) + (sqdl * sqdr) * flip_sign(wrs - wls, bn)) * inv;
  }
  // a contact that stands exactly still (gas at rest): the mean of both sides' fluxes; the
  // right side's is evaluated here, where its operands are still at hand
  T f0[NFLX];
#pragma unroll
  for (int n = 0; n < NFLX; ++n) f0[n] = T(0);
  if (both) {
    const StarSide<T> Q{R, bsqr, ptr, sr, srmr, nr, yr, drs, vrs, wrs, byrs, bzrs, sqdr, srs};
    star_region_flux<LHLLD>(Q, false, single, bn, gm1, rgm1, sm, pts, vss, wss, byss, bzss, f0);
  }
  const StarSide<T> Q{{left ? L.d : R.d, left ? L.u : R.u, left ? L.v : R.v, left ? L.w : R.w,
                       left ? L.p : R.p, left ? L.by : R.by, left ? L.bz : R.bz},
                      left ? bsql : bsqr, left ? ptl : ptr, left ? sl : sr, left ? slml : srmr, left ? nl : nr,
                      left ? yl : yr, left ? dls : drs, left ? vls : vrs, left ? wls : wrs, left ? byls : byrs,
                      left ? bzls : bzrs, left ? sqdl : sqdr, left ? sls : srs};
  star_region_flux<LHLLD>(Q, left, single, bn, gm1, rgm1, sm, pts, vss, wss, byss, bzss, f);
  if (both) {
#pragma unroll
    for (int n = 0; n < NFLX; ++n) f[n] = T(0.5) * (f[n] + f0[n]);
  }
  // a quotient of a numerator that overflowed is NaN, and so is then the energy flux
  return ok && finite_q(f[FEN]);
}

}  // namespace chq
