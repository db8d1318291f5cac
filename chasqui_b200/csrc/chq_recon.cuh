// chasqui_b200 — reconstruction in per-cell form.
//
// The reference reconstructs per FACE from a 6-cell stencil (src/recon.hpp:1-7), so every
// cell's limited parabola is evaluated twice (once for each of its faces). Here each cell c
// produces its own pair (aL, aR) = (value at its left face, value at its right face) from the
// 5 cells q5[0..4] = q_{c-2..c+2}; face i then takes ql = aR_{i-1}, qr = aL_i. Every
// expression is evaluated with the same operands in the same order as the reference's
// per-face form, so both give bitwise-identical face states (this is checked against the
// reference library in the tests). The mirror-symmetric grouping of sums is part of the
// parity contract and is kept as published (Fleischmann, Adami & Adams 2019).
#pragma once
#include "chq_common.cuh"
#include "chq_quot.cuh"

namespace chq {

// van Leer harmonic slope (src/recon.hpp:14-18); dl and dr have one sign where it is not zero
template <class T> CHQ_D T vl_slope(T qm, T q0, T qp) {
  const T dl = q0 - qm, dr = qp - q0;
  const T d2 = dl * dr, s = dl + dr;
  return (d2 > T(0)) ? flip_sign(quot_pos(T(2) * d2, fabs_(s)), s) : T(0);
}

// The pieces below are written without branches: a warp's cells differ in which limiter
// applies, and a branch costs its lanes both sides. Scaling by a power of two is exact, so
// factors of 2, 1/2 and 1/4 are moved to where they cost nothing; every rounded operation has
// the published operands. In FP32 a product and the sum it enters round once (mad), also where
// the product is shared: with 3 q and 11 q, 5 q, 3 q of WENO-Z rounded first, the error of the
// FP32 face fluxes against FP64 was 1 to 7 % (PPM) and up to 0.6 % (WENO-Z) larger on smooth states.

// twice the monotonised central slope, CW84 eq. 1.8 (src/recon.hpp:21-27):
// sgn(dc) min(|dc|, 2 min(|dl|, |dr|)) with dc = (qp - qm)/2, zero at an extremum
template <class T> CHQ_HD T mc_slope2(T qm, T q0, T qp) {
  const T dl = q0 - qm, dr = qp - q0, d2 = qp - qm;
  const T al = fabs_(dl), ar = fabs_(dr), a2 = fabs_(d2);
  const T lim = T(4) * ((al < ar) ? al : ar);
  const T m = flip_sign((a2 < lim) ? a2 : lim, d2);
  return (dl * dr > T(0)) ? m : T(0);
}

// CW84 interface value between cells a and b (src/recon.hpp:42-44) from their doubled slopes:
// (qa + qb)/2 + (sa - sb)/6
template <class T> CHQ_HD T ppm_face2(T qa, T qb, T sa2, T sb2) {
  return fma_(T(0.5), qa + qb, twelfth(sa2 - sb2));
}

// CW84 parabola monotonisation of one cell (src/recon.hpp:47-57)
template <class T> CHQ_HD void ppm_limit(T q, T &qL, T &qR) {
  const T l = qL, r = qR;
  const bool flat = (r - q) * (q - l) <= T(0);
  const T d = r - l;
  const T c = fma_(T(-0.5), l + r, q);
  const T t = sixth(d * d), dc = d * c;
  const T nl = (dc > t) ? mad(T(3), q, T(-2) * r) : l;
  const T nr = (dc < -t) ? mad(T(3), q, T(-2) * l) : r;
  qL = flat ? q : nl;
  qR = flat ? q : nr;
}

// extremum-preserving 4th-order interface between q0 and qp1 (src/recon.hpp:85-100)
template <class T> CHQ_HD T ppmx_face(T qm1, T q0, T qp1, T qp2) {
  const T s = q0 + qp1;
  const T qf = (T(7) / T(12)) * s - (T(1) / T(12)) * (qm1 + qp2);
  const T d2 = T(3) * fma_(T(-2), qf, s);
  const T d2l = fma_(T(-2), q0, qm1 + qp1);
  const T d2r = fma_(T(-2), qp1, q0 + qp2);
  const T al = fabs_(d2l), ar = fabs_(d2r), a2 = fabs_(d2);
  const T lim = T(1.25) * ((al < ar) ? al : ar);
  const T m = flip_sign((lim < a2) ? lim : a2, d2);
  const T d2lim = (d2 * d2l > T(0) && d2 * d2r > T(0)) ? m : T(0);
  const T lin = fma_(T(0.5), s, -sixth(d2lim));
  return ((qf - q0) * (qp1 - qf) < T(0)) ? lin : qf;
}

// extremum-preserving limiter of one cell's parabola (src/recon.hpp:104-127)
template <class T> CHQ_D void ppmx_limit(T qm2, T qm1, T q, T qp1, T qp2, T &qL, T &qR) {
  const T l = qL, r = qR;
  const T dqm = q - l, dqp = r - q;
  const bool extremum = (dqm * dqp <= T(0)) || ((qp1 - q) * (q - qm1) <= T(0));
  if (extremum) {
    const T d2 = T(6) * fma_(T(-2), q, l + r);
    const T d2c = fma_(T(-2), q, qm1 + qp1);
    const T d2l = fma_(T(-2), qm1, qm2 + q);
    const T d2r = fma_(T(-2), qp1, q + qp2);
    const T al = fabs_(d2l), ar = fabs_(d2r), ac = fabs_(d2c), a2 = fabs_(d2);
    const T lr = (al < ar) ? al : ar;
    const T lim = T(1.25) * ((lr < ac) ? lr : ac);
    const T m = (lim < a2) ? lim : a2;
    const bool same = d2 * d2c > T(0) && d2 * d2l > T(0) && d2 * d2r > T(0);
    const T thr = T(1e-12) * (fabs_(q) + fabs_(qm1) + fabs_(qp1)) + Tiny<T>::v;
    const T rho = (same && a2 > thr) ? quot_pos(m, a2) : T(0);
    if (rho < T(1) - T(1e-12)) {
      qL = q - rho * dqm;
      qR = q + rho * dqp;
    }
  } else {
    const T am = fabs_(dqm), ap = fabs_(dqp);
    qL = (am >= T(2) * ap) ? fma_(T(-2), dqp, q) : l;
    qR = (ap >= T(2) * am) ? fma_(T(2), dqm, q) : r;
  }
}

// WENO-Z (Borges et al. 2008), both interface values of one cell (src/recon.hpp:144-164): aR
// from the stencil (f_{-2}, .., f_{+2}) and aL from its mirror image. Mirroring maps the
// smoothness indicators (b0, b1, b2) to (b2, b1, b0) with equal values (the sums are commutative
// and a square does not see the sign), and tau to itself, so both sides share the three
// indicators and the three quotients tau / (b + eps): 5 divisions per cell instead of 8.
template <class T> struct WenoLimit;   // indicators and weights above this: plain divisions
template <> struct WenoLimit<double> { static constexpr double v = 0x1p+300; };
template <> struct WenoLimit<float> { static constexpr float v = 0x1p+96f; };

// six times the substencils' values at the face above the middle cell (the outer, the middle
// and the inner one, cells in order towards the face)
template <class T> CHQ_HD T weno_outer(T a, T b, T c) { return mad(T(11), c, mad(T(-7), b, T(2) * a)); }
template <class T> CHQ_HD T weno_mid(T a, T b, T c) { return fma_(T(2), c, mad(T(5), b, -a)); }
template <class T> CHQ_HD T weno_inner(T a, T b, T c) { return mad(T(5), b, T(2) * a) - c; }

template <bool PLAIN, class T> CHQ_D bool wenoz_both(const T q[5], T &aL, T &aR) {
  const T eps = Tiny<T>::weno_eps;
  const T c13 = T(13) / T(12);
  const T b0 = c13 * sqr(fma_(T(-2), q[1], q[0] + q[2])) + T(0.25) * sqr(fma_(T(-4), q[1], mad(T(3), q[2], q[0])));
  const T b1 = c13 * sqr(fma_(T(-2), q[2], q[1] + q[3])) + T(0.25) * sqr(q[1] - q[3]);
  const T b2 = c13 * sqr(fma_(T(-2), q[3], q[4] + q[2])) + T(0.25) * sqr(fma_(T(-4), q[3], mad(T(3), q[2], q[4])));
  const T tau = fabs_(b0 - b2);
  auto ratio = [&](T b) { return PLAIN ? tau / b : quot(tau, b, rcp_a(b)); };
  const T d0 = T(1) + ratio(b0 + eps), d1 = T(1) + ratio(b1 + eps), d2 = T(1) + ratio(b2 + eps);
  const T a1 = T(0.6) * d1;
  const T l0 = T(0.1) * d2, l2 = T(0.3) * d0, r0 = T(0.1) * d0, r2 = T(0.3) * d2;
  const T sr = r0 + a1 + r2, sl = l0 + a1 + l2;
  const T ir = PLAIN ? T(1) / sr : rcp_rn(sr), il = PLAIN ? T(1) / sl : rcp_rn(sl);
  aR = ir * (r0 * sixth(weno_outer(q[0], q[1], q[2])) + a1 * sixth(weno_mid(q[1], q[2], q[3])) +
             r2 * sixth(weno_inner(q[2], q[3], q[4])));
  aL = il * (l0 * sixth(weno_outer(q[4], q[3], q[2])) + a1 * sixth(weno_mid(q[3], q[2], q[1])) +
             l2 * sixth(weno_inner(q[2], q[1], q[0])));
  return sr < WenoLimit<T>::v && sl < WenoLimit<T>::v && (b0 + b1) + b2 < WenoLimit<T>::v;
}
template <class T> __device__ __noinline__ void wenoz_plain(T *v) {
  const T q[5] = {v[0], v[1], v[2], v[3], v[4]};
  wenoz_both<true>(q, v[5], v[6]);
}
template <class T> CHQ_D void wenoz_cell(const T q[5], T &aL, T &aR) {
  if (wenoz_both<false>(q, aL, aR)) return;
  T v[7] = {q[0], q[1], q[2], q[3], q[4]};
  wenoz_plain(v);
  aL = v[5];
  aR = v[6];
}

// CW84 flattening coefficient of the cell with pressures p5 = p_{c-2..c+2} and normal
// velocities um1 = u_{c-1}, up1 = u_{c+1} (src/recon.hpp:179-187)
template <class T> CHQ_HD T flattening(const T p5[5], T um1, T up1) {
  const T dp = p5[3] - p5[1];
  const T dp2 = p5[4] - p5[0];
  const T pmin = fmin_(p5[1], p5[3]);
  const bool strong = (fabs_(dp) > T(0.33) * pmin) && (um1 > up1);
  if (!strong) return T(0);
  const T ratio = (fabs_(dp2) > Tiny<T>::v) ? dp / dp2 : T(0);
  return fmin_(T(1), fmax_(T(0), T(10) * (ratio - T(0.75))));
}

// Number of stencil cells each side of the centre that scheme R reads.
template <int R> struct Reach { static constexpr int v = (R == R_DC) ? 0 : (R == R_PLM) ? 1 : 2; };

// Per-cell reconstruction: q5[0..4] = q_{c-2..c+2} (only q5[1..3] for PLM, q5[2] for DC).
// aL = value at the cell's left face (face c), aR = value at its right face (face c+1).
template <int R, class T> CHQ_D void recon_cell(const T q5[5], T &aL, T &aR) {
  if constexpr (R == R_DC) {
    aL = q5[2];
    aR = q5[2];
  } else if constexpr (R == R_PLM) {
    const T s = vl_slope(q5[1], q5[2], q5[3]);
    aR = q5[2] + T(0.5) * s;
    aL = q5[2] - T(0.5) * s;
  } else if constexpr (R == R_PPM) {
    const T sm = mc_slope2(q5[0], q5[1], q5[2]);
    const T s0 = mc_slope2(q5[1], q5[2], q5[3]);
    const T sp = mc_slope2(q5[2], q5[3], q5[4]);
    aL = ppm_face2(q5[1], q5[2], sm, s0);
    aR = ppm_face2(q5[2], q5[3], s0, sp);
    ppm_limit(q5[2], aL, aR);
  } else if constexpr (R == R_PPMX) {
    aL = ppmx_face(q5[0], q5[1], q5[2], q5[3]);
    aR = ppmx_face(q5[1], q5[2], q5[3], q5[4]);
    ppmx_limit(q5[0], q5[1], q5[2], q5[3], q5[4], aL, aR);
  } else {
    wenoz_cell(q5, aL, aR);
  }
}

}  // namespace chq
