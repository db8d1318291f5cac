// chasqui_b200 — quotients, reciprocals and square roots without branches.
//
// The flux kernel divides some forty times per face. A compiled IEEE division is a call-sized
// sequence of its own with a branch to a slow path, and a warp pays every branch for all its
// lanes (the FP64 y/z sweep spent 200 of its 1370 operations per face on control flow and ran
// 24 of 32 lanes on average). Here several quotients share one reciprocal, nothing branches,
// and the caller checks once per face that every divisor was in range.
//
//   rcp_a(b)        1/b to about half an ulp: the hardware seed and, in FP64, one third-order
//                   Newton step (Householder's method of order 2 for 1/x)
//   rcp_n(b)        the same, for divisors that may lie next to a power of two (below)
//   rcp_rn(b)       RN(1/b): one more Newton step (Markstein, IBM J. Res. Dev. 34 (1990) 111)
//   quot(a, b, y)   RN(a/b) for y = RN(1/b): Markstein's correction of q = RN(a y) by the
//                   exact remainder. rcp_a is RN(1/b) unless 1/b lies within 2^-7 ulp of a rounding
//                   midpoint, and then the corrected value still differs from a/b by less than
//                   2^-51 ulp before its rounding.
//                   The remainder is formed as b q - a and subtracted, which keeps the sign of a
//                   zero numerator for b > 0.
//   sqrt_q(x, ih)   RN(sqrt x) by Goldschmidt's iteration from the reciprocal-square-root seed
//                   with a third-order step and Markstein's final correction of a root from
//                   below (so that 1 - 2^-53, whose root lies just below a midpoint, is not
//                   corrected from 1); ih receives 1 / sqrt(x) to about an ulp, from which
//                   rcp_root makes the reciprocal of the root with one Newton step
// Reciprocals close to a midpoint by more than chance are those of divisors b = 2^n (1 - k 2^-53)
// with small odd k: the densities and wave speeds of a gas in units of its own, their roots, sums of weights. There the seed is
// so good that rcp_a rounds correctly, but for k = 1, a significand of all ones: 1/b is 2^-106
// above the midpoint of 1 and 1 + 2^-52, the step lands on the midpoint and ties to 1.
// rcp_n and rcp_root set the last bit there, rcp_rn steps from an approximation rounded up.
// FP32 uses the hardware seeds as they are: on a B200 rcp_rn and sqrt_q are IEEE for every
// significand, and of 8 10^8 quotients over all significands of the divisor some ten were one unit off.
// tests/test_quot.py compares all of them with the IEEE operations, on the device and, with
// coarser seeds, on the host.
// Valid for finite numerators and for divisors and radicands that in_range accepts (FP64
// 2^-300 .. 2^300, FP32 2^-60 .. 2^60, positive: in FP32 the square of a divisor and that of its
// reciprocal are then normal numbers); outside it the caller takes
// the plain operations. Compiles for the host as well, with the seeds emulated: 20 bits in FP64,
// and in FP32 a reciprocal one unit above and a root of 22 bits.
#pragma once
#include "chq_divide.cuh"
#include <cfenv>
#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define CHQ_DIV_D __device__ __forceinline__
#else
#define CHQ_DIV_D inline
#endif

namespace chq {

#if defined(__CUDA_ARCH__)
CHQ_DIV_HD double rcp_seed(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
}
CHQ_DIV_HD double rsqrt_seed(double b) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
}
CHQ_DIV_HD float rcp_seed(float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return y;
}
CHQ_DIV_HD float rsqrt_seed(float b) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return y;
}
CHQ_DIV_HD bool in_range(double x) { return (unsigned)__double2hiint(x) - 0x2D300000u < 0x25800000u; }
CHQ_DIV_HD bool in_range(float x) { return (unsigned)__float_as_int(x) - 0x21800000u < 0x3C000000u; }
// the wider range of a lone quotient
CHQ_DIV_HD bool quot_range(double x) { return in_range(x); }
CHQ_DIV_HD bool quot_range(float x) { return (unsigned)__float_as_int(x) - 0x0F800000u < 0x60000000u; }
CHQ_DIV_HD bool finite_q(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
CHQ_DIV_HD bool finite_q(float x) { return (__float_as_int(x) & 0x7f800000) != 0x7f800000; }
CHQ_DIV_HD double fma_up(double a, double b, double c) { return __fma_ru(a, b, c); }
CHQ_DIV_HD double fma_down(double a, double b, double c) { return __fma_rd(a, b, c); }
// y with its last bit set when b's significand is all ones
CHQ_DIV_HD double ones_up(double b, double y) {
  const int ones = ((__double2hiint(b) | (int)0xfff00000) & __double2loint(b)) == -1;
  return __hiloint2double(__double2hiint(y), __double2loint(y) | ones);
}
// x with its sign flipped when s is negative
CHQ_DIV_HD double flip_sign(double x, double s) {
  return __hiloint2double(__double2hiint(x) ^ (__double2hiint(s) & (int)0x80000000), __double2loint(x));
}
CHQ_DIV_HD float flip_sign(float x, float s) {
  return __int_as_float(__float_as_int(x) ^ (__float_as_int(s) & (int)0x80000000));
}
#else
// host emulation: the seeds' leading bits only
inline double chop(double y, int bits) {
  uint64_t u;
  std::memcpy(&u, &y, 8);
  u &= ~((1ull << (52 - bits)) - 1);
  std::memcpy(&y, &u, 8);
  return y;
}
inline double rcp_seed(double b) { return chop(1.0 / b, 20); }
inline double rsqrt_seed(double b) { return chop(1.0 / ::sqrt(b), 20); }
inline float rcp_seed(float b) {   // one unit at most, from above
  const float y = (float)(1.0 / (double)b);
  return (double)y < 1.0 / (double)b ? std::nextafterf(y, HUGE_VALF) : y;
}
inline float rsqrt_seed(float b) { return (float)chop(1.0 / ::sqrt((double)b), 22); }
inline bool in_range(double x) { return x >= 0x1p-300 && x < 0x1p+300; }
inline bool in_range(float x) { return x >= 0x1p-60f && x < 0x1p+60f; }
inline bool quot_range(double x) { return in_range(x); }
inline bool quot_range(float x) { return x >= 0x1p-96f && x < 0x1p+96f; }
template <class T> bool finite_q(T x) { return std::isfinite(x); }
inline double fma_mode(int mode, double a, double b, double c) {
  const int old = std::fegetround();
  std::fesetround(mode);
  volatile double x = a;
  volatile double r = fma_(x, b, c);
  std::fesetround(old);
  return r;
}
inline double fma_up(double a, double b, double c) { return fma_mode(FE_UPWARD, a, b, c); }
inline double fma_down(double a, double b, double c) { return fma_mode(FE_DOWNWARD, a, b, c); }
inline double ones_up(double b, double y) {
  uint64_t u, v;
  std::memcpy(&u, &b, 8);
  std::memcpy(&v, &y, 8);
  v |= (u & 0xfffffffffffffull) == 0xfffffffffffffull;
  std::memcpy(&y, &v, 8);
  return y;
}
inline double flip_sign(double x, double s) { return std::signbit(s) ? -x : x; }
inline float flip_sign(float x, float s) { return std::signbit(s) ? -x : x; }
#endif

CHQ_DIV_HD double rcp_a(double b) {
  const double y = rcp_seed(b);
  const double e = fma_(-b, y, 1.0);
  return fma_(y, fma_(e, e, e), y);
}
CHQ_DIV_HD float rcp_a(float b) { return rcp_seed(b); }
CHQ_DIV_HD double rcp_n(double b) { return ones_up(b, rcp_a(b)); }
CHQ_DIV_HD float rcp_n(float b) { return rcp_seed(b); }

template <class T> CHQ_DIV_HD T rcp_step(T b, T y) { return fma_(fma_(-b, y, T(1)), y, y); }
CHQ_DIV_HD double rcp_rn(double b) {
  const double y = rcp_seed(b);
  const double e = fma_(-b, y, 1.0);
  return rcp_step(b, fma_up(y, fma_(e, e, e), y));
}
CHQ_DIV_HD float rcp_rn(float b) { return rcp_step(b, rcp_seed(b)); }

template <class T> CHQ_DIV_HD T quot(T a, T b, T y) {
  const T q = mul_rn(a, y);
  return fma_(fma_(b, q, -a), -y, q);
}

CHQ_DIV_HD double sqrt_q(double x, double &ih) {
  const double y = rsqrt_seed(x);
  const double g = mul_rn(x, y), h = 0.5 * y;
  const double e = fma_(-g, h, 0.5);           // sqrt(x) = g (1 - 2e)^(-1/2)
  const double p = fma_(mul_rn(1.5, e), e, e); // (1 - 2e)^(-1/2) - 1 to third order
  const double g1 = fma_down(g, p, g), h1 = fma_(h, p, h);
  ih = h1 + h1;
  return fma_(fma_(-g1, g1, x), h1, g1);
}
CHQ_DIV_HD float sqrt_q(float x, float &ih) {
  ih = rsqrt_seed(x);
  const float g = mul_rn(x, ih), h = 0.5f * ih;
  return fma_(fma_(-g, g, x), h, g);
}
CHQ_DIV_HD double rcp_root(double r, double ih) { return ones_up(r, rcp_step(r, ih)); }
CHQ_DIV_HD float rcp_root(float, float ih) { return ih; }
template <class T> CHQ_DIV_HD T sqrt_q(T x) {
  T ih;
  return sqrt_q(x, ih);
}

// a b + c in the form's own arithmetic: two roundings in FP64, one in FP32 (the mixed form lets
// products contract). Written out where a product is shared by several sums, which the compiler
// would otherwise round once for all of them.
CHQ_DIV_HD double mad(double a, double b, double c) { return a * b + c; }
CHQ_DIV_HD float mad(float a, float b, float c) { return fma_(a, b, c); }

// radicands below this are negligible beside any in_range value they are added to the root of
// (their root is at most 2^-150 resp. 2^-24 of it) and count as zero
template <class T> struct RootFloor;
template <> struct RootFloor<double> { static constexpr double v = 0x1p-900; };
template <> struct RootFloor<float> { static constexpr float v = 0x1p-120f; };

// upper end of in_range
template <class T> struct QuotMax;
template <> struct QuotMax<double> { static constexpr double v = 0x1p+300; };
template <> struct QuotMax<float> { static constexpr float v = 0x1p+60f; };

// a / b for a >= 0, b > 0 (either may be out of range: then the plain division, out of line)
#if defined(__CUDACC__)
template <class T> __device__ __noinline__ T div_plain(T a, T b) { return a / b; }
#else
template <class T> T div_plain(T a, T b) { return a / b; }
#endif
template <class T> CHQ_DIV_D T quot_pos(T a, T b) {
  const T r = quot(a, b, rcp_a(b));
  return quot_range(b) && finite_q(a) ? r : div_plain(a, b);
}

// x / 6 and x / 12 with one product and the exact remainder (div6 in chq_divide.cuh has the
// proof); exact for every finite x whose quotient is normal, off by at most one unit in the
// last place of the smallest subnormal below that
template <class T> CHQ_DIV_HD T sixth(T x) { return quot(x, T(6), DivConst<T>::sixth); }
template <class T> CHQ_DIV_HD T twelfth(T x) { return quot(x, T(12), T(0.5) * DivConst<T>::sixth); }

}  // namespace chq
