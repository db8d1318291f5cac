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
//   rcp_rn(b)       one more Newton step: RN(1/b) (Markstein, IBM J. Res. Dev. 34 (1990) 111)
//   quot(a, b, y)   RN(a/b) for y = rcp_a(b): Markstein's correction of q = RN(a y) by the
//                   exact remainder. The corrected value differs from a/b by less than
//                   2^-51 ulp before its rounding, so it can miss RN(a/b) only when a/b lies
//                   that close to a rounding midpoint. FP32 uses the hardware seed as it
//                   is (one unit at most): every reciprocal's correction, every root and 2^30
//                   quotients over all significands of the divisor came out IEEE on a B200.
//                   The remainder is formed as b q - a and subtracted, which keeps the sign of
//                   a zero numerator for b > 0.
//   sqrt_q(x, ih)   RN(sqrt x) by Goldschmidt's iteration from the reciprocal-square-root seed
//                   with a third-order step and Markstein's final correction (as accurate as
//                   quot); ih receives 1 / sqrt(x) to about an ulp, so that a quotient by the
//                   root needs no reciprocal of its own
// A divisor whose significand is all ones is the theorem's one exception: its reciprocal and
// the quotients of powers of two by it may be one unit off.
// Valid for finite numerators and for divisors and radicands that in_range accepts (FP64
// 2^-300 .. 2^300, FP32 2^-36 .. 2^60, positive); outside it the caller takes the plain
// operations. Compiles for the host with the seeds emulated at their documented 20 (FP64) and
// 22 (FP32) bits (tests/quot_check.cpp compares every function with the IEEE operation; with
// the coarser FP32 seed one quotient in 10^5 is one unit off there).
#pragma once
#include "chq_divide.cuh"
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
CHQ_DIV_HD bool in_range(float x) { return (unsigned)__float_as_int(x) - 0x2D800000u < 0x30000000u; }
// the wider range of a lone quotient
CHQ_DIV_HD bool quot_range(double x) { return in_range(x); }
CHQ_DIV_HD bool quot_range(float x) { return (unsigned)__float_as_int(x) - 0x0F800000u < 0x60000000u; }
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
inline float rcp_seed(float b) { return (float)chop(1.0 / (double)b, 22); }
inline float rsqrt_seed(float b) { return (float)chop(1.0 / ::sqrt((double)b), 22); }
inline bool in_range(double x) { return x >= 0x1p-300 && x < 0x1p+300; }
inline bool in_range(float x) { return x >= 0x1p-36f && x < 0x1p+60f; }
inline bool quot_range(double x) { return in_range(x); }
inline bool quot_range(float x) { return x >= 0x1p-96f && x < 0x1p+96f; }
inline double flip_sign(double x, double s) { return std::signbit(s) ? -x : x; }
inline float flip_sign(float x, float s) { return std::signbit(s) ? -x : x; }
#endif

CHQ_DIV_HD double rcp_a(double b) {
  const double y = rcp_seed(b);
  const double e = fma_(-b, y, 1.0);
  return fma_(y, fma_(e, e, e), y);
}
CHQ_DIV_HD float rcp_a(float b) { return rcp_seed(b); }

template <class T> CHQ_DIV_HD T rcp_rn(T b) {
  const T y = rcp_a(b);
  return fma_(fma_(-b, y, T(1)), y, y);
}

template <class T> CHQ_DIV_HD T quot(T a, T b, T y) {
  const T q = mul_rn(a, y);
  return fma_(fma_(b, q, -a), -y, q);
}

CHQ_DIV_HD double sqrt_q(double x, double &ih) {
  const double y = rsqrt_seed(x);
  const double g = mul_rn(x, y), h = 0.5 * y;
  const double e = fma_(-g, h, 0.5);           // sqrt(x) = g (1 - 2e)^(-1/2)
  const double p = fma_(mul_rn(1.5, e), e, e); // (1 - 2e)^(-1/2) - 1 to third order
  const double g1 = fma_(g, p, g), h1 = fma_(h, p, h);
  ih = h1 + h1;
  return fma_(fma_(-g1, g1, x), h1, g1);
}
CHQ_DIV_HD float sqrt_q(float x, float &ih) {
  ih = rsqrt_seed(x);
  const float g = mul_rn(x, ih), h = 0.5f * ih;
  return fma_(fma_(-g, g, x), h, g);
}
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

// a / b for a >= 0, b > 0 (either may be out of range: then the plain division, out of line)
#if defined(__CUDACC__)
template <class T> __device__ __noinline__ T div_plain(T a, T b) { return a / b; }
#else
template <class T> T div_plain(T a, T b) { return a / b; }
#endif
template <class T> CHQ_DIV_D T quot_pos(T a, T b) {
  const T r = quot(a, b, rcp_a(b));
  return quot_range(b) ? r : div_plain(a, b);
}

// x / 6 and x / 12 with one product and the exact remainder (div6 in chq_divide.cuh has the
// proof); exact for every finite x whose quotient is normal, off by at most one unit in the
// last place of the smallest subnormal below that
template <class T> CHQ_DIV_HD T sixth(T x) { return quot(x, T(6), DivConst<T>::sixth); }
template <class T> CHQ_DIV_HD T twelfth(T x) { return quot(x, T(12), T(0.5) * DivConst<T>::sixth); }

}  // namespace chq
