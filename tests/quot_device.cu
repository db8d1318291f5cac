// Device check of chasqui_b200/csrc/chq_quot.cuh for tests/test_quot.py: FP32 over every
// significand of [1, 4); FP64 over the 2^20 values next to a power of two and to 4/3 on either side, where
// reciprocals, quotients and roots lie closest to rounding midpoints, and over as many scattered
// ones. Every result against the IEEE operation; prints "ok" or the counts. FP32 quotients by an
// uncorrected seed may be one unit off once in 10^7.
#include <cstdio>
#include "chq_quot.cuh"

using namespace chq;
__device__ unsigned long long wrong[16];
__device__ double where[16];
__device__ unsigned units;   // how far an FP32 quotient is off
template <class T> __device__ void check(int what, T got, T want, T at) {
  if (got == want) return;
  if (what == 2 || what == 3) atomicMax(&units, (unsigned)(fabs((double)got / (double)want - 1.0) * 0x1p23 + 0.999));
  atomicAdd(&wrong[what], 1ull);
  where[what] = (double)at;
}
__device__ float div(float a, float b) { return __fdiv_rn(a, b); }
__device__ double div(double a, double b) { return __ddiv_rn(a, b); }
__device__ float root(float a) { return __fsqrt_rn(a); }
__device__ double root(double a) { return __dsqrt_rn(a); }

template <class T> __device__ void one(int base, T b, unsigned seed) {
  const T ulp = sizeof(T) == 8 ? T(0x1p-52) : T(0x1p-23f);
  const T y = rcp_n(b);
  T ih;
  const T r = sqrt_q(b, ih), yr = rcp_root(r, ih);
  check(base, rcp_rn(b), div(T(1), b), b);
  check(base + 1, r, root(b), b);
  for (int j = 0; j < 24; ++j) {
    T a = T(1) + T(j) * ulp;
    if (j >= 8) a = T(1) - T(j - 7) * (ulp / 2);
    if (j >= 14) a = b + T(j - 16) * ulp;   // and next to the divisor
    if (j >= 18) a = T(1) + T((seed = seed * 1664525u + 1013904223u) >> 9) * T(0x1p-23f);
    check(base + 2, quot(a, b, y), div(a, b), b);
    check(base + 3, quot(a, r, yr), div(a, r), b);
    if (sizeof(T) == 8) check(base + 4, quot(a, b * b, y * y), div(a, b * b), b);
    check(base + 5, sixth(a), div(a, T(6)), a);
    check(base + 6, twelfth(a), div(a, T(12)), a);
  }
}
__global__ void floats(int n) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) one<float>(0, __uint_as_float(0x3f800000u + (unsigned)q), (unsigned)q);
}
__global__ void doubles(int n) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const double k = (double)(q + 1);
  one<double>(8, 1.0 - k * 0x1p-53, (unsigned)q);
  one<double>(8, 1.0 + k * 0x1p-52, (unsigned)q);
  one<double>(8, 2.0 - k * 0x1p-52, (unsigned)q);
  one<double>(8, 2.0 + k * 0x1p-51, (unsigned)q);
  one<double>(8, 4.0 / 3.0 + (k - 4.0) * 0x1p-52, (unsigned)q);
  one<double>(8, 4.0 - k * 0x1p-51, (unsigned)q);
  one<double>(8, 1.0 + 3.0 * (double)(((unsigned long long)q * 0x9E3779B97F4A7C15ull) >> 11) * 0x1p-53, (unsigned)q);
}

int main() {
  const int nf = 1 << 24, nd = 1 << 20;
  floats<<<(nf + 255) / 256, 256>>>(nf);
  doubles<<<(nd + 255) / 256, 256>>>(nd);
  unsigned long long w[16];
  double at[16];
  unsigned off;
  if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(w, wrong, sizeof w) != cudaSuccess ||
      cudaMemcpyFromSymbol(at, where, sizeof at) != cudaSuccess ||
      cudaMemcpyFromSymbol(&off, units, sizeof off) != cudaSuccess)
    return std::printf("%s\n", cudaGetErrorString(cudaGetLastError())), 1;
  static const char *name[8] = {"rcp_rn", "sqrt_q", "quot", "quot by root", "quot by square", "sixth", "twelfth", ""};
  int bad = 0;
  for (int q = 2; q < 4; ++q)
    if (off <= 1 && w[q] * 10000000ull <= 24ull * nf) w[q] = 0;
  for (int q = 0; q < 16; ++q)
    if (w[q]) bad = std::printf("%s %s: %llu wrong, last at %a\n", q < 8 ? "FP32" : "FP64", name[q & 7], w[q], at[q]);
  if (!bad) std::printf("ok\n");
  return bad != 0;
}
