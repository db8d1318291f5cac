// Host check of chasqui_b200/csrc/chq_quot.cuh with the seeds emulated: rcp_rn, quot, sqrt_q,
// sixth and twelfth against the IEEE operations bit for bit (FP64; FP32: at most one unit off,
// in fewer than 1 of 10^4) over random significands and exponents inside the stated ranges,
// significands next to 1 and 2 (all ones among them) and signed zeros. Built and run by tests/test_quot.py; prints "ok <cases>" or a mismatch.
#include <cstdio>
#include <cstdlib>
#include "chq_quot.cuh"

static uint64_t s = 0x9E3779B97F4A7C15ull;
static uint64_t next() {   // splitmix64
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
template <class T> static T draw(int elo, int ehi) {
  const int p = sizeof(T) == 8 ? 52 : 23;
  uint64_t m = next() & ((1ull << p) - 1);
  switch (next() & 7) {   // near 1, near 2, short significands
    case 0: m &= 0xff; break;
    case 1: m |= ~0xffull & ((1ull << p) - 1); break;
    case 2: m &= ~((1ull << (p - 4)) - 1); break;
    default: break;
  }
  return (T)std::ldexp(1.0 + std::ldexp((double)m, -p), elo + (int)(next() % (uint64_t)(ehi - elo)));
}
static bool same(double a, double b) { return a == b && std::signbit(a) == std::signbit(b); }
static long off = 0;   // FP32 results one unit off
static bool same(float a, float b) {
  if (a == b && std::signbit(a) == std::signbit(b)) return true;
  ++off;
  return std::nextafter(a, b) == b;
}

template <class T> static long run(long n, int elo, int ehi, const char *name) {
  for (long q = 0; q < n; ++q) {
    T b = draw<T>(elo, ehi);
    T a = draw<T>(elo, ehi);
    if (next() & 1) a = -a;
    if ((next() & 63) == 0) a = std::copysign(T(0), a);
    const T y = chq::rcp_n(b);
    if (!same(chq::quot(a, b, y), a / b)) return std::printf("%s quot %a / %a\n", name, (double)a, (double)b), 1;
    if (!same(chq::rcp_rn(b), T(1) / b)) return std::printf("%s rcp_rn %a\n", name, (double)b), 1;
    T ih;
    const T r = chq::sqrt_q(b, ih);
    if (!same(r, (T)std::sqrt(b))) return std::printf("%s sqrt_q %a\n", name, (double)b), 1;
    if (!same(chq::quot(a, r, chq::rcp_root(r, ih)), a / r)) return std::printf("%s quot by root %a / %a\n", name, (double)a, (double)r), 1;
    const T d = b * b, z = y * y;   // the reciprocal of a square from that of its root
    if (sizeof(T) == 8 && !same(chq::quot(a, d, z), a / d)) return std::printf("%s quot by square %a\n", name, (double)b), 1;
    if (!same(chq::sixth(a), a / T(6))) return std::printf("%s sixth %a\n", name, (double)a), 1;
    if (!same(chq::twelfth(a), a / T(12))) return std::printf("%s twelfth %a\n", name, (double)a), 1;
  }
  return 0;
}

int main(int argc, char **argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 2000000;
  if (run<double>(n, -300, 300, "double") || run<double>(n, -3, 3, "double near one")) return 1;
  if (run<float>(n, -60, 60, "float") || run<float>(n, -3, 3, "float near one")) return 1;
  if (off * 10000 > 2 * n) return std::printf("float: %ld of %ld results one unit off\n", off, 2 * n), 1;
  std::printf("ok %ld\n", 4 * n);
  return 0;
}
