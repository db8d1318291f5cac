// The reconstruction's limiter and substencils (chasqui_b200/csrc/chq_recon.cuh) on the host, in
// single precision, for tests/test_recon_rounding.py.
#include "chq_recon.cuh"

extern "C" __attribute__((visibility("default"))) void ppm(long n, const float *q, float *l, float *r) {
  for (long m = 0; m < n; ++m) chq::ppm_limit(q[m], l[m], r[m]);
}
extern "C" __attribute__((visibility("default"))) void weno(long n, const float *a, const float *b, const float *c, float *out) {
  for (long m = 0; m < n; ++m) {
    out[m] = chq::weno_outer(a[m], b[m], c[m]);
    out[n + m] = chq::weno_mid(a[m], b[m], c[m]);
    out[2 * n + m] = chq::weno_inner(a[m], b[m], c[m]);
  }
}
