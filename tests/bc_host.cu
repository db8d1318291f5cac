// The ghost fill's source mapping (bc_source, chasqui_b200/csrc/chq_kernels.cuh) applied on the
// host to packed arrays, for tests/test_ghost_fill.py: every frame point that bc_shape
// enumerates takes the value of its source.
#include "chq_kernels.cuh"

extern "C" __attribute__((visibility("default"))) int fill(int nx1, int nx2, int nx3, int ng, const int bc[3],
                                                            double *u, double *b1, double *b2, double *b3) {
  chq::Geom g{};
  g.nx1 = nx1; g.nx2 = nx2; g.nx3 = nx3; g.ng = ng;
  g.two_d = nx2 > 1; g.three_d = nx3 > 1;
  g.ni = nx1 + 2 * ng;
  g.nj = g.two_d ? nx2 + 2 * ng : 1;
  g.nk = g.three_d ? nx3 + 2 * ng : 1;
  g.is = ng; g.ie = ng + nx1 - 1;
  g.js = g.two_d ? ng : 0; g.je = g.two_d ? ng + nx2 - 1 : 0;
  g.ks = g.three_d ? ng : 0; g.ke = g.three_d ? ng + nx3 - 1 : 0;
  const chq::BcShape b = chq::bc_shape(g);
  double *f[3] = {b1, b2, b3};
  long count = 0;
  for (int k = 0; k <= g.nk; ++k)
    for (int j = 0; j <= g.nj; ++j)
      for (int i = 0; i <= g.ni; ++i) {
        const bool gk = g.three_d && (k < g.ks || k > g.ke), gj = g.two_d && (j < g.js || j > g.je), gi = i < g.is || i > g.ie;
        if (!(gk || gj || gi)) continue;
        ++count;
        for (int kind = 0; kind < 4; ++kind) {
          int sk, sj, si;
          bool fl[3];
          if (!chq::bc_source(g, bc, 3, kind, k, j, i, sk, sj, si, fl)) continue;
          if (kind == 0) {
            for (int n = 0; n < 6; ++n) {
              const bool neg = n >= 1 && n <= 3 && fl[n - 1];
              const double v = u[((n * g.nk + sk) * (long)g.nj + sj) * g.ni + si];
              u[((n * g.nk + k) * (long)g.nj + j) * g.ni + i] = neg ? -v : v;
            }
          } else {
            const double v = f[kind - 1][(sk * (long)(g.nj + 1) + sj) * (g.ni + 1) + si];
            f[kind - 1][(k * (long)(g.nj + 1) + j) * (g.ni + 1) + i] = fl[kind - 1] ? -v : v;
          }
        }
      }
  return count == b.nz + b.ny + b.nx ? 0 : 1;   // the launch covers exactly the ghost points
}
