// chasqui_b200 — K1: the fused face-flux kernel of one Runge-Kutta stage.
//
// Per face: reconstruct both sides from the primitives, apply flattening and the
// donor-cell floor fallback, optionally the low-Mach velocity blend, solve the Riemann
// problem in registers and write the 6 conserved fluxes plus the two face EMF components
// (E_t2 = -F(B_t1), E_t1 = +F(B_t2)). Same face ranges and outputs as the reference's
// Fluxes<DIR,R,S> (src/physics.hpp:66-226); the left/right face states never leave the SM.
//
// Work decomposition, two launches per stage:
//   flux_x_kernel : one warp = 32 consecutive cells of the rows laid end to end; lane l computes the (aL, aR)
//             pair of its cell once (stencil from L1) and receives its left neighbour's aR by
//             __shfl_up_sync, so a warp emits 31 faces and no cell parabola is evaluated twice
//             (PPM: slopes and unlimited interface values are shared between lanes too, and a
//             warp emits 29 faces).
//   flux_yz_kernel: lanes run along i, rows end to end (coalesced); each thread marches `slen`
//             faces along y or z with its stencil in a shared-memory window that cp.async
//             refills one cell ahead, and parks the previous cell's aR in shared memory
//             during the Riemann solve (PPM: the march carries each quantity's slope and
//             unlimited interface value to the next cell). z warps come first, then y.
// The batched forms (flux_x_batched, flux_yz_batched) run the same sweeps for many meshes.
#pragma once
#include <cuda.h>   // CUtensorMap (the TMA descriptor type; no driver call is made from here)
#include "chq_common.cuh"
#include "chq_recon.cuh"
#include "chq_riemann.cuh"
#include "chq_eigen.cuh"

namespace chq {

struct StepCtl;   // device-resident time-step control (chq_ctl.cuh)

template <class P> struct FluxArgs {
  Geom g;
  EOSp eos;
  const P *w;          // primitives, 6 components
  const P *bcc;        // cell-centred B, 3 components
  const double *bn[3]; // face-normal field of the stage's current state, per direction
  P *flx[3];           // fluxes, 6 components, per direction
  P *et2[3];           // E_{t2} on faces of each direction (e3x1, e1x2, e2x3)
  P *et1[3];           // E_{t1} on faces of each direction (e2x1, e3x2, e1x3)
  int flatten, low_mach;
  double lhlld_phi;
  P rgm1;              // 1 / (gamma - 1), rounded once
  // inclusive face ranges per direction: lo[dir][0..2] = (k, j, i)
  int lo[3][3], hi[3][3];
  int active[3];
  int slen[3];         // faces per thread along y/z sweeps (at most the march length)
  int nseg[3];         // march segments per y/z column
  int ncol[3];         // y/z: columns (i, outer) of the direction, i fastest
  int nblk[3];         // y/z: blocks of the direction (kYzThreads columns each x segments)
  int nxent, nxrow;    // x: cells a row contributes (faces + XLead), rows
  int nxwarp;          // x: warps
  int nchunk;          // TMA staging: 32-wide i chunks (aligned to i = 0)
  int xvar;            // x-sweep kernel variant (register cap, FluxMinBlocks); picked by the autotuner
  const int *skip;     // optional device flag: nonzero -> kernel returns immediately
  int yzvar;           // y/z staging of the FP64 streaming-PPM march: 0 cp.async, 1 TMA (autotuner)
  const void *yzmaps;  // host copy of the two tensor maps of the TMA staging (YzMaps), or null
  int *err;            // device error word: a TMA wait that gave up sets it (and its warp stops)
};

// Tensor maps of the TMA staging: the primitives w (6 components) and the centred field bcc
// (3 components) of one mesh as 4-D tensors (i over the row pitch, j, k, component), boxes of
// one 32-cell row segment of one component.
struct YzMaps {
  CUtensorMap w, b;
};

// ---------------------------------------------------------------------------------------
// Per-direction views: the 8 reconstructed quantities (d, u, v, w, p, by, bz, s) of the
// frame of direction d and the output slots of its faces. Built once per warp; the
// arithmetic is identical for every direction, so one code copy serves the y and z sweeps.
template <class P> struct DirView {
  const P *src[8];     // cell fields in face-frame order
  const P *bx;         // cell-centred normal field (characteristic projection)
  int st;              // stride along the sweep (offsets within a component fit in 32 bits)
  int s1, s2;          // strides of the two transverse directions (LHLLD detector)
  int has1, has2;
  const double *bn;    // face-normal field of the stage's current state
  P *out[8];           // flux slots (d, u, v, w, E, s) then E_t2, E_t1
};

template <class P> CHQ_D DirView<P> dir_view(const FluxArgs<P> &A, int d) {
  DirView<P> v;
  const long vs = A.g.vstride;
  const int ivu = IVX + d, ivv = IVX + (d + 1) % 3, ivw = IVX + (d + 2) % 3;
  const int t1 = (d + 1) % 3, t2 = (d + 2) % 3;
  const int strides[3] = {1, (int)A.g.sj, (int)A.g.sk};
  v.src[0] = A.w + IDN * vs;
  v.src[1] = A.w + ivu * vs;
  v.src[2] = A.w + ivv * vs;
  v.src[3] = A.w + ivw * vs;
  v.src[4] = A.w + IPR * vs;
  v.src[5] = A.bcc + t1 * vs;
  v.src[6] = A.bcc + t2 * vs;
  v.src[7] = A.w + IENT * vs;
  v.bx = A.bcc + d * vs;
  v.st = strides[d];
  v.s1 = strides[t1];
  v.s2 = strides[t2];
  v.has1 = (t1 == 0) || (t1 == 1 && A.g.two_d) || (t1 == 2 && A.g.three_d);
  v.has2 = (t2 == 0) || (t2 == 1 && A.g.two_d) || (t2 == 2 && A.g.three_d);
  v.bn = A.bn[d];
  P *f = A.flx[d];
  v.out[0] = f + IDN * vs;
  v.out[1] = f + ivu * vs;
  v.out[2] = f + ivv * vs;
  v.out[3] = f + ivw * vs;
  v.out[4] = f + IEN * vs;
  v.out[5] = f + IENT * vs;
  v.out[6] = A.et2[d];
  v.out[7] = A.et1[d];
  return v;
}

// ---------------------------------------------------------------------------------------
// Flattening toward the cell value (PPM, PPMX, WENO-Z; src/recon.hpp:179-187 applied as in
// src/physics.hpp:152-162) and the donor-cell fallback of a side that reconstructed to
// rho <= floor or p <= floor, on the cell's (aL, aR) pairs of the 8 quantities.
template <int R, class P>
CHQ_D void finish_states(const FluxArgs<P> &A, P aL[8], P aR[8], const P qc[8], const P p5[5], P um1, P up1) {
  if constexpr (R == R_PPM || R == R_PPMX || R == R_WENOZ) {
    if (A.flatten) {
      const P f = flattening<P>(p5, um1, up1);
      if (f > P(0)) {
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          aL[n] += f * (qc[n] - aL[n]);
          aR[n] += f * (qc[n] - aR[n]);
        }
      }
    }
  }
  const P dfl = P(A.eos.dfloor), pfl = P(A.eos.pfloor);
  if (aL[0] <= dfl || aL[4] <= pfl) {
#pragma unroll
    for (int n = 0; n < 8; ++n) aL[n] = qc[n];
  }
  if (aR[0] <= dfl || aR[4] <= pfl) {
#pragma unroll
    for (int n = 0; n < 8; ++n) aR[n] = qc[n];
  }
}

// ---------------------------------------------------------------------------------------
// Cell work: the (aL, aR) pair of cell `lc` (linear index) for the 8 reconstructed
// quantities in the frame of the view's direction. Each quantity is reconstructed as soon
// as its stencil is loaded, so only the cell values (for flattening and the floor
// fallback) stay live across quantities.
template <int R, bool CHAR, class P, class Stencil>
CHQ_D void cell_states_from(const FluxArgs<P> &A, const DirView<P> &V, int lc, P aL[8], P aR[8], const Stencil &ld) {
  constexpr int RE = Reach<R>::v;
  P qc[8];
  P p5[5], um1 = P(0), up1 = P(0);
  if constexpr (!CHAR || R == R_DC) {
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      P q5[5];
      ld(n, q5);
#pragma unroll
      for (int m = RE + 1; m <= 2; ++m) { q5[2 + m] = q5[2 + RE]; q5[2 - m] = q5[2 - RE]; }
      recon_cell<R>(q5, aL[n], aR[n]);
      qc[n] = q5[2];
      if (n == 1) { um1 = q5[1]; up1 = q5[3]; }
      if (n == 4) {
#pragma unroll
        for (int m = 0; m < 5; ++m) p5[m] = q5[m];
      }
    }
  } else {
    // characteristic projection with this cell's own eigenvectors (src/physics.hpp:108-150)
    P q[7][5];
#pragma unroll
    for (int n = 0; n < 7; ++n) {
      ld(n, q[n]);
#pragma unroll
      for (int m = RE + 1; m <= 2; ++m) { q[n][2 + m] = q[n][2 + RE]; q[n][2 - m] = q[n][2 - RE]; }
      qc[n] = q[n][2];
    }
    um1 = q[1][1];
    up1 = q[1][3];
#pragma unroll
    for (int m = 0; m < 5; ++m) p5[m] = q[4][m];
    Eigen7<P> E;
    eigensystem<P>(q[0][2], q[4][2], q[5][2], q[6][2], ldg(V.bx + lc), P(A.eos.gamma), E);
    P cL[7], cR[7];
#pragma unroll
    for (int kk = 0; kk < 7; ++kk) {
      P c5[5];
#pragma unroll
      for (int m = 2 - RE; m <= 2 + RE; ++m) {
        P acc = P(0);
#pragma unroll
        for (int n = 0; n < 7; ++n) acc += E.L[kk][n] * q[n][m];
        c5[m] = acc;
      }
#pragma unroll
      for (int m = RE + 1; m <= 2; ++m) { c5[2 + m] = c5[2 + RE]; c5[2 - m] = c5[2 - RE]; }
      recon_cell<R>(c5, cL[kk], cR[kk]);
    }
#pragma unroll
    for (int n = 0; n < 7; ++n) {
      P accL = P(0), accR = P(0);
#pragma unroll
      for (int kk = 0; kk < 7; ++kk) {
        accL += E.R[n][kk] * cL[kk];
        accR += E.R[n][kk] * cR[kk];
      }
      aL[n] = accL;
      aR[n] = accR;
    }
    // entropy scalar, always primitive
    P q5[5];
    ld(7, q5);
#pragma unroll
    for (int m = RE + 1; m <= 2; ++m) { q5[2 + m] = q5[2 + RE]; q5[2 - m] = q5[2 - RE]; }
    recon_cell<R>(q5, aL[7], aR[7]);
    qc[7] = q5[2];
  }
  finish_states<R, P>(A, aL, aR, qc, p5, um1, up1);
}

// Stencil sources of cell_states_from: q5[2-RE .. 2+RE] of quantity n of the cell.
// Global: cached loads along the sweep (the x-sweep, whose stencil lies in the lanes' lines).
template <int RE, class P> struct GlobalStencil {
  const DirView<P> &V;
  int lc;
  CHQ_D void operator()(int n, P q5[5]) const {
#pragma unroll
    for (int m = -RE; m <= RE; ++m) q5[2 + m] = ldg(V.src[n] + lc + m * V.st);
  }
};

template <int R, bool CHAR, class P>
CHQ_D void cell_states(const FluxArgs<P> &A, const DirView<P> &V, int lc, P aL[8], P aR[8]) {
  cell_states_from<R, CHAR, P>(A, V, lc, aL, aR, GlobalStencil<Reach<R>::v, P>{V, lc});
}

// asynchronous global -> shared copies of one element (cp.async, completed per thread)
CHQ_D void cp_async_elem(double *dst, const double *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
CHQ_D void cp_async_elem(float *dst, const float *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
CHQ_D void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
CHQ_D void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Tensor-memory-access (TMA) staging: an mbarrier in shared memory counts the bytes the
// bulk tensor copies deliver (complete_tx); threads wait on its phase parity.
CHQ_D unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
CHQ_D void mbar_init(unsigned long long *mb, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(mb)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
CHQ_D void mbar_expect_tx(unsigned long long *mb, unsigned bytes) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(smem_addr(mb)),
               "r"(bytes)
               : "memory");
}
// bounded wait for the phase of the given parity; false when the limit ran out
CHQ_D bool mbar_wait(unsigned long long *mb, unsigned parity) {
  const unsigned a = smem_addr(mb);
  for (int it = 0; it < (1 << 24); ++it) {
    unsigned ok = 0;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(a), "r"(parity)
                 : "memory");
    if (ok) return true;
  }
  return false;
}
// generic-proxy accesses of shared memory before the async-proxy writes that follow
CHQ_D void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// one box of a 4-D tensor map over this GPU's own memory into this CTA's shared memory only,
// completing on mb
CHQ_D void tma_load_4d(void *dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, unsigned long long *mb) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(
          smem_addr(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_addr(mb))
      : "memory");
}

// Threads per block of the y/z kernels (the stride of their shared-memory columns).
#ifndef CHQ_FLUXYZ_THREADS
#define CHQ_FLUXYZ_THREADS 128
#endif
constexpr int kYzThreads = CHQ_FLUXYZ_THREADS;

// Lane mapping of the y/z sweeps: the direction's columns (i, outer index) are numbered with i
// fastest and a block takes the next kYzThreads of them for one march segment, so a warp may
// hold the end of one row and the start of the next. Warps cut at 32-cell boundaries of each
// row left 4 of 32 lanes busy in every last warp (130 columns at 128^3: 5 warps a row, 81 % of
// the lanes; 66 at 64^2: 3 warps, 69 %).
template <class P> CHQ_D bool yz_place(const FluxArgs<P> &A, int d, int blk, int &i, int &outer, int &seg) {
  const int cb = blk / A.nseg[d];
  seg = blk - cb * A.nseg[d];
  const int col = cb * kYzThreads + (int)threadIdx.x;
  if (col >= A.ncol[d]) return false;
  const int w = A.hi[d][2] - A.lo[d][2] + 1;
  outer = col / w;
  i = A.lo[d][2] + (col - outer * w);
  return true;
}

// Marching window: one shared-memory column per thread and quantity, 2RE+1 slots. For the
// current cell c, slots 0..2RE-1 hold q[c-RE .. c+RE-1] and slot 2RE holds q[c+RE], copied
// asynchronously one step earlier. Reading the stencil shifts the window down by one slot
// (every slot value is consumed by that shift before the next copy into slot 2RE is issued,
// so the copy cannot overtake the read) and starts the copy of q[c+RE+1] for the next cell.
template <int RE, class P> struct WindowStencil {
  P *col;            // this thread's column: slot m of quantity n at col[(n*(2RE+1) + m) * kYzThreads]
  const DirView<P> &V;
  int lc;
  bool prefetch;     // false on the last cell of the march
  CHQ_D void operator()(int n, P q5[5]) const {
    P *w = col + n * (2 * RE + 1) * kYzThreads;
#pragma unroll
    for (int m = 0; m <= 2 * RE; ++m) q5[2 - RE + m] = w[m * kYzThreads];
#pragma unroll
    for (int m = 0; m < 2 * RE; ++m) w[m * kYzThreads] = q5[3 - RE + m];
    if (prefetch) cp_async_elem(w + 2 * RE * kYzThreads, V.src[n] + lc + (RE + 1) * V.st);
  }
};

// ---------------------------------------------------------------------------------------
// Face work: Riemann solve of the face `lf` (between cells lf - stride and lf).
//
// What bounds it: FP64 issue (61 % of the FP64 pipe's cycles in the y/z launch, 70 % in the x
// launch at 128^3; 746 FP64 operations a face and thread). With compiled divisions and branching
// limiters a face took 2200 warp instructions at 24 of 32 active lanes and waited on instruction
// fetch; with chq_quot.cuh and selects it takes 1380 at 31.6, and the FP64 PPM + HLLD flux launch
// went from 0.880 to 0.45 ms at 128^3 (blast), 5.21 to 3.24 ms at 256^3 (mixed: 2.89 to 1.85 ms),
// WENO-Z from 1.92 to 0.78 ms at 128^3, OT 256^2 from 43 to 16 us (rows laid end to end and
// balanced marches included).

// low-Mach blend of the normal velocities, Thornber et al. (2008) (src/physics.hpp:170-178)
template <class P> CHQ_D void low_mach_blend(MState<P> &L, MState<P> &R, P cl, P cr) {
  const P z = fmin_(P(1), fmax_(divz(fabs_(L.u), cl), divz(fabs_(R.u), cr)));
  const P um = P(0.5) * (L.u + R.u), ud = P(0.5) * (z * (L.u - R.u));
  L.u = um + ud;
  R.u = um - ud;
}

// The face solved again from memory with plain divisions (hlld), for the rare face whose
// divisors leave the range of hlld_q: both cells' states by the per-cell reconstruction, which
// gives the sweeps' states bit for bit. Not inlined and given nothing but the face's place, so
// that the hot code keeps none of its operands alive for it.
template <int R, int S, bool CHAR, class P>
__device__ __noinline__ void face_plain(const FluxArgs<P> *args, int d, int lf);

// Solver only; b_n: the face-normal field of the face. PLAIN: hlld with plain divisions.
// Returns false when hlld_q's divisors left their range (f is then undefined).
template <int S, bool PLAIN, class P>
CHQ_D bool face_solve(const FluxArgs<P> &A, const DirView<P> &V, int lf, const P wl[8], const P wr[8], const P b_n, P f[NFLX]) {
  const P gamma = P(A.eos.gamma), gm1 = P(A.eos.gm1);
  MState<P> L{wl[0], wl[1], wl[2], wl[3], wl[4], wl[5], wl[6]};
  MState<P> R{wr[0], wr[1], wr[2], wr[3], wr[4], wr[5], wr[6]};
  if constexpr (S == S_HLLE) {
    if (A.low_mach) low_mach_blend(L, R, fast_speed(L, b_n, gamma), fast_speed(R, b_n, gamma));
    hlle(L, R, b_n, gamma, gm1, f);
    return true;
  }
  const P bnsq = b_n * b_n;
  const P bsql = bnsq + L.by * L.by + L.bz * L.bz, bsqr = bnsq + R.by * R.by + R.bz * R.bz;
  bool ok = true;
  P cl, cr;
  if constexpr (PLAIN) {
    cl = fast_speed(L, b_n, gamma);
    cr = fast_speed(R, b_n, gamma);
  } else {
    cl = fast_speed_q(L, b_n, bsql, gamma, ok);
    cr = fast_speed_q(R, b_n, bsqr, gamma, ok);
  }
  if (A.low_mach) low_mach_blend(L, R, cl, cr);
  if constexpr (S == S_HLLD) {
    if constexpr (PLAIN) hlld<false>(L, R, b_n, gamma, gm1, f, P(1), P(1));
    else ok = hlld_q<false>(L, R, b_n, gm1, A.rgm1, bsql, bsqr, cl, cr, P(1), P(1), f) && ok;
  } else if constexpr (S == S_LHLLD) {
    // shock detector theta and low-Mach factor phi (src/physics.hpp:183-211)
    const int lL = lf - V.st;
    const P cfmax = fmax_(cl, cr);
    const P *wu = V.src[1], *wv = V.src[2], *ww = V.src[3];
    const int s1 = V.s1, s2 = V.s2;
    const P du = ldg(wu + lf) - ldg(wu + lL);
    P dvw = P(0);
    if (V.has1) {
      const P d1 = fmin_(fmin_(ldg(wv + lL) - ldg(wv + lL - s1), ldg(wv + lL + s1) - ldg(wv + lL)),
                         fmin_(ldg(wv + lf) - ldg(wv + lf - s1), ldg(wv + lf + s1) - ldg(wv + lf)));
      dvw = fmin_(dvw, d1);
    }
    if (V.has2) {
      const P d2 = fmin_(fmin_(ldg(ww + lL) - ldg(ww + lL - s2), ldg(ww + lL + s2) - ldg(ww + lL)),
                         fmin_(ldg(ww + lf) - ldg(ww + lf - s2), ldg(ww + lf + s2) - ldg(ww + lf)));
      dvw = fmin_(dvw, d2);
    }
    const P num = -fmin_(du, P(0)) + cfmax, den = -dvw + cfmax;
    P ratio, chi;
    if constexpr (PLAIN) {
      ratio = num / den;
      chi = divz(fmax_(flow_speed_u(L, b_n), flow_speed_u(R, b_n)), cfmax);
    } else {
      ok = ok && in_range(den) && in_range(cfmax);
      ratio = quot(num, den, rcp_n(den));
      chi = quot(fmax_(flow_speed_q(L, b_n, ok), flow_speed_q(R, b_n, ok)), cfmax, rcp_n(cfmax));
    }
    ratio = fmin_(P(1), ratio);
    chi = fmin_(P(1), chi);
    const P r2 = ratio * ratio;
    const P theta = r2 * r2;
    const P phi = (A.lhlld_phi >= 0.0) ? P(A.lhlld_phi) : chi * (P(2) - chi);
    if constexpr (PLAIN) hlld<true>(L, R, b_n, gamma, gm1, f, theta, phi);
    else ok = hlld_q<true>(L, R, b_n, gm1, A.rgm1, bsql, bsqr, cl, cr, theta, phi, f) && ok;
  }
  return ok;
}

// the face's outputs from its fluxes
template <class P>
CHQ_D void face_store(const DirView<P> &V, int lf, const P f[NFLX], P sl, P sr) {
  V.out[0][lf] = f[FD];
  V.out[1][lf] = f[FMU];
  V.out[2][lf] = f[FMV];
  V.out[3][lf] = f[FMW];
  V.out[4][lf] = f[FEN];
  // entropy flux upwinded with the mass flux (the published mean at an exact zero is zero too)
  V.out[5][lf] = f[FD] * ((f[FD] > P(0)) ? sl : sr);
  V.out[6][lf] = -f[FBY];
  V.out[7][lf] = f[FBZ];
}

// d: the direction of the view
template <int R, int S, bool CHAR, class P>
CHQ_D void face_flux(const FluxArgs<P> &A, const DirView<P> &V, int d, int lf, const P wl[8], const P wr[8], const P b_n) {
  P f[NFLX];
  const bool ok = face_solve<S, false, P>(A, V, lf, wl, wr, b_n, f);
  face_store<P>(V, lf, f, wl[7], wr[7]);
  if constexpr (S != S_HLLE) {
    if (!ok) face_plain<R, S, CHAR, P>(&A, d, lf);
  }
}

template <int R, int S, bool CHAR, class P>
__device__ __noinline__ void face_plain(const FluxArgs<P> *args, int d, int lf) {
  const FluxArgs<P> &A = *args;
  const DirView<P> V = dir_view(A, d);
  P aL[8], aR[8], wl[8], f[NFLX];
  cell_states<R, CHAR, P>(A, V, lf - V.st, aL, wl);
  cell_states<R, CHAR, P>(A, V, lf, aL, aR);
  face_solve<S, true, P>(A, V, lf, wl, aL, P(V.bn[lf]), f);
  face_store<P>(V, lf, f, wl[7], aL[7]);
}

// ---------------------------------------------------------------------------------------
// Lane mapping of the x sweep. The rows (k, j) are laid end to end, each with the cells its
// faces need (nxent = faces + XLead), and a warp takes the next 32 of them, overlapping the
// warp before by the 32 - XFaces lanes whose states only feed their neighbours. A row end thus
// costs XLead lanes instead of the rest of a warp: at 128 faces a row 89 % of the lanes emit
// faces, with warps cut at the row ends it was 81 % (64: 87 and 68 %, 256: 89 and 89 %).
//
// Faces per x-sweep warp: 31 in the per-cell form (lane 0 contributes only its right state),
// 29 in the streaming PPM form (lanes 0 and 31 contribute only their slope and interface
// value, so the states of lanes 1..30 are complete and lanes 2..30 emit faces). XLead: cells
// before (XBack) and after a row's faces.
template <int R, bool CHAR> struct XFaces {
  static constexpr bool stream = (R == R_PPM && !CHAR);
  static constexpr int v = stream ? 29 : 31;
  static constexpr int back = stream ? 2 : 1, lead = stream ? 3 : 1;
};

// row and cell of this lane's place; false past the last row
template <class P> CHQ_D bool x_place(const FluxArgs<P> &A, int wid, int per, int back, int &k, int &j, int &c) {
  const int E = A.nxent, lane = threadIdx.x & 31;
  const int base = wid * per;
  int row = base / E;
  int e = base - row * E + lane;
  while (e >= E) {
    e -= E;
    ++row;
  }
  const bool have = row < A.nxrow;
  row = min(row, A.nxrow - 1);
  const int nj = A.hi[0][1] - A.lo[0][1] + 1;
  const int q = row / nj;
  k = A.lo[0][0] + q;
  j = A.lo[0][1] + (row - q * nj);
  c = A.lo[0][2] - back + e;
  return have;
}

template <int R, int S, bool CHAR, class P>
CHQ_D void sweep_x(const FluxArgs<P> &A, int wid) {
  using X = XFaces<R, CHAR>;
  int k, j, c;
  const bool have = x_place(A, wid, X::v, X::back, k, j, c);   // this lane's cell
  const DirView<P> V = dir_view(A, 0);
  P aL[8], aR[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) { aL[n] = P(0); aR[n] = P(0); }
  const int lc = A.g.idx32(k, j, c);
  const P bnf = have ? P(ldg(V.bn + lc)) : P(0);   // loaded before the reconstruction
  if (have) cell_states<R, CHAR, P>(A, V, lc, aL, aR);
  P wl[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) wl[n] = __shfl_up_sync(0xffffffffu, aR[n], 1);
  if (have && (threadIdx.x & 31) > 0 && c >= A.lo[0][2]) face_flux<R, S, CHAR, P>(A, V, 0, lc, wl, aL, bnf);
}

// Streaming PPM (CW84, src/recon.hpp:21-78) along a row of 32 cells, one per lane. The
// reference evaluates, for face i, the limited parabolas of cells i-1 and i from their
// monotonised slopes and unlimited interface values, so each slope is evaluated three times
// and each unlimited interface value twice over a row. Here lane c evaluates its own slope
// s_c and the unlimited value at its right interface F_{c+1/2} once; the slope of cell c+1
// and the value F_{c-1/2} come from the neighbouring lanes by warp shuffle. The operands of
// every expression are the reference's, so the limited states are bitwise the same.
template <int S, class P>
CHQ_D void sweep_x_ppm(const FluxArgs<P> &A, int wid) {
  using X = XFaces<R_PPM, false>;
  const int lane = threadIdx.x & 31;
  int k, j, c;
  const bool have = x_place(A, wid, X::v, X::back, k, j, c);   // this lane's cell
  // lanes past the row's last face (and lane 0's stencil at the row start) read clamped
  // indices inside the row; their states are never used
  const int last = A.g.ni - 1;
  const int cm2 = max(c - 2, 0), cm1 = max(c - 1, 0), c0 = min(c, last), cp1 = min(c + 1, last),
            cp2 = min(c + 2, last);
  const int base = A.g.idx32(k, j, 0);
  const DirView<P> V = dir_view(A, 0);
  const P bnf = P(ldg(V.bn + base + c0));   // this lane's face-normal field, loaded before the reconstruction
  P aL[8], aR[8], qc[8], p5[5], um1 = P(0), up1 = P(0);
  // every stencil load of the lane is issued before any arithmetic: a warp handles one row
  // segment, so nothing else hides the latency of its loads (measured: the x sweep ~20 %
  // faster in FP64 than with the loads interleaved with each quantity's reconstruction)
  P QM[8], Q0[8], QP[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const P *src = V.src[n] + base;
    QM[n] = ldg(src + cm1);
    Q0[n] = ldg(src + c0);
    QP[n] = ldg(src + cp1);
  }
  const P pm2 = ldg(V.src[4] + base + cm2), pp2 = ldg(V.src[4] + base + cp2);
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const P qm = QM[n], q0 = Q0[n], qp = QP[n];
    const P sc = mc_slope2(qm, q0, qp);
    const P sp = __shfl_down_sync(0xffffffffu, sc, 1);    // s_{c+1}
    const P fp = ppm_face2(q0, qp, sc, sp);                 // F_{c+1/2}, unlimited
    P l = __shfl_up_sync(0xffffffffu, fp, 1), r = fp;     // F_{c-1/2}
    ppm_limit(q0, l, r);
    aL[n] = l;
    aR[n] = r;
    qc[n] = q0;
    if (n == 1) { um1 = qm; up1 = qp; }
    if (n == 4) { p5[0] = pm2; p5[1] = qm; p5[2] = q0; p5[3] = qp; p5[4] = pp2; }
  }
  finish_states<R_PPM, P>(A, aL, aR, qc, p5, um1, up1);
  P wl[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) wl[n] = __shfl_up_sync(0xffffffffu, aR[n], 1);
  if (have && lane >= 2 && lane <= 30 && c >= A.lo[0][2] && c <= A.hi[0][2]) face_flux<R_PPM, S, false, P>(A, V, 0, base + c, wl, aL, bnf);
}

// Streaming PPM along a y/z march. Each thread's shared-memory column keeps, per quantity,
// q_c, q_{c+1}, q_{c+2} (the last copied asynchronously one cell ahead), the slope s_c and
// the unlimited interface value F_{c-1/2} computed at the previous cell; the velocity adds
// u_{c-1} and the pressure p_{c-2}, p_{c-1} (flattening). A cell then evaluates one slope
// (s_{c+1}) and one interface value (F_{c+1/2}) per quantity instead of three and two, with
// the reference's operands (bitwise the same limited states as the per-cell form). In FP64
// the face-normal field of the next face is copied asynchronously one cell ahead as well,
// into one of two slots per thread (alternating, so a copy never lands in the slot being
// read), instead of a load at the Riemann solve.
struct PpmWin {
  static constexpr int nslot = 43;
  enum : int { Q0 = 0, Q1 = 1, Q2 = 2, S = 3, F = 4, X1 = 5, X2 = 6 };
  CHQ_HD static constexpr int off(int n) {
    return (n == 0) ? 0 : (n == 1) ? 5 : (n == 2) ? 11 : (n == 3) ? 16 : (n == 4) ? 21 : (n == 5) ? 28 : (n == 6) ? 33 : 38;
  }
};

// TMA (FP64 only, maps and mbar given): instead of one cp.async per quantity and thread, one
// lane of the warp issues, one cell ahead, eight bulk tensor copies of the next cell's 32-wide
// row of each quantity straight into the warp's rows of the window's q_{c+2} slots; the warp
// waits on its mbarrier's phase. Same slots, same values: the states are bitwise those of the
// cp.async form.
template <int S, class P, bool TMA = false>
CHQ_D void sweep_yz_ppm(const FluxArgs<P> &A, int d, int blk, P *park, P *win, const YzMaps *maps = nullptr,
                        unsigned long long *mbar = nullptr) {
  unsigned mask = 0xffffffffu;
  bool leader = false;
  int i, outer, seg, chunk = 0;
  if constexpr (TMA) {
    // whole 32-cell row segments: one warp per i chunk, outer index and segment (blk: the warp)
    chunk = blk % A.nchunk;
    const int rest = blk / A.nchunk;
    seg = rest % A.nseg[d];
    outer = rest / A.nseg[d];
    i = 32 * chunk + (threadIdx.x & 31);
    const bool act = !(i < A.lo[d][2] || i > A.hi[d][2]);
    mask = __ballot_sync(0xffffffffu, act);
    leader = act && ((threadIdx.x & 31) == __ffs(mask) - 1);
    if (!act) return;
  } else {
    if (!yz_place(A, d, blk, i, outer, seg)) return;
  }
  const int sweep_lo = (d == 1) ? A.lo[1][1] : A.lo[2][0];
  const int sweep_hi = (d == 1) ? A.hi[1][1] : A.hi[2][0];
  const int f0 = sweep_lo + A.slen[d] * seg;
  const int f1 = min(f0 + A.slen[d] - 1, sweep_hi);
  const DirView<P> V = dir_view(A, d);
  const int st = V.st;
  int lc = (d == 1) ? A.g.idx32(A.lo[1][0] + outer, f0 - 1, i) : A.g.idx32(f0 - 1, A.lo[2][1] + outer, i);
  const int t = threadIdx.x;
  P *col = win + t;
  constexpr bool PFB = (sizeof(P) == 8);
  double *bnw = reinterpret_cast<double *>(win + PpmWin::nslot * kYzThreads) + t;
  // TMA staging: this warp's mbarrier, its rows of the q_{c+2} slots, the tensor coordinates
  unsigned long long *mb = TMA ? mbar + (t >> 5) : nullptr;
  unsigned phase = 0;
  const int outer_idx = (d == 1) ? A.lo[1][0] + outer : A.lo[2][1] + outer;
  auto issue = [&](int pos) {   // the rows of the cell at sweep position pos, all 8 quantities
    mbar_expect_tx(mb, 8u * 32u * (unsigned)sizeof(P));
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      // component of quantity n in w (0, 1, 2, 3, 4, 7) or bcc (5, 6), as dir_view orders them
      const int comp = (n == 0) ? IDN : (n == 1) ? IVX + d : (n == 2) ? IVX + (d + 1) % 3 : (n == 3) ? IVX + (d + 2) % 3
                     : (n == 4) ? IPR : (n == 5) ? (d + 1) % 3 : (n == 6) ? (d + 2) % 3 : IENT;
      const CUtensorMap *map = (n == 5 || n == 6) ? &maps->b : &maps->w;
      P *row = win + (PpmWin::off(n) + PpmWin::Q2) * kYzThreads + (t & ~31);
      if (d == 1) tma_load_4d(row, map, 32 * chunk, pos, outer_idx, comp, mb);
      else tma_load_4d(row, map, 32 * chunk, outer_idx, pos, comp, mb);
    }
  };
  if constexpr (TMA) {
    if (leader) mbar_init(mb, 1);
    __syncwarp(mask);
  }
#define CHQ_SLOT(n, k) col[(PpmWin::off(n) + PpmWin::k) * kYzThreads]
  // cell f0-1: its slope, its left interface value and the window, from direct loads
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const P *src = V.src[n] + lc;
    const P qm2 = ldg(src - 2 * st), qm1 = ldg(src - st), q0 = ldg(src), qp1 = ldg(src + st);
    const P sm = mc_slope2(qm2, qm1, q0), sc = mc_slope2(qm1, q0, qp1);
    CHQ_SLOT(n, Q0) = q0;
    CHQ_SLOT(n, Q1) = qp1;
    CHQ_SLOT(n, S) = sc;
    CHQ_SLOT(n, F) = ppm_face2(qm1, q0, sm, sc);
    if (n == 1) CHQ_SLOT(1, X1) = qm1;
    if (n == 4) {
      CHQ_SLOT(4, X1) = qm2;
      CHQ_SLOT(4, X2) = qm1;
    }
    if constexpr (!TMA) cp_async_elem(&CHQ_SLOT(n, Q2), src + 2 * st);
  }
  cp_async_commit();
  if constexpr (TMA) {
    if (leader) issue(f0 + 1);
  }
  P wl[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) wl[n] = P(0);
  for (int f = f0 - 1; f <= f1; ++f, lc += st) {
    cp_async_wait_all();
    if constexpr (TMA) {
      // q_{c+2} rows of this cell: the warp gives up together if the copies never land
      const bool ok = __all_sync(mask, mbar_wait(mb, phase & 1u));
      ++phase;
      if (!ok) {
        if (leader && A.err) atomicExch(A.err, 3);
        return;
      }
    }
    const bool pre = (f < f1);
    P bnv = P(0);
    if constexpr (PFB) {
      if (f >= f0) bnv = P(bnw[(f & 1) * kYzThreads]);
      if (pre) cp_async_elem(bnw + ((f + 1) & 1) * kYzThreads, V.bn + lc + st);
    }
    P aL[8], aR[8], qc[8], p5[5], um1 = P(0), up1 = P(0);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const P q0 = CHQ_SLOT(n, Q0), q1 = CHQ_SLOT(n, Q1), q2 = CHQ_SLOT(n, Q2);
      const P sc = CHQ_SLOT(n, S), fm = CHQ_SLOT(n, F);
      const P sp = mc_slope2(q0, q1, q2);          // s_{c+1}
      const P fp = ppm_face2(q0, q1, sc, sp);      // F_{c+1/2}, unlimited
      P l = fm, r = fp;
      ppm_limit(q0, l, r);
      aL[n] = l;
      aR[n] = r;
      qc[n] = q0;
      if (n == 1) {
        um1 = CHQ_SLOT(1, X1);
        up1 = q1;
        CHQ_SLOT(1, X1) = q0;
      }
      if (n == 4) {
        p5[0] = CHQ_SLOT(4, X1);
        p5[1] = CHQ_SLOT(4, X2);
        p5[2] = q0;
        p5[3] = q1;
        p5[4] = q2;
        CHQ_SLOT(4, X1) = p5[1];
        CHQ_SLOT(4, X2) = q0;
      }
      CHQ_SLOT(n, Q0) = q1;
      CHQ_SLOT(n, Q1) = q2;
      CHQ_SLOT(n, S) = sp;
      CHQ_SLOT(n, F) = fp;
      if constexpr (!TMA) {
        if (pre) cp_async_elem(&CHQ_SLOT(n, Q2), V.src[n] + lc + 3 * st);
      }
    }
    cp_async_commit();
    if constexpr (TMA) {
      if (pre) {
        __syncwarp(mask);   // every lane has read its q_{c+2} slots before the copies overwrite them
        if (leader) {
          fence_proxy_async();
          issue(f + 3);
        }
      }
    }
    finish_states<R_PPM, P>(A, aL, aR, qc, p5, um1, up1);
#pragma unroll
    for (int n = 0; n < 8; ++n) park[n * kYzThreads + t] = aR[n];
    if (f >= f0) {
      face_flux<R_PPM, S, false, P>(A, V, d, lc, wl, aL, PFB ? bnv : P(V.bn[lc]));
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) wl[n] = park[n * kYzThreads + t];
  }
#undef CHQ_SLOT
}

// y (d = 1) or z (d = 2) sweep: one code copy, direction in the view. The right state
// carried to the next face is parked in this thread's shared-memory slot during the
// Riemann solve, which keeps it out of the registers at the solver's peak. With WIN the
// stencil comes from the thread's marching window in shared memory (WindowStencil): one
// asynchronous copy per quantity and cell, issued a whole cell ahead, instead of 2RE+1
// cached loads whose lines a y/z march cannot keep in L1.
template <int R, int S, bool CHAR, bool WIN, class P>
CHQ_D void sweep_yz(const FluxArgs<P> &A, int d, int blk, P *park, P *win) {
  if constexpr (R == R_PPM && !CHAR && WIN) {
    sweep_yz_ppm<S, P>(A, d, blk, park, win);
    return;
  }
  int i, outer, seg;
  if (!yz_place(A, d, blk, i, outer, seg)) return;
  const int sweep_lo = (d == 1) ? A.lo[1][1] : A.lo[2][0];
  const int sweep_hi = (d == 1) ? A.hi[1][1] : A.hi[2][0];
  const int f0 = sweep_lo + A.slen[d] * seg;
  const int f1 = min(f0 + A.slen[d] - 1, sweep_hi);
  const DirView<P> V = dir_view(A, d);
  // cell f0-1 first (its right state only), then cell f and face f for f = f0..f1; one copy
  // of the cell code in the loop keeps the kernel's instruction footprint small
  int lc = (d == 1) ? A.g.idx32(A.lo[1][0] + outer, f0 - 1, i) : A.g.idx32(f0 - 1, A.lo[2][1] + outer, i);
  P wl[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) wl[n] = P(0);
  const int t = threadIdx.x;
  constexpr int RE = Reach<R>::v;
  constexpr bool use_win = WIN && (RE > 0);
  P *col = use_win ? win + t : nullptr;
  // FP64: the next face's normal field copied one cell ahead into two alternating slots
  // after the window (as in the streaming-PPM march)
  constexpr bool PFB = use_win && (sizeof(P) == 8);
  double *bnw = PFB ? reinterpret_cast<double *>(win + 8 * (2 * RE + 1) * kYzThreads) + t : nullptr;
  if constexpr (use_win) {
    // window of cell f0-1: q[c-RE .. c+RE-1] now, q[c+RE] asynchronously
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      P *w = col + n * (2 * RE + 1) * kYzThreads;
#pragma unroll
      for (int m = 0; m < 2 * RE; ++m) w[m * kYzThreads] = ldg(V.src[n] + lc + (m - RE) * V.st);
      cp_async_elem(w + 2 * RE * kYzThreads, V.src[n] + lc + RE * V.st);
    }
    cp_async_commit();
  }
  for (int f = f0 - 1; f <= f1; ++f, lc += V.st) {
    P aL[8], aR[8];
    P bnv = P(0);
    if constexpr (use_win) {
      cp_async_wait_all();
      if constexpr (PFB) {
        if (f >= f0) bnv = P(bnw[(f & 1) * kYzThreads]);
        if (f < f1) cp_async_elem(bnw + ((f + 1) & 1) * kYzThreads, V.bn + lc + V.st);
      }
      cell_states_from<R, CHAR, P>(A, V, lc, aL, aR, WindowStencil<RE, P>{col, V, lc, f < f1});
      cp_async_commit();
    } else {
      cell_states<R, CHAR, P>(A, V, lc, aL, aR);
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) park[n * kYzThreads + t] = aR[n];
    if (f >= f0) {
      face_flux<R, S, CHAR, P>(A, V, d, lc, wl, aL, PFB ? bnv : P(V.bn[lc]));
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) wl[n] = park[n * kYzThreads + t];
  }
}

// Resident 128-thread blocks per SM the x-sweep kernel is compiled for (register cap), in two
// variants that the autotuner chooses between per scheme, precision and mesh: V = 0 at 4
// (FP64, 128 registers) / 8 (FP32, 64 registers) blocks, V = 1 at 5 / 10 blocks (more resident
// warps, fewer registers, some spilling to L1). Since the solver has no branches its two sides
// and the quantities interleave, so registers hide more latency than warps do: FP64 PPM flux
// launches at 256^3 measured 3.86 ms with 5 blocks and 3.77 ms with 4 (3: 3.70 against 3.54 in
// the final build), the mixed form 2.18 / 2.13 ms with 10 / 8.
#ifndef CHQ_FLUX_MINB_D
#define CHQ_FLUX_MINB_D 4
#endif
#ifndef CHQ_FLUX_MINB_F
#define CHQ_FLUX_MINB_F 8
#endif
template <class P, int V = 0> struct FluxMinBlocks {
  static constexpr int v = (sizeof(P) == 8) ? CHQ_FLUX_MINB_D + V : CHQ_FLUX_MINB_F + 2 * V;
};
constexpr int kFluxXVariants = 2;

// Single-mesh launches split by sweep: the x-sweep kernel needs no shared window, so it keeps
// the full L1 and the register cap above; the y/z kernel holds 8 + 8(2RE+1) shared columns
// per thread (53 KB per block in FP64 PPM). 3 blocks (168 registers) beat 4 (128 registers) by
// 6 % and 2 by 9 % in FP64 PPM at 256^3, although 4 would fit: see the x sweep's caps.
#ifndef CHQ_FLUXYZ_MINB_D
#define CHQ_FLUXYZ_MINB_D 3
#endif
#ifndef CHQ_FLUXYZ_MINB_F
#define CHQ_FLUXYZ_MINB_F 6
#endif
template <class P> struct FluxYzMinBlocks { static constexpr int v = (sizeof(P) == 8) ? CHQ_FLUXYZ_MINB_D : CHQ_FLUXYZ_MINB_F; };

template <int R, class P> __host__ __device__ constexpr size_t flux_yz_smem() {
  // park (8) + window: streaming PPM 43 slots (the characteristic PPM form uses 40 of them),
  // otherwise 8 quantities x (2 reach + 1); in FP64 every windowed march adds two face-field slots
  return (size_t)(8 + ((R == R_PPM) ? PpmWin::nslot : (Reach<R>::v > 0) ? 8 * (2 * Reach<R>::v + 1) : 0)) *
             kYzThreads * sizeof(P) +
         ((Reach<R>::v > 0 && sizeof(P) == 8) ? 2 * kYzThreads * sizeof(double) : 0);
}

template <int R, int S, bool CHAR, class P, int V = 0>
__global__ void __launch_bounds__(128, (FluxMinBlocks<P, V>::v)) flux_x_kernel(const __grid_constant__ FluxArgs<P> A) {
  // (it shares no data with the y/z launch, but reads what con2prim wrote before that: only its
  // own wait makes those writes visible to it)
  pdl_begin();
  if (A.skip && *A.skip) return;
  const int wid = (int)blockIdx.x * 4 + (int)(threadIdx.x >> 5);
  if (wid < A.nxwarp) {
    if constexpr (R == R_PPM && !CHAR) sweep_x_ppm<S, P>(A, wid);
    else sweep_x<R, S, CHAR, P>(A, wid);
  }
}

template <int R, int S, bool CHAR, class P>
__global__ void __launch_bounds__(kYzThreads, FluxYzMinBlocks<P>::v) flux_yz_kernel(const __grid_constant__ FluxArgs<P> A) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char flux_dsm[];
  P *park = reinterpret_cast<P *>(flux_dsm);
  P *win = park + 8 * kYzThreads;
  if (A.skip && *A.skip) return;
  const int b = (int)blockIdx.x;
  if (b < A.nblk[2]) sweep_yz<R, S, CHAR, true, P>(A, 2, b, park, win);
  else if (b < A.nblk[2] + A.nblk[1]) sweep_yz<R, S, CHAR, true, P>(A, 1, b - A.nblk[2], park, win);
}

// The FP64 streaming-PPM y/z kernel with TMA staging (FluxArgs::yzvar = 1): dynamic shared
// memory of flux_yz_kernel plus one mbarrier per warp; the tensor maps are kernel parameters.
constexpr size_t flux_yz_tma_smem() { return flux_yz_smem<R_PPM, double>() + (kYzThreads / 32) * sizeof(unsigned long long); }

// its warps of direction d
template <class P> CHQ_HD int tma_warps(const FluxArgs<P> &A, int d) {
  const int o = (d == 1) ? 0 : 1;   // the outer index: k for y sweeps, j for z sweeps
  return A.nblk[d] ? A.nchunk * (A.hi[d][o] - A.lo[d][o] + 1) * A.nseg[d] : 0;
}

template <int S>
__global__ void __launch_bounds__(kYzThreads, FluxYzMinBlocks<double>::v)
    flux_yz_tma_kernel(const __grid_constant__ FluxArgs<double> A, const __grid_constant__ YzMaps maps) {
  pdl_begin();
  extern __shared__ __align__(128) unsigned char flux_tma_dsm[];
  double *park = reinterpret_cast<double *>(flux_tma_dsm);
  double *win = park + 8 * kYzThreads;
  unsigned long long *mbar = reinterpret_cast<unsigned long long *>(flux_tma_dsm + flux_yz_smem<R_PPM, double>());
  if (A.skip && *A.skip) return;
  const int wid = (int)blockIdx.x * (kYzThreads / 32) + (int)(threadIdx.x >> 5);
  const int nz = tma_warps(A, 2), nyz = nz + tma_warps(A, 1);
  if (wid < nz) sweep_yz_ppm<S, double, true>(A, 2, wid, park, win, &maps, mbar);
  else if (wid < nyz) sweep_yz_ppm<S, double, true>(A, 1, wid - nz, park, win, &maps, mbar);
}

// batched forms: the blocks of many meshes in one launch per sweep kind (chq_batch); each
// block copies its mesh's arguments to shared memory first
template <int R, int S, bool CHAR, class P, int V = 0>
__global__ void __launch_bounds__(128, (FluxMinBlocks<P, V>::v)) flux_x_batched(const FluxArgs<P> *args, const BatchSlot *slots, int n) {
  pdl_begin();
  __shared__ __align__(16) unsigned char sa[sizeof(FluxArgs<P>)];
  const int j = batch_job(slots, n, blockIdx.x);
  const FluxArgs<P> &A = stage_args(args, j, sa);
  if (A.skip && *A.skip) return;
  const int wid = (int)(blockIdx.x - slots[j].off) * 4 + (int)(threadIdx.x >> 5);
  if (wid < A.nxwarp) {
    if constexpr (R == R_PPM && !CHAR) sweep_x_ppm<S, P>(A, wid);
    else sweep_x<R, S, CHAR, P>(A, wid);
  }
}

template <int R, class P> __host__ __device__ constexpr size_t flux_yz_batched_smem() {
  return flux_yz_smem<R, P>() + (sizeof(FluxArgs<P>) + 15) / 16 * 16;
}

template <int R, int S, bool CHAR, class P>
__global__ void __launch_bounds__(kYzThreads, FluxYzMinBlocks<P>::v) flux_yz_batched(const FluxArgs<P> *args, const BatchSlot *slots, int n) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char flux_dsm[];
  P *park = reinterpret_cast<P *>(flux_dsm);
  P *win = park + 8 * kYzThreads;
  const int j = batch_job(slots, n, blockIdx.x);
  const FluxArgs<P> &A = stage_args(args, j, flux_dsm + flux_yz_smem<R, P>());
  if (A.skip && *A.skip) return;
  const int b = (int)(blockIdx.x - slots[j].off);
  if (b < A.nblk[2]) sweep_yz<R, S, CHAR, true, P>(A, 2, b, park, win);
  else if (b < A.nblk[2] + A.nblk[1]) sweep_yz<R, S, CHAR, true, P>(A, 1, b - A.nblk[2], park, win);
}

}  // namespace chq
