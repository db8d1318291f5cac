// chasqui_b200 — instantiation unit of the face-flux kernel for one (precision, scheme).
// Compiled once per pair with -DCHQ_P=<double|float> -DCHQ_R=<0..4>.
#include <cstring>
#include "chq_launch.h"

#ifndef CHQ_P
#error "CHQ_P must be defined (double or float)"
#endif
#ifndef CHQ_R
#error "CHQ_R must be defined (reconstruction enum)"
#endif

namespace chq {

// per-device one-time opt-in to the dynamic shared memory of a y/z kernel
template <class K>
static cudaError_t allow_smem(K kern, size_t smem, bool *ready) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && ready[dev]) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess && dev >= 0 && dev < 64) ready[dev] = true;
  return e;
}

// In a captured cycle the x sweep is a parallel node of the y/z sweeps up to this many x blocks (in
// cycles without a graph it runs on the mesh's second stream): its blocks fill what the y/z launch's last waves leave idle. us a cycle in series and in parallel: OT 64^2
// 94 and 82, 256^2 154 and 122, 512^2 279 and 269, 128^3 2313 and 2288 (mixed 96, 87 at 128^2, 221, 207
// at 512^2, 1674, 1584 at 128^3); 256^3, whose two launches are many waves each, 16 635 and 16 660
// (11 255 and 11 301).
constexpr unsigned kForkXBlocks = 148 * 256;
// A batch's march fills whole waves already, so only its small launches gain: 3 x 64^2 137 and 123 us,
// 4 x 32^3 426 and 393 (mixed 320, 299); 24 x 32^3 (8950 blocks) 2032 and 2044 (mixed 1479, 1462).
constexpr unsigned kForkXBlocksBatched = 148 * 20;
static bool fork_begin(const FluxFork *f, unsigned nyz, unsigned nx, unsigned most, cudaStream_t s, cudaError_t &e) {
  e = cudaSuccess;
  if (!f || !nyz || !nx || nx > most) return false;
  e = cudaEventRecord(f->fork, s);   // the branch starts where the y/z sweeps do
  if (e == cudaSuccess) e = cudaStreamWaitEvent(f->side, f->fork, 0);
  return true;
}
static cudaError_t fork_join(const FluxFork *f, cudaStream_t s) {
  cudaError_t e = cudaEventRecord(f->join, f->side);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(s, f->join, 0);
  pdl_plain = true;   // the next launch depends on both sweeps
  return e;
}

// y/z sweeps (shared marching window, dynamic shared memory) then the x-sweep, one stream
template <int S, bool C>
static cudaError_t go(const FluxArgs<CHQ_P> &a, const FluxFork *f, cudaStream_t s) {
  const unsigned nyz = (unsigned)(a.nblk[1] + a.nblk[2]), nx = (unsigned)((a.nxwarp + 3) / 4);
  cudaError_t ef;
  const bool forked = fork_begin(f, nyz, nx, kForkXBlocks, s, ef);
  if (ef != cudaSuccess) return ef;
  bool yz_done = false;
  if constexpr (CHQ_R == R_PPM && !C && sizeof(CHQ_P) == 8) {
    // TMA staging of the streaming-PPM march (picked by the autotuner; FP64 only)
    if (nyz && a.yzvar == 1 && a.yzmaps) {
      constexpr size_t smem = flux_yz_tma_smem();
      static bool ready_tma[64] = {};
      const cudaError_t ea = allow_smem(flux_yz_tma_kernel<S>, smem, ready_tma);
      if (ea != cudaSuccess) return ea;
      YzMaps maps;
      std::memcpy(&maps, a.yzmaps, sizeof(maps));
      constexpr int wpb = kYzThreads / 32;
      pdl(flux_yz_tma_kernel<S>, (tma_warps(a, 1) + tma_warps(a, 2) + wpb - 1) / wpb, kYzThreads, smem, s, a, maps);
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      yz_done = true;
    }
  }
  if (nyz && !yz_done) {
    constexpr size_t smem = flux_yz_smem<CHQ_R, CHQ_P>();
    static bool ready[64] = {};
    const cudaError_t ea = allow_smem(flux_yz_kernel<CHQ_R, S, C, CHQ_P>, smem, ready);
    if (ea != cudaSuccess) return ea;
    pdl(flux_yz_kernel<CHQ_R, S, C, CHQ_P>, nyz, kYzThreads, smem, s, a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (nx) {
    pdl_plain = forked;   // the branch's first launch
    cudaStream_t sx = forked ? f->side : s;
    if (a.xvar) pdl(flux_x_kernel<CHQ_R, S, C, CHQ_P, 1>, nx, 128, 0, sx, a);
    else pdl(flux_x_kernel<CHQ_R, S, C, CHQ_P, 0>, nx, 128, 0, sx, a);
  }
  if (forked && (ef = fork_join(f, s)) != cudaSuccess) return ef;
  return cudaGetLastError();
}

template <>
cudaError_t launch_flux<CHQ_P, CHQ_R>(const FluxArgs<CHQ_P> &a, int rsolver, int charac, const FluxFork *f, cudaStream_t s) {
  const bool c = (charac != 0) && (CHQ_R != R_DC);
  switch (rsolver) {
    case S_HLLE: return c ? go<S_HLLE, true>(a, f, s) : go<S_HLLE, false>(a, f, s);
    case S_HLLD: return c ? go<S_HLLD, true>(a, f, s) : go<S_HLLD, false>(a, f, s);
    case S_LHLLD: return c ? go<S_LHLLD, true>(a, f, s) : go<S_LHLLD, false>(a, f, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int S, bool C>
static cudaError_t gob(const FluxArgs<CHQ_P> *a, const BatchSlot *sx, const BatchSlot *syz, int n, unsigned nbx,
                       unsigned nbyz, int xvar, const FluxFork *f, cudaStream_t s) {
  cudaError_t ef;
  const bool forked = fork_begin(f, nbyz, nbx, kForkXBlocksBatched, s, ef);
  if (ef != cudaSuccess) return ef;
  if (nbyz) {
    constexpr size_t smem = flux_yz_batched_smem<CHQ_R, CHQ_P>();
    static bool ready[64] = {};
    const cudaError_t e = allow_smem(flux_yz_batched<CHQ_R, S, C, CHQ_P>, smem, ready);
    if (e != cudaSuccess) return e;
    pdl(flux_yz_batched<CHQ_R, S, C, CHQ_P>, nbyz, kYzThreads, smem, s, a, syz, n);
    const cudaError_t e2 = cudaGetLastError();
    if (e2 != cudaSuccess) return e2;
  }
  if (nbx) {
    pdl_plain = forked;
    cudaStream_t x = forked ? f->side : s;
    if (xvar) pdl(flux_x_batched<CHQ_R, S, C, CHQ_P, 1>, nbx, 128, 0, x, a, sx, n);
    else pdl(flux_x_batched<CHQ_R, S, C, CHQ_P, 0>, nbx, 128, 0, x, a, sx, n);
  }
  if (forked && (ef = fork_join(f, s)) != cudaSuccess) return ef;
  return cudaGetLastError();
}

template <>
cudaError_t launch_flux_batched<CHQ_P, CHQ_R>(const FluxArgs<CHQ_P> *a, const BatchSlot *sx, const BatchSlot *syz, int n,
                                               int rsolver, int charac, unsigned nbx, unsigned nbyz, int xvar,
                                               const FluxFork *f, cudaStream_t s) {
  if (nbx == 0 && nbyz == 0) return cudaSuccess;
  const bool c = (charac != 0) && (CHQ_R != R_DC);
  switch (rsolver) {
    case S_HLLE: return c ? gob<S_HLLE, true>(a, sx, syz, n, nbx, nbyz, xvar, f, s) : gob<S_HLLE, false>(a, sx, syz, n, nbx, nbyz, xvar, f, s);
    case S_HLLD: return c ? gob<S_HLLD, true>(a, sx, syz, n, nbx, nbyz, xvar, f, s) : gob<S_HLLD, false>(a, sx, syz, n, nbx, nbyz, xvar, f, s);
    case S_LHLLD: return c ? gob<S_LHLLD, true>(a, sx, syz, n, nbx, nbyz, xvar, f, s) : gob<S_LHLLD, false>(a, sx, syz, n, nbx, nbyz, xvar, f, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int S, bool C>
static int regs() {
  cudaFuncAttributes at{};
  if (cudaFuncGetAttributes(&at, flux_yz_kernel<CHQ_R, S, C, CHQ_P>) != cudaSuccess) return -1;
  return at.numRegs;
}

template <>
int flux_regs<CHQ_P, CHQ_R>(int rsolver, int charac) {
  const bool c = (charac != 0) && (CHQ_R != R_DC);
  switch (rsolver) {
    case S_HLLE: return c ? regs<S_HLLE, true>() : regs<S_HLLE, false>();
    case S_HLLD: return c ? regs<S_HLLD, true>() : regs<S_HLLD, false>();
    case S_LHLLD: return c ? regs<S_LHLLD, true>() : regs<S_LHLLD, false>();
    default: return -1;
  }
}

}  // namespace chq
