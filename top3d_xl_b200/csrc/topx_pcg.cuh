// Scalars of the PCG on the device: start, stop test, and the decision at the head of the kernel that takes the
// residual pass's sums.
#pragma once

#include "topx_kernels.cuh"

namespace topx {

__device__ __forceinline__ void pcg_start(PcgScalars* sc, double bb, double tol, int maxIT) {
  sc->normB = sqrt(bb);
  sc->tol = tol;
  sc->maxIT = maxIT;
  sc->its = 0;
  sc->done = 0;
  sc->first = 1;
  sc->beta = 0.0;
}
// after step number its
__device__ __forceinline__ void pcg_stop_test(PcgScalars* sc, double rr, int its) {
  sc->rr = rr;
  sc->resnorm = sqrt(rr) / sc->normB;
  sc->first = 0;
  if (sc->resnorm < sc->tol)
    sc->done = 1;
  else if (its >= sc->maxIT)
    sc->done = 2;
}
// The solve had ended before the residual pass whose result this kernel takes.  With parts.rr given, pcg_decide writes
// done in this launch, so that its CTAs (and the warps of one) could read different values of it: ended is the residual
// pass's copy.  No word that a launch of the PCG reads is written by another CTA of that launch.
__device__ __forceinline__ bool pcg_ended(const PcgScalars* sc, const PcgParts& parts) {
  return (parts.rr.n ? sc->ended : sc->done) != 0;
}
// parts.rr given: sums the residual pass's r'r (b'b) and r'D r.  Every CTA takes the same decision, the first one writes
// it down.  True: the solve has ended.
__device__ __forceinline__ bool pcg_decide(PcgScalars* sc, const PcgParts& parts, bool init, double tol, int maxIT) {
  if (!parts.rr.n) return false;
  const bool one = blockIdx.x + blockIdx.y + blockIdx.z == 0, first = one && threadIdx.x + threadIdx.y == 0;
  const double rr = parts_sum(parts.rr);
  if (one) {
    const double rd = parts_sum(parts.rd);
    if (first) sc->rdr = rd;
    if (first && init) pcg_start(sc, rr, tol, maxIT);
  }
  if (init) return false;
  const int its = sc->its_next;
  if (first) {
    sc->its = its;
    pcg_stop_test(sc, rr, its);
  }
  return sqrt(rr) / sc->normB < sc->tol || its >= sc->maxIT;
}

}  // namespace topx
