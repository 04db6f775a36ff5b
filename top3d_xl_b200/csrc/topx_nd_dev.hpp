// Device buffers of the nested-dissection factorisation of the coarsest level (topx_nd.hpp) and
// its launches (topx_nd.cu).
#pragma once

#include <cuda_runtime.h>

#include "topx_kernels.cuh"
#include "topx_nd.hpp"

namespace topx {

struct NDDevice {
  const NDFront* fronts = nullptr;
  const NDTask* tasks = nullptr;
  const NDAsm* asmb = nullptr;
  const int64_t* pad = nullptr;
  const int32_t* upd_map = nullptr;
  const int32_t* sep_dof = nullptr;
  const int32_t* upd_dof = nullptr;
  const int32_t* src0 = nullptr;
  const int32_t* src1 = nullptr;
  double* pool = nullptr;   // tiles (FP64)
  double* scr = nullptr;    // P^-1 and R_j tiles of the level being swept
  double* wvec = nullptr;   // per position: F11^-1 f1 and the update vectors
  double* part = nullptr;   // per solve task: partial sums of its chunk (64)
  unsigned* cnt = nullptr;  // per output tile: chunks done (zero between launches)
  // coop_ctas > 0: the solve runs as one persistent dataflow launch of this many CTAs, over the
  // tasks in dependency order (NDPlan::flow) with 2 x fronts counters and the control words
  int coop_ctas = 0;
  const NDTask* flow = nullptr;
  unsigned* flow_done = nullptr;
  CoopControl* ctl = nullptr;
  // assembly, extend-add and the sweep of every front: pool <- the factor of the coarsest
  // matrix whose element operators (576 per dense element of grid g) are Ks
  void factor(cudaStream_t st, const NDPlan& P, Grid g, const double* Ks) const;
  // x = K^-1 b on the coarsest grid's SoA DOF vectors; tiles: pool or an FP32 copy of it.  With
  // sc given, every launch returns at once once sc->done is set (a converged PCG).
  template <typename T, typename TM>
  void solve(cudaStream_t st, const NDPlan& P, const TM* tiles, const T* b, T* x, const PcgScalars* sc) const;
};

// The coarse part of the V-cycle of a small grid in one launch (small_coarse): the x and z passes of the level-1
// restriction, the restriction to the coarsest level, its solve with the one front's inverse, and the prolongation
// to level 2.  TC: the preconditioner's type.
template <typename TC>
struct SmallCoarse {
  const double* tmp;    // y pass of the level-1 restriction
  Grid g0, g1, g2;      // levels 1, 2 and 3 (the coarsest)
  TC *r1, *r2, *x2, *x1;
  double* r1_64;        // FP64 copy of r1 (null when TC is double)
  const TC* d1;
  const uint8_t* present1;
  NDFront front;
  const TC* tiles;
  const int32_t* sep_dof;
  PcgScalars* sc;
  PcgParts parts;       // inside the PCG (dot), else empty
  bool dot, init;
  double tol, omega;
  int maxIT;
};
constexpr int kSmallCoarseCtas = 16;  // one cluster, a tile row of the front each
bool small_coarse(const NDPlan& P, int levels, Grid g1);
template <typename TC>
void launch_small_coarse(cudaStream_t st, const SmallCoarse<TC>& a);

// kernel attributes (once per device; outside stream capture)
void prepare_nd_kernels();
// CTAs of the persistent solve on the current device (all resident), or 0 when the device has
// no cooperative launch
int nd_solve_coop_ctas();

}  // namespace topx
