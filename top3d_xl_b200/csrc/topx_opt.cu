// Optimiser-side kernels of the TOP3D_XL B200 path: objective/sensitivities
// (TOP3D_XL.m:124-130), OC bisection (TOP3D_XL.m:145-163), MMA subproblem and
// dual interior-point steps (TOP3D_XL.m:1804-2049) and the Heaviside chain of
// the LOCAL driver (TOP3D_XL.m:333-382).
#include "topx_kernels.cuh"
#include "topx_opt.cuh"

#include <algorithm>

namespace topx {

static inline unsigned grid1d(int64_t n, int threads, int cap = 148 * 16) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return unsigned(b);
}

template <typename T>
__global__ void k_scatter_elems(const double* __restrict__ src, const int32_t* __restrict__ emb0, int64_t Ne,
                                T* __restrict__ dst) {
  pdl_wait();
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x)
    dst[emb0[e]] = T(src[e]);
}
template <typename T>
void launch_scatter_elems_t(cudaStream_t st, const double* src, const int32_t* eleMapBack0, int64_t Ne, T* dstE) {
  launch_pdl(st, k_scatter_elems<T>, grid1d(Ne, 256), 256, 0, src, eleMapBack0, Ne, dstE);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// objective and sensitivities (TOP3D_XL.m:124-130 / 323-328)
// ---------------------------------------------------------------------------
__global__ void k_objective(int64_t Ne, const double* __restrict__ ce, const double* __restrict__ xPhys, double cSolid,
                            double Emin, double E0, double penal, double* __restrict__ dc, ObjState* os,
                            RedScratch rs) {
  pdl_wait();
  double sc = 0.0, sv = 0.0;
  const double dsimp = penal * (E0 - Emin);
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    const double x = xPhys[e];
    const double cn = ce[e] / cSolid;
    const double E = Emin + pow(x, penal) * (E0 - Emin);
    sc += E * cn;
    sv += x;
    dc[e] = -(dsimp * pow(x, penal - 1)) * cn;
  }
  double v[2] = {sc, sv}, tot[2];
  if (reduce_publish<2>(v, rs, tot) && threadIdx.x == 0) {
    os->cObj = tot[0];
    os->xsum = tot[1];
  }
}
void launch_objective(cudaStream_t st, int64_t Ne, const double* ce, const double* xPhys, double cSolid, double Emin,
                      double E0, double penal, double* dc, ObjState* os, RedScratch rs) {
  launch_pdl(st, k_objective, grid1d(Ne, 256), 256, 0, Ne, ce, xPhys, cSolid, Emin, E0, penal, dc, os, rs);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_fill(int64_t n, double value, double* __restrict__ out) {
  pdl_wait();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = value;
}
void launch_fill(cudaStream_t st, int64_t n, double value, double* out) {
  launch_pdl(st, k_fill, grid1d(n, 256), 256, 0, n, value, out);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_dot(int64_t n, const double* __restrict__ a, const double* __restrict__ b, double* out,
                      RedScratch rs) {
  pdl_wait();
  double s = 0.0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    s += b ? a[i] * b[i] : a[i];
  double v[1] = {s}, tot[1];
  if (reduce_publish<1>(v, rs, tot) && threadIdx.x == 0) *out = tot[0];
}
void launch_sum(cudaStream_t st, int64_t n, const double* a, const double* b, double* out, RedScratch rs) {
  launch_pdl(st, k_dot, grid1d(n, 256), 256, 0, n, a, b, out, rs);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_ewise(int op, int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                        double* __restrict__ out, double s) {
  pdl_wait();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    double v;
    switch (op) {
      case EW_MUL:
        v = a[i] * b[i];
        break;
      case EW_DIV_MAXX:  // a ./ max(s, b)
        v = a[i] / fmax(s, b[i]);
        break;
      default:
        v = a[i];
    }
    out[i] = v;
  }
}
void launch_ewise(cudaStream_t st, int op, int64_t n, const double* a, const double* b, double* out, double s) {
  launch_pdl(st, k_ewise, grid1d(n, 256), 256, 0, op, n, a, b, out, s);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// OC update with Lagrange-multiplier bisection (TOP3D_XL.m:145-156).  Each
// launch evaluates three or four bisection steps as one grid reduction; once
// the interval test fails the remaining launches return at once.
// ---------------------------------------------------------------------------
// x sqrt(-dc / lmid) evaluated as w * r with w = x sqrt(-dc) formed once per OC iteration
// (k_oc_prep) and r = 1 / sqrt(lmid) once per bisection step: the bisection then streams x and w
// with two multiplications per element instead of a division and a square root (the result
// differs from the reference's evaluation order by a few ulps).
__device__ __forceinline__ double oc_xnew(double x, double w, double r, double move) {
  return fmax(0.0, fmax(x - move, fmin(1.0, fmin(x + move, w * r))));
}

__global__ void k_oc_prep(int64_t Ne, const double* __restrict__ x, const double* __restrict__ dc,
                          double* __restrict__ w) {
  pdl_wait();
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x)
    w[e] = x[e] * sqrt(-dc[e]);
}
void launch_oc_prep(cudaStream_t st, int64_t Ne, const double* x, const double* dc, double* w) {
  launch_pdl(st, k_oc_prep, grid1d(Ne, 256), 256, 0, Ne, x, dc, w);
  TOPX_CUDA_OK(cudaGetLastError());
}

// D bisection steps per launch.  The multipliers the next D
// steps can try form a binary tree below the current interval (l1, l2): node 0 is its midpoint,
// child 2j+1 the midpoint of node j's lower half (the step found the volume too low, l2 = lmid),
// child 2j+2 of its upper half (l1 = lmid).  One pass over x and w sums the volume change of all
// 2^D - 1 nodes; the last block then walks the tree taking exactly the decisions, interval test
// included, that D launches of a one-step kernel take.  Every node's midpoint and sum are
// formed as the one-step kernel forms them (same expressions, same per-thread order, same
// block-order reduction), so l1, l2, lmid and the step count come out bit-identical.
// Up to 2^20 elements bound by the launch and the reduction, whose 15 sums cost a block as much as a dozen elements do:
// four steps a launch, two blocks an SM, more elements a thread (four of its loads in flight).  Beyond, the nodes' FP64
// operations bound it: three steps.  The bisection and the final pass, us, with a thread per element and three
// steps a launch, three steps, four, five (its sums spill): 50 x 100 x 50 elements 258, 185, 179, 306;
// 64 x 128 x 64: 419, 223, 213, 398; 96 x 192 x 96: 550, 355, 369, 710; 128 x 256 x 128: 755, 586, 752.
// In the per-element clamp, max(0, max(x - move, min(1, min(x + move, t)))) is regrouped as
// max(lo, min(hi, t)) with lo = max(0, x - move), hi = min(1, x + move) formed once per element,
// and the two outer selections are written as comparisons (a NaN t, from a positive dc, selects
// hi as fmin does): min and max select one operand exactly, so neither changes a value (up to
// the sign of a zero term of the sum).
constexpr int oc_nodes(int steps) { return (1 << steps) - 1; }

// 1/sqrt(lmid) of node j: its interval follows the path from the root
__device__ __forceinline__ double oc_node(int j, double a, double b) {
  int depth = 0;
  while ((j + 1) >> (depth + 1)) ++depth;  // node j sits at depth floor(log2(j + 1))
  for (int d = depth - 1; d >= 0; --d) {   // the branch taken at each level, root first
    const int node = ((j + 1) >> (d + 1)) - 1;
    const double lmid = 0.5 * (b + a);
    if (j + 1 - ((node + 1) << (d + 1)) < (1 << d))  // lower half: l2 = lmid
      b = lmid;
    else
      a = lmid;
  }
  return 1.0 / sqrt(0.5 * (b + a));
}

// the decisions of D steps on the nodes' sums; true once the interval test fails
template <int D>
__device__ __forceinline__ bool oc_walk(double fval, const double* tot, double& l1, double& l2, double& lmid,
                                        int& steps) {
  int j = 0;
  for (int d = 0; d < D; ++d) {
    lmid = 0.5 * (l2 + l1);
    if (fval + tot[j] > 0) {
      l1 = lmid;
      j = 2 * j + 2;
    } else {
      l2 = lmid;
      j = 2 * j + 1;
    }
    steps += 1;
    if (!((l2 - l1) / (l1 + l2) > 1e-6)) return true;
  }
  return false;
}

template <int D>
__global__ void __launch_bounds__(256, 2) k_oc_bisect(int64_t Ne, const double* __restrict__ x,
                                                   const double* __restrict__ w, const uint8_t* __restrict__ passive,
                                                   OcState* os, RedScratch rs, double move) {
  constexpr int kOcNodes = oc_nodes(D);
  pdl_wait();
  if (os->converged) return;
  __shared__ double sr[kOcNodes];
  if (threadIdx.x < kOcNodes) sr[threadIdx.x] = oc_node(threadIdx.x, os->l1, os->l2);
  __syncthreads();
  double r[kOcNodes];
#pragma unroll
  for (int j = 0; j < kOcNodes; ++j) r[j] = sr[j];
  double s[kOcNodes];
#pragma unroll
  for (int j = 0; j < kOcNodes; ++j) s[j] = 0.0;
  constexpr int BATCH = 4;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t e0 = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e0 < Ne; e0 += BATCH * stride) {
    double xv[BATCH], wv[BATCH];
    bool pas[BATCH];
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int64_t e = e0 + b * stride;
      xv[b] = e < Ne ? x[e] : 0.0;
      wv[b] = e < Ne ? w[e] : 0.0;
      pas[b] = passive && e < Ne && passive[e];
    }
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      if (e0 + b * stride >= Ne) break;
      if (pas[b]) {
#pragma unroll
        for (int j = 0; j < kOcNodes; ++j) s[j] += 1.0 - xv[b];
      } else {
        const double lo = fmax(0.0, xv[b] - move), hi = fmin(1.0, xv[b] + move);
#pragma unroll
        for (int j = 0; j < kOcNodes; ++j) {
          const double t = wv[b] * r[j];
          const double u = t < hi ? t : hi;
          s[j] += (u > lo ? u : lo) - xv[b];
        }
      }
    }
  }
  double tot[kOcNodes];
  if (reduce_publish<kOcNodes>(s, rs, tot, gridDim.x) && threadIdx.x == 0) {
    double l1 = os->l1, l2 = os->l2, lmid = os->lmid;
    int steps = os->steps;
    const bool conv = oc_walk<D>(os->fval, tot, l1, l2, lmid, steps);
    os->l1 = l1;
    os->l2 = l2;
    os->lmid = lmid;
    os->steps = steps;
    os->converged = conv;
  }
}
void launch_oc_bisect(cudaStream_t st, int64_t Ne, const double* x, const double* w, const uint8_t* passive,
                      OcState* os, RedScratch rs, double move, int steps) {
  const unsigned nb = grid1d(Ne, 256, 2 * 148);
  static_assert(size_t(oc_nodes(4)) * 148 * 2 <= size_t(kMaxRedBlocks) * kMaxRedSlots, "reduction slots");
  launch_pdl(st, steps == 4 ? k_oc_bisect<4> : k_oc_bisect<3>, nb, 256, 0, Ne, x, w, passive, os, rs, move);
  TOPX_CUDA_OK(cudaGetLastError());
}

// The whole bisection in one launch for a small design: a cluster of eight CTAs keeps x and w in shared memory, and the
// CTAs leave their sums of the 15 nodes in one another's, so that a round of four steps costs a cluster barrier instead
// of a launch and its reduction's tail.  Every CTA adds the eight parts in the same order and takes the same decisions.
// The bisection and the final pass, us, as launches and as a cluster: 16 x 32 x 16 elements 124, 80; 25 x 50 x 25: 127,
// 119; 32 x 32 x 32: 128, 116; from there on its eight SMs' arithmetic takes longer than the launches.
constexpr unsigned OCC_CTAS = 8, OCC_THREADS = 512;
constexpr int OCC_ELEMS = 8, OCC_STEPS = 4;
static_assert(kOcClusterElems == int64_t(OCC_CTAS) * OCC_THREADS * OCC_ELEMS, "elements of a cluster");

__global__ void __launch_bounds__(OCC_THREADS) k_oc_cluster(int Ne, const double* __restrict__ x,
                                                            const double* __restrict__ w,
                                                            const uint8_t* __restrict__ passive, OcState* os,
                                                            double move) {
  constexpr int kOcNodes = oc_nodes(OCC_STEPS);
  pdl_wait();
  __shared__ double part[2][OCC_CTAS][kOcNodes];  // by round parity: a CTA ahead writes the other
  __shared__ double sr[kOcNodes], tot[kOcNodes];
  const int tid = threadIdx.x;
  extern __shared__ double2 occ_xw[];  // x and w of the CTA's elements; a thread reads its own only
  const int nb = (Ne + int(OCC_CTAS * OCC_THREADS) - 1) / int(OCC_CTAS * OCC_THREADS);  // elements a thread
  unsigned pas = 0;
  for (int b = 0; b < nb; ++b) {
    const int e = (b * int(OCC_CTAS) + int(blockIdx.x)) * int(OCC_THREADS) + tid;
    // beyond the last element x = w = 0 adds zero to every sum
    occ_xw[b * int(OCC_THREADS) + tid] = e < Ne ? make_double2(x[e], w[e]) : make_double2(0.0, 0.0);
    if (passive && e < Ne && passive[e]) pas |= 1u << b;
  }
  double l1 = os->l1, l2 = os->l2, lmid = os->lmid;
  const double fval = os->fval;
  int steps = os->steps;
  bool conv = os->converged != 0;
  cluster_sync();  // every CTA runs: its shared memory may be written
  for (int round = 0; !conv && round < kOcMostSteps / OCC_STEPS; ++round) {
    if (tid < kOcNodes) sr[tid] = oc_node(tid, l1, l2);
    __syncthreads();
    double r[kOcNodes], s[kOcNodes];
#pragma unroll
    for (int j = 0; j < kOcNodes; ++j) {
      r[j] = sr[j];
      s[j] = 0.0;
    }
#pragma unroll 1
    for (int b = 0; b < nb; ++b) {
      const double2 xw = occ_xw[b * int(OCC_THREADS) + tid];
      if (pas >> b & 1u) {
#pragma unroll
        for (int j = 0; j < kOcNodes; ++j) s[j] += 1.0 - xw.x;
      } else {
        const double lo = fmax(0.0, xw.x - move), hi = fmin(1.0, xw.x + move);
#pragma unroll
        for (int j = 0; j < kOcNodes; ++j) {
          const double t = xw.y * r[j];
          const double u = t < hi ? t : hi;
          s[j] += (u > lo ? u : lo) - xw.x;
        }
      }
    }
    block_sum<kOcNodes>(s);
    double* const mine = part[round & 1][blockIdx.x];
    if (tid < 32) {  // the sums are in every lane of warp 0: lane p tells CTA p
      if (tid < int(OCC_CTAS))
#pragma unroll
        for (int j = 0; j < kOcNodes; ++j) cluster_store(mine + j, unsigned(tid), s[j]);
    }
    cluster_sync();
    if (tid < kOcNodes) {
      double t = 0.0;
#pragma unroll
      for (unsigned p = 0; p < OCC_CTAS; ++p) t += part[round & 1][p][tid];
      tot[tid] = t;
    }
    __syncthreads();
    conv = oc_walk<OCC_STEPS>(fval, tot, l1, l2, lmid, steps);
  }
  if (blockIdx.x == 0 && tid == 0) {
    os->l1 = l1;
    os->l2 = l2;
    os->lmid = lmid;
    os->steps = steps;
    os->converged = conv;
  }
}
void prepare_oc_kernels() {
  TOPX_CUDA_OK(cudaFuncSetAttribute(k_oc_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int(OCC_ELEMS * OCC_THREADS * sizeof(double2))));
}
void launch_oc_cluster(cudaStream_t st, int64_t Ne, const double* x, const double* w, const uint8_t* passive,
                       OcState* os, double move) {
  // x and w of the elements that a CTA has
  const int64_t nb = (Ne + OCC_CTAS * OCC_THREADS - 1) / (OCC_CTAS * OCC_THREADS);
  launch_clusters(st, k_oc_cluster, OCC_CTAS, OCC_THREADS, size_t(nb) * OCC_THREADS * sizeof(double2), OCC_CTAS, int(Ne),
                  x, w, passive, os, move);
  TOPX_CUDA_OK(cudaGetLastError());
}

// x = xnew(lmid); xPhys = x (passive = 1); change = max|xnew - x|; sharpness
__global__ void k_oc_final(int64_t Ne, double* __restrict__ x, const double* __restrict__ w,
                           const uint8_t* __restrict__ passive, double* __restrict__ xPhys, OcState* os,
                           RedScratch rs, RedScratch rs2, double move) {
  pdl_wait();
  const double lmid = os->lmid;
  const double r = 1.0 / sqrt(lmid);
  double ch = 0.0, sh = 0.0;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    const double xv = x[e];
    const bool pas = passive && passive[e];
    const double xn = pas ? 1.0 : oc_xnew(xv, w[e], r, move);
    ch = fmax(ch, fabs(xn - xv));
    x[e] = xn;
    xPhys[e] = xn;
    sh += xn * (1.0 - xn);
  }
  double v[1] = {sh}, tot[1];
  if (reduce_publish<1>(v, rs, tot) && threadIdx.x == 0) os->sharpsum = tot[0];
  double mx;
  if (reduce_publish_max(ch, rs2, mx) && threadIdx.x == 0) os->change = mx;
}
void launch_oc_final(cudaStream_t st, int64_t Ne, double* x, const double* w, const uint8_t* passive, double* xPhys,
                     OcState* os, RedScratch rs, RedScratch rs2, double move) {
  launch_pdl(st, k_oc_final, grid1d(Ne, 256), 256, 0, Ne, x, w, passive, xPhys, os, rs, rs2, move);
  TOPX_CUDA_OK(cudaGetLastError());
}

template void launch_scatter_elems_t<double>(cudaStream_t, const double*, const int32_t*, int64_t, double*);
template void launch_scatter_elems_t<float>(cudaStream_t, const double*, const int32_t*, int64_t, float*);

}  // namespace topx

namespace topx {

// ---------------------------------------------------------------------------
// MMA with one constraint (MMAseq/GenSub/SolveDIP, TOP3D_XL.m:1804-2049).
// Elements flagged passive are not part of the subproblem (activeEles).
// ---------------------------------------------------------------------------
constexpr double kMmaFeps = 1.0e-6;
constexpr double kMmaC = 1000.0;

__global__ void k_mma_gensub(int64_t n, int iter, double move, const double* __restrict__ xval,
                             const uint8_t* __restrict__ passive, double* __restrict__ xold1,
                             double* __restrict__ xold2, double* __restrict__ low, double* __restrict__ upp,
                             const double* __restrict__ dfdx, const double* __restrict__ dgdx, double gx, int64_t nact,
                             double* __restrict__ alpha, double* __restrict__ beta, double* __restrict__ p0,
                             double* __restrict__ q0, double* __restrict__ pij, double* __restrict__ qij,
                             MmaState* ms, RedScratch rs) {
  pdl_wait();
  double bs = 0.0;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n; e += int64_t(gridDim.x) * blockDim.x) {
    if (passive && passive[e]) continue;
    const double xv = xval[e];
    const double xmn = fmax(0.0, xv - move), xmx = fmin(1.0, xv + move);
    const double xo1 = xold1[e], xo2 = xold2[e];
    double lo, up;
    if (iter < 3) {
      lo = xv - 0.5 * (xmx - xmn);
      up = xv + 0.5 * (xmx - xmn);
    } else {
      const double zzz = (xv - xo1) * (xo1 - xo2);
      const double gam = zzz > 0 ? 1.2 : (zzz < 0 ? 0.7 : 1.0);
      lo = xv - gam * (xo1 - low[e]);
      up = xv + gam * (upp[e] - xo1);
      lo = fmax(lo, xv - 10.0 * (xmx - xmn));
      lo = fmin(lo, xv - 0.01 * (xmx - xmn));
      up = fmin(up, xv + 10.0 * (xmx - xmn));
      up = fmax(up, xv + 0.01 * (xmx - xmn));
    }
    double al = 0.9 * lo + 0.1 * xv;
    if (al - xmn < 0) al = xmn;
    double be = 0.9 * up + 0.1 * xv;
    if (be - xmx > 0) be = xmx;
    const double df = dfdx[e], dg = dgdx[e];
    const double ux = up - xv, xl = xv - lo;
    const double dfp = df < 0.0 ? 0.0 : df, dfm = -df < 0.0 ? 0.0 : -df;
    const double P0 = ux * ux * (dfp + 0.001 * fabs(df) + 0.5 * kMmaFeps / (up - lo));
    const double Q0 = xl * xl * (dfm + 0.001 * fabs(df) + 0.5 * kMmaFeps / (up - lo));
    const double dgp = dg < 0.0 ? 0.0 : dg, dgm = -dg < 0.0 ? 0.0 : -dg;
    const double extra = 0.001 * fabs(dg) + 0.5 * kMmaFeps / (up - lo);
    const double Pij = ux * ux * (dgp + extra), Qij = xl * xl * (dgm + extra);
    bs += Pij / ux + Qij / xl;
    low[e] = lo;
    upp[e] = up;
    alpha[e] = al;
    beta[e] = be;
    p0[e] = P0;
    q0[e] = Q0;
    pij[e] = Pij;
    qij[e] = Qij;
    xold2[e] = xo1;
    xold1[e] = xv;
  }
  double v[1] = {bs}, tot[1];
  if (reduce_publish<1>(v, rs, tot) && threadIdx.x == 0) {
    ms->b = -gx + tot[0];
    ms->lam = kMmaC / 2.0;
    ms->mu = 1.0;
    ms->epsi = 1.0;
    ms->err = 1.0;
    ms->tol = 1.0e-9 * sqrt(double(nact) + 1.0);
    ms->inner = 0;
    ms->total = 0;
    ms->finished = 0;
    ms->stepped = 0;
  }
}

void launch_mma_gensub(cudaStream_t st, int64_t n, int iter, double move, const double* xval, const uint8_t* passive,
                       double* xold1, double* xold2, double* low, double* upp, const double* dfdx, const double* dgdx,
                       double gx, int64_t nact, double* alpha, double* beta, double* p0, double* q0, double* pij,
                       double* qij, MmaState* ms, RedScratch rs) {
  launch_pdl(st, k_mma_gensub, grid1d(n, 256), 256, 0, n, iter, move, xval, passive, xold1, xold2, low, upp, dfdx,
             dgdx, gx, nact, alpha, beta, p0, q0, pij, qij, ms, rs);
  TOPX_CUDA_OK(cudaGetLastError());
}

__device__ __forceinline__ void mma_x(double lam, double lo, double up, double al, double be, double P0, double Q0,
                                      double Pij, double Qij, double& xcl, double& xun, double& pj, double& qj) {
  pj = P0 + Pij * lam;
  qj = Q0 + Qij * lam;
  const double sp = sqrt(pj), sq = sqrt(qj);
  xun = (sp * lo + sq * up) / (sp + sq);
  xcl = xun;
  if (xcl - al < 0) xcl = al;
  if (xcl - be > 0) xcl = be;
}

// One pass of the dual interior point method at the multiplier lam: x(lam) and the dual residual of the Newton step that
// led to lam, with the epsilon schedule (XYZofLAMBDA, DualResidual: TOP3D_XL.m:1967-1984, 2033-2049; not on the first
// pass, which follows no step), and, unless that ends the solve, the next Newton step (DualGrad, DualHess,
// DualLineSearch: TOP3D_XL.m:1930-2031).  Bound by reading the eight arrays; residual and Newton step need the same x,
// so that a step reads them once (128 x 256 x 128 elements, two loops of 11 steps each: 43.18 ms with a pass each, now 42.44).
__global__ void k_mma_step(int64_t n, const uint8_t* __restrict__ passive, const double* __restrict__ low,
                           const double* __restrict__ upp, const double* __restrict__ alpha,
                           const double* __restrict__ beta, const double* __restrict__ p0,
                           const double* __restrict__ q0, const double* __restrict__ pij,
                           const double* __restrict__ qij, double* __restrict__ x, MmaState* ms, RedScratch rs) {
  pdl_wait();
  if (ms->finished) return;
  const double lam = fmax(ms->lam, 0.0);
  double sg = 0.0, sh = 0.0, sp = 0.0, sq = 0.0;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n; e += int64_t(gridDim.x) * blockDim.x) {
    if (passive && passive[e]) continue;
    const double lo = low[e], up = upp[e], al = alpha[e], be = beta[e], pe = pij[e], qe = qij[e];
    double xc, xu, pj, qj;
    mma_x(lam, lo, up, al, be, p0[e], q0[e], pe, qe, xc, xu, pj, qj);
    x[e] = xc;
    const double ux = up - xc, xl = xc - lo;
    const double pu = pe / ux, ql = qe / xl;
    sp += pu;
    sq += ql;
    sg += pu + ql;
    const double PQ = pe / (ux * ux) - qe / (xl * xl);
    double df2 = -1.0 / (2.0 * pj / (ux * ux * ux) + 2.0 * qj / (xl * xl * xl));
    if (xu - al < 0) df2 = 0.0;
    if (xu - be > 0) df2 = 0.0;
    sh += PQ * df2 * PQ;
  }
  double v[4] = {sg, sh, sp, sq}, tot[4];
  if (reduce_publish<4>(v, rs, tot) && threadIdx.x == 0) {
    const double L = lam, y = fmax(L - kMmaC, 0.0);
    double mu = ms->mu, epsi = ms->epsi;
    ms->lam = L;
    if (ms->stepped) {
      double r1 = -ms->b - 0.0 - y + mu;
      r1 = r1 + tot[2] + tot[3];
      const double r2 = mu * L - epsi;
      double err = 0.0;
      if (err < fabs(r1)) err = fabs(r1);
      if (err < fabs(r2)) err = fabs(r2);
      ms->err = err;
      ms->inner += 1;
      ms->total += 1;
      if (!(err > 0.9 * epsi && ms->inner < 100)) {
        epsi *= 0.1;
        ms->epsi = epsi;
        ms->inner = 0;
        if (!(epsi > ms->tol)) {
          ms->finished = 1;
          return;
        }
      }
    }
    double grad = -ms->b - 0.0 - y + tot[0];
    grad = -1.0 * grad - epsi / L;
    double H = tot[1];
    if (L > kMmaC) H -= 1.0;
    H -= mu / L;
    double corr = 1e-4 * H / 1.0;
    if (-1.0 * corr < 1.0e-7) corr = -1.0e-7;
    H += corr;
    const double s1 = grad / H;
    const double s2 = -mu + epsi / L - s1 * mu / L;
    double theta = 1.005;
    if (theta < -1.01 * s1 / L) theta = -1.01 * s1 / L;
    if (theta < -1.01 * s2 / mu) theta = -1.01 * s2 / mu;
    theta = 1.0 / theta;
    ms->lam = L + theta * s1;
    ms->mu = mu + theta * s2;
    ms->grad = grad;
    ms->hess = H;
    ms->stepped = 1;
  }
}

void launch_mma_step(cudaStream_t st, int64_t n, const uint8_t* passive, const double* low, const double* upp,
                     const double* alpha, const double* beta, const double* p0, const double* q0, const double* pij,
                     const double* qij, double* x, MmaState* ms, RedScratch rs) {
  launch_pdl(st, k_mma_step, grid1d(n, 256), 256, 0, n, passive, low, upp, alpha, beta, p0, q0, pij, qij, x, ms, rs);
  TOPX_CUDA_OK(cudaGetLastError());
}

// x = xmma on active elements, 1 on passive ones; change = max |xmma - xval| (xval kept in xold1)
__global__ void k_mma_finish(int64_t n, const uint8_t* __restrict__ passive, const double* __restrict__ xmma,
                             const double* __restrict__ xold1, double* __restrict__ x, MmaState* ms, RedScratch rs) {
  pdl_wait();
  double ch = 0.0;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n; e += int64_t(gridDim.x) * blockDim.x) {
    if (passive && passive[e]) {
      x[e] = 1.0;
      continue;
    }
    ch = fmax(ch, fabs(xmma[e] - xold1[e]));
    x[e] = xmma[e];
  }
  double mx;
  if (reduce_publish_max(ch, rs, mx) && threadIdx.x == 0) ms->change = mx;
}

void launch_mma_finish(cudaStream_t st, int64_t n, const uint8_t* passive, const double* xmma, const double* xold1,
                       double* x, MmaState* ms, RedScratch rs) {
  launch_pdl(st, k_mma_finish, grid1d(n, 256), 256, 0, n, passive, xmma, xold1, x, ms, rs);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// LOCAL driver elementwise chain (TOP3D_XL.m:333-350, 380-382)
// ---------------------------------------------------------------------------
__global__ void k_pnorm(int64_t Ne, const double* __restrict__ xhat, double Ve0, double pP, double* out,
                        RedScratch rs) {
  pdl_wait();
  double s = 0.0;
  const double vm = pow(Ve0, pP);
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x)
    s += pow(xhat[e], pP) / vm;
  double v[1] = {s}, tot[1];
  if (reduce_publish<1>(v, rs, tot) && threadIdx.x == 0) *out = tot[0];
}
void launch_pnorm_terms(cudaStream_t st, int64_t Ne, const double* xhat, double Ve0, int pPIO, double* out_sum,
                        RedScratch rs) {
  launch_pdl(st, k_pnorm, grid1d(Ne, 256), 256, 0, Ne, xhat, Ve0, double(pPIO), out_sum, rs);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_local_sens(int64_t Ne, const double* __restrict__ xhat, const double* __restrict__ xTilde,
                             const double* __restrict__ dc, double Ve0, double pP, double pn, double bt, double eta,
                             double* __restrict__ dfdx_pde, double* __restrict__ dx, double* __restrict__ dcdx) {
  pdl_wait();
  const double f = pow(pn, 1.0 / pP - 1.0);
  const double vm = pow(Ve0, pP);
  const double den = tanh(bt * eta) + tanh(bt * (1 - eta));
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    dfdx_pde[e] = f * (pow(xhat[e], pP - 1) / vm) / double(Ne);
    const double th = tanh(bt * (xTilde[e] - eta));
    const double d = bt * (1 - th * th) / den;
    dx[e] = d;
    dcdx[e] = dc[e] * d;
  }
}
void launch_local_sens(cudaStream_t st, int64_t Ne, const double* xhat, const double* xTilde, const double* dc,
                       double Ve0, int pPIO, double pn, double betaPIO, double etaPIO, double* dfdx_pde, double* dx,
                       double* dcdx) {
  launch_pdl(st, k_local_sens, grid1d(Ne, 256), 256, 0, Ne, xhat, xTilde, dc, Ve0, double(pPIO), pn, betaPIO, etaPIO,
             dfdx_pde, dx, dcdx);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_heaviside(int64_t Ne, const double* __restrict__ xTilde, const uint8_t* __restrict__ passive,
                            double bt, double eta, double* __restrict__ xPhys, double* sharpsum, RedScratch rs) {
  pdl_wait();
  const double a = tanh(bt * eta), den = tanh(bt * eta) + tanh(bt * (1 - eta));
  double s = 0.0;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    double v = (a + tanh(bt * (xTilde[e] - eta))) / den;
    if (passive && passive[e]) v = 1.0;
    xPhys[e] = v;
    s += v * (1.0 - v);
  }
  double vv[1] = {s}, tot[1];
  if (reduce_publish<1>(vv, rs, tot) && threadIdx.x == 0) *sharpsum = tot[0];
}
void launch_heaviside(cudaStream_t st, int64_t Ne, const double* xTilde, const uint8_t* passive, double betaPIO,
                      double etaPIO, double* xPhys, double* sharpsum, RedScratch rs) {
  launch_pdl(st, k_heaviside, grid1d(Ne, 256), 256, 0, Ne, xTilde, passive, betaPIO, etaPIO, xPhys, sharpsum, rs);
  TOPX_CUDA_OK(cudaGetLastError());
}

}  // namespace topx
