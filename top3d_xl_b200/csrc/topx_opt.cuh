// Launch wrappers of the optimiser-side kernels (filter, objective, OC, MMA).
#pragma once

#include "topx_kernels.cuh"

namespace topx {

struct ObjState {
  double cObj;  // E . ceNorm
  double xsum;  // sum(xPhys)
};

struct OcState {
  double l1, l2, lmid, fval;
  double change, sharpsum;
  int converged;
  int steps;
};

enum EwOp { EW_COPY = 0, EW_MUL = 1, EW_DIV_MAXX = 2 };

// --- PDE filter ------------------------------------------------------------
// The Helmholtz filter's element matrix (TOP3D_XL.m:845-853) in the basis of sums and differences along the
// axes is diagonal, by the number of differences; dp: inverse diagonal of a node with 0..8 solid elements
template <typename T>
struct FilterKe {
  T h[4];
  T dp[9];
};
template <typename T>
FilterKe<T> filter_ke(const double* KF64);
// Tiles of the filter operator's launch: TY x TX nodes written by PY x PX threads, zc planes per CTA
struct FilterShape {
  int PY, PX, TY, TX, zc;
  dim3 grid;
};
FilterShape filter_shape(Grid g, int rows, int bytes);  // bytes: of the filter's type
// tiles that own a node of the domain, and per tile its planes that hold a present node (lo | hi << 16)
std::vector<uint32_t> filter_active_tiles(Grid g, int rows, const FilterShape& f, const std::vector<uint8_t>& present,
                                          std::vector<uint32_t>& zranges);
template <typename T>
struct FilterArgs {
  Grid g;
  FilterShape sh;
  FilterKe<T> ke;
  T *r, *y, *q;
  T *pin, *pout;         // the previous direction, and the buffer that takes the new one
  const uint8_t* flags;  // per node its number of solid elements, | 128 when the element above it (lowest corner) is solid
  PcgScalars* sc;
  RedScratch rs;
  const uint32_t* active;  // filter_active_tiles, or null
  const uint32_t* zr;
  int ntiles;
  const uint32_t* act;  // chunk mask (chunk_active), or null
  int* err;             // takes kCoopErrCopy (report_copy_wait)
  double tol;
  int maxIT;
};
// r = node sums of the element source (on the grid, at the elements' lowest nodes), and the CG's scalars
template <typename T>
void launch_filter_start(cudaStream_t st, const FilterArgs<T>& a, const T* srcE);
// p = D r (+ beta p), q = A p, p'q; the previous step's y += lam p
template <typename T>
void launch_filter_ku(cudaStream_t st, const FilterArgs<T>& a);
// r -= lam q, the stop test and beta from r'r and r'D r
template <typename T>
void launch_filter_update(cudaStream_t st, const FilterArgs<T>& a);
// element means of y + lam p, p the last direction (in pin when the number of steps is even, else in pout)
template <typename T>
void launch_filter_n2e(cudaStream_t st, const FilterArgs<T>& a, const int32_t* eleMapBack0, int64_t Ne, double* out);
void prepare_filter_kernels();
template <typename T>
void launch_scatter_elems_t(cudaStream_t st, const double* src, const int32_t* eleMapBack0, int64_t Ne, T* dstE);

// --- objective / OC --------------------------------------------------------
void launch_objective(cudaStream_t st, int64_t Ne, const double* ce, const double* xPhys, double cSolid, double Emin,
                      double E0, double penal, double* dc, ObjState* os, RedScratch rs);
void launch_fill(cudaStream_t st, int64_t n, double value, double* out);
void launch_sum(cudaStream_t st, int64_t n, const double* a, const double* b, double* out, RedScratch rs);
void launch_ewise(cudaStream_t st, int op, int64_t n, const double* a, const double* b, double* out, double s);
// OC bisection (TOP3D_XL.m:145-156): w = x sqrt(-dc) once, then bisection steps on lmid,
// `steps` (4 or 3) of them per launch of launch_oc_bisect
inline int oc_steps_per_launch(int64_t Ne) { return Ne <= (int64_t(1) << 20) ? 4 : 3; }
constexpr int kOcMostSteps = 268;
void launch_oc_prep(cudaStream_t st, int64_t Ne, const double* x, const double* dc, double* w);
void launch_oc_bisect(cudaStream_t st, int64_t Ne, const double* x, const double* w, const uint8_t* passive,
                      OcState* os, RedScratch rs, double move, int steps);
// all steps in one launch, for up to kOcClusterElems elements
constexpr int64_t kOcClusterElems = 32768;
void prepare_oc_kernels();
void launch_oc_cluster(cudaStream_t st, int64_t Ne, const double* x, const double* w, const uint8_t* passive,
                       OcState* os, double move);
void launch_oc_final(cudaStream_t st, int64_t Ne, double* x, const double* w, const uint8_t* passive, double* xPhys,
                     OcState* os, RedScratch rs, RedScratch rs2, double move);

// --- MMA (m = 1) -------------------------------------------------------------
struct MmaState {
  double lam, mu, epsi, err, tol;
  double b;  // constraint constant of the subproblem
  double grad, hess;
  double change;  // max |xnew - xval|
  int inner;      // Newton steps at the current epsilon
  int total;      // Newton steps overall
  int finished;
  int stepped;    // a Newton step led to lam
};
void launch_mma_gensub(cudaStream_t st, int64_t n, int iter, double move, const double* xval, const uint8_t* passive,
                       double* xold1, double* xold2, double* low, double* upp, const double* dfdx, const double* dgdx,
                       double gx, int64_t nact, double* alpha, double* beta, double* p0, double* q0, double* pij,
                       double* qij, MmaState* ms, RedScratch rs);
void launch_mma_step(cudaStream_t st, int64_t n, const uint8_t* passive, const double* low, const double* upp,
                     const double* alpha, const double* beta, const double* p0, const double* q0, const double* pij,
                     const double* qij, double* x, MmaState* ms, RedScratch rs);
void launch_mma_finish(cudaStream_t st, int64_t n, const uint8_t* passive, const double* xmma, const double* xold1,
                       double* x, MmaState* ms, RedScratch rs);
// LOCAL driver elementwise chain (TOP3D_XL.m:333-382)
void launch_pnorm_terms(cudaStream_t st, int64_t Ne, const double* xhat, double Ve0, int pPIO, double* out_sum,
                        RedScratch rs);
void launch_local_sens(cudaStream_t st, int64_t Ne, const double* xhat, const double* xTilde, const double* dc,
                       double Ve0, int pPIO, double pn, double betaPIO, double etaPIO, double* dfdx_pde, double* dx,
                       double* dcdx);
void launch_heaviside(cudaStream_t st, int64_t Ne, const double* xTilde, const uint8_t* passive, double betaPIO,
                      double etaPIO, double* xPhys, double* sharpsum, RedScratch rs);

}  // namespace topx
