// Launch wrappers of the TOP3D_XL sm_100a kernels (all asynchronous on `st`).
#pragma once

#include <cstdint>
#include <vector>
#include <stdexcept>
#include <string>

#include "topx_device.cuh"

namespace topx {

struct CudaError : std::runtime_error {
  cudaError_t code;
  CudaError(cudaError_t e, const char* expr, const char* file, int line)
      : std::runtime_error(std::string(cudaGetErrorString(e)) + " at " + file + ":" + std::to_string(line) +
                           " (" + expr + ")"),
        code(e) {}
};
// Launch of a kernel that begins with pdl_wait(): its start overlaps the end of the launch before it.
// cluster: CTAs of a cluster along x.
template <typename... P, typename... A>
void launch_clusters(cudaStream_t st, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, unsigned cluster,
                     A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) throw CudaError(e, "cudaLaunchKernelEx", __FILE__, __LINE__);
  count_launch();
}
template <typename... P, typename... A>
void launch_pdl(cudaStream_t st, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
  launch_clusters(st, kernel, grid, block, smem, 1u, args...);
}
// A bounded device wait gave up (its poll limit ran out); the engine has cleared the error word
// and stays usable.
struct DeviceWaitError : std::runtime_error {
  using std::runtime_error::runtime_error;
};

// Dense padded grid of one multigrid level: ny, nx, nz elements (level-1 elements are stored at the index of
// their lowest node); node fields
// are SoA with plane stride `stride` (>= (ny+1)(nx+1)(nz+1)).
struct Grid {
  int ny = 0, nx = 0, nz = 0;
  int64_t stride = 0;
  __host__ __device__ int nny() const { return ny + 1; }
  __host__ __device__ int nnx() const { return nx + 1; }
  __host__ __device__ int nnz() const { return nz + 1; }
  __host__ __device__ int64_t nnodes() const { return int64_t(ny + 1) * (nx + 1) * (nz + 1); }
  __host__ __device__ int64_t nelems() const { return int64_t(ny) * nx * nz; }
};

// KU_PLAIN: out = K in.  The PCG modes form p = z (first step) or z + beta*p_in, out = K p, store p into pout,
// reduce p'q into sc->pq and apply the previous step's y += sc->lam * p_in (not on the first step):
// KU_P_UPDATE with z given, KU_FUSED with z = omega2 (r D) + P xc formed from the residual r
enum KuMode { KU_PLAIN = 0, KU_P_UPDATE = 2, KU_FUSED = 3 };

// The sums of a fused PCG step that the next kernel forms (Parts): p'q of K*u, r'r (or b'b) and r'D r of the residual
// pass, and the level-2 part of z'r
struct PcgParts {
  Parts pq, rr, rd, dot;
};
int residual_blocks(Grid g, Grid gc);
int prolong_blocks(Grid gf);

// element matrices in constant memory
void upload_ke(const double* Ke576);

// --- level-1 elasticity --------------------------------------------------
// Ke in the basis of sums and differences along the three axes (topx_ku.cu): normal strains a - b on the
// diagonal and b, shear g, bending p and q, torsion r - s and s, triple differences h
struct KuModes {
  double a_b, b, g, p, q, r_s, s, h;
};
KuModes ku_modes(const double* Ke576);
// Tile of the level-1 K*u: TY x TX nodes written by PY x PX threads, zc planes per CTA
struct KuShape {
  int PY, PX, TY, TX, zc;
  dim3 grid;
};
KuShape ku_shape(Grid g, int rows);  // rows: node rows along y to cover
constexpr int KU_SPAN = 4;  // span of level 2 in the fused PCG step (the first coarsening of every hierarchy)
struct KuArgs {
  Grid g, gc;  // level 1, level 2 (fused)
  KuShape sh;
  KuModes K;
  const double* in;   // u, z, or (fused) r
  const double* D;    // fused: inverse diagonal of a node's free DOFs
  const void* xc;     // fused: level-2 correction, float with pre32, else double
  bool pre32;
  double omega2;      // twice the Jacobi weight
  const double* pin;  // the previous direction
  double* pout;       // takes the new one (another buffer)
  double* out;
  const double* E;
  const uint8_t* flags;  // bits 0-2: fixed x, y, z; bit 3: present
  const double *cfix, *icfix;  // a fixed DOF's diagonal, and its inverse (fused)
  PcgScalars* sc;
  RedScratch rs;
  PcgParts parts;  // fused
  const uint32_t* active;  // the tiles that own a node of the domain (ku_active_tiles), or null for all
  const uint32_t* zr;      // per listed tile, the planes [lo, hi) of its z-chunk that hold a present node (lo | hi << 16)
  double* yacc;
  const int32_t* compact;  // KU_PLAIN: out in compact DOF order through this map, or null
  int* err;                // takes kCoopErrCopy (report_copy_wait)
};
// tiles of the launch that own a node of the domain; zranges (optional): the z-range entry of each
std::vector<uint32_t> ku_active_tiles(Grid g, int rows, const KuShape& k, const std::vector<uint8_t>& present,
                                      std::vector<uint32_t>* zranges = nullptr);
// ntiles: entries of args.active
void launch_ku(cudaStream_t st, KuMode mode, const KuArgs& args, int ntiles);
// d: all DOFs; d0: one value per node, that of its free DOFs
template <typename T>
void launch_diag_l1(cudaStream_t st, Grid g, const double* E, const uint8_t* fixbits, const double* cfix,
                    const uint8_t* present, T* d, double* d0);
// 'Standard' V-cycle only: r -= lambda q; ||r|| stop test into sc; lambda goes to sc->lam, for the next K*u
// (yacc) or launch_pcg_flush to apply
void launch_pcg_update(cudaStream_t st, Grid g, double* r, const double* q, PcgScalars* sc, RedScratch rs,
                       const uint32_t* act = nullptr);
// y += sc->lam * p: the solution step of the last PCG iteration
void launch_pcg_flush(cudaStream_t st, Grid g, double* y, const double* p, const PcgScalars* sc,
                      const uint32_t* act = nullptr);
void launch_residual_init(cudaStream_t st, Grid g, const double* b, const double* Ay, double* r, PcgScalars* sc,
                          RedScratch rs, double tol, int maxIT);
// One pass over the level-1 residual: RES_INIT r = b - q (and the PCG scalars), RES_UPDATE r -= lambda q (stop test
// into sc), RES_KEEP r as it is; with the y pass of its restriction into tmp, and (INIT, UPDATE) sc->rdr = r'D r
enum ResidualMode { RES_KEEP = 0, RES_INIT = 1, RES_UPDATE = 2 };
struct ResidualArgs {
  Grid g;
  double* r;
  const double *b, *q;
  const double* D;  // inverse diagonal of a node's free DOFs
  bool pre32;       // a fixed DOF's is rounded to float
  const uint8_t* flags;
  const double* icfix;  // inverse diagonal of a fixed DOF
  double* tmp;  // 3 x (coarse y nodes x fine x and z nodes)
  const uint32_t* act;
  PcgScalars* sc;
  RedScratch rs;
  PcgParts parts;
  double tol;
  int maxIT;
};
void launch_residual(cudaStream_t st, ResidualMode mode, const ResidualArgs& args, Grid gc);
// --- transfers -----------------------------------------------------------
// the x and z passes of the level-1 restriction: tmp -> out, and out64 when given
template <typename T>
// inside the PCG (parts) it also takes the residual pass's sums, which the stop test needs (init: the solve's start)
void launch_restrict_xz(cudaStream_t st, const double* tmp, Grid gf, T* out, double* out64, Grid gc, PcgScalars* sc,
                        const PcgParts* parts = nullptr, bool init = false, double tol = 0.0, int maxIT = 0);
// restriction between coarse levels (span 2)
template <typename T>
void launch_restrict(cudaStream_t st, const T* in, Grid gf, T* tmp1, T* tmp2, T* out, Grid gc, const PcgScalars* sc);
constexpr int64_t kRestrictOneLaunch = int64_t(1) << 21;  // nodes of the fine grid up to which tmp1 and tmp2 are not used
// x = omega*(r/d) + P(xc) + (omega*r)/d on present fine nodes.  rc (level 2 inside the PCG): the restricted
// residual in FP64; rc'x goes into dot, or z'r = omega2 sc->rdr + rc'x and beta into sc
template <typename TX, typename T, typename TD>
// act: the fine grid's chunk mask (chunk_active), or null
void launch_prolong_smooth(cudaStream_t st, int span, const TX* xc, Grid gc, const T* r, const TD* d,
                           const uint8_t* present, T* x, Grid gf, double omega, const double* rc, Parts dot,
                           PcgScalars* sc, RedScratch rs, const uint32_t* act = nullptr);
// 'Standard' V-cycle (TX:758-763, 772-777): x = omega*(r/d) + P(xc) without the smoothing term;
// x = omega*(r/d); q = r - q; x += omega*(r - q)/d (with dot: z.r into sc as above); coarse-level
// K*u with the stored Galerkin matrices Ks (dense elements x 576).  All skip once sc->done.
template <typename TX, typename T, typename TD>
void launch_prolong_add(cudaStream_t st, int span, const TX* xc, Grid gc, const T* r, const TD* d,
                        const uint8_t* present, T* x, Grid gf, double omega, PcgScalars* sc);
template <typename TR, typename T, typename TD>
void launch_jacobi_pre(cudaStream_t st, Grid g, const TR* r, const TD* d, const uint8_t* present, T* x, double omega,
                       const PcgScalars* sc);
template <typename TR, typename T>
void launch_residual_inplace(cudaStream_t st, Grid g, const TR* r, const uint8_t* present, T* q, const PcgScalars* sc);
template <typename TR, typename T, typename TD>
void launch_jacobi_correct(cudaStream_t st, Grid g, const TR* r, const T* q, const TD* d, const uint8_t* present,
                           T* x, double omega, bool dot, bool init, PcgScalars* sc, RedScratch rs);
void launch_ku_coarse(cudaStream_t st, Grid g, const double* Ks, const uint8_t* epresent, const uint8_t* present,
                      const double* u, double* y, const PcgScalars* sc);
// --- conversions -----------------------------------------------------------
template <typename TA, typename TB>
void launch_convert(cudaStream_t st, const TA* a, TB* b, int64_t n);
template <typename T>
void launch_compact_to_grid_nodes(cudaStream_t st, const double* src, T* dst, Grid g, const int32_t* nodMapBack0,
                                  int64_t numNodes);
// node_id: compact id of a grid node (n of them), or -1
void launch_index_nodes(cudaStream_t st, const int32_t* nodMapBack0, int64_t numNodes, int32_t* node_id, int64_t n);
// out = 1 / a, 0 where a is
void launch_invert(cudaStream_t st, int64_t n, const double* a, double* out);
void launch_fill_grid_nodes(cudaStream_t st, const double* src, double* dst, Grid g, const int32_t* node_id);
template <typename T>
void launch_grid_to_compact_nodes(cudaStream_t st, const T* src, double* dst, Grid g, const int32_t* nodMapBack0,
                                  int64_t numNodes);
void launch_simp_scatter(cudaStream_t st, const double* xPhys, const int32_t* eleMapBack0, int64_t Ne, double Emin,
                         double E0, double penal, double* Ed, float* Ef);
void launch_fill_scatter(cudaStream_t st, const int32_t* eleMapBack0, int64_t Ne, double val, double* Ed, float* Ef);
// ce_e = u_e^T Ke u_e (load-case weighted, accumulated into ce when accumulate)
void launch_unit_compliance(cudaStream_t st, Grid g, const double* U, const int32_t* eleMapBack0, int64_t Ne,
                            double weight, bool accumulate, double* ce);

// --- coarse levels -----------------------------------------------------------
// flagged: per level-2 element, whether it is one of the nflag elements with BC-modified templates (fl_*)
void launch_galerkin_l2(cudaStream_t st, Grid gf, Grid gc, const double* Efine, const double* Tm, int nflag,
                        const int32_t* fl_elem, const int32_t* fl_tsel, const double* fl_F, const uint8_t* flagged,
                        double* Ks);
void launch_galerkin_span2(cudaStream_t st, Grid gc, const double* Ksf, const uint8_t* cpresent, double* Ks);
template <typename T>
void launch_diag_coarse(cudaStream_t st, Grid g, const double* Ks, const uint8_t* present, T* d);

// shared-memory limits of the K*u launches (call once per device, outside capture)
void prepare_ku_kernels();

// Control words of the persistent coarse solve (zeroed before first use; err != 0 after a CTA
// gave up waiting, and then the words, and the solve's counters, must be zeroed again).
struct CoopControl {
  unsigned idle;   // a counter that nothing raises (the wait self-test); zero
  unsigned exits;  // CTAs that left the launch (the last one re-arms the counters); zero between launches
  int err;         // 0, or kCoopErrWait once a wait gave up
  int pad;
};
constexpr int kCoopErrWait = 1;  // a wait for another CTA's tasks (dataflow solve) gave up
constexpr int kCoopErrCopy = 2;  // a wait for asynchronous copies into shared memory (K*u, filter) gave up; has its own word
// Self-test of the dataflow solve's bounded dependency wait: one CTA waits for a counter that
// nothing raises, gives up within about a second and sets ctl->err to kCoopErrWait.
void launch_coop_wait_selftest(cudaStream_t st, CoopControl* ctl);
// The same for the K*u's wait for copies: one CTA waits for a barrier that no copy completes.
void launch_copy_wait_selftest(cudaStream_t st, int* err);

}  // namespace topx
