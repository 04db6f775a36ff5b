// Coarse-level kernels of the TOP3D_XL B200 path (Solving_AssembleFEAstencil,
// TOP3D_XL.m:919-1018): Galerkin element operators per level and their Jacobi diagonals.
// The coarsest level's direct solver is in topx_nd.cu.
#include <algorithm>
#include <mutex>

#include "topx_kernels.cuh"

namespace topx {

static inline unsigned grid1d(int64_t n, int threads, int cap = 148 * 16) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return unsigned(b);
}

// ---------------------------------------------------------------------------
// Level-2 Galerkin operators (TOP3D_XL.m:946-978): Ks2_j = sum_c E_c T_c over the
// 64 children of every dense level-2 element (void children have E = 0).
// ---------------------------------------------------------------------------
// Blocks [0, nflag): one level-2 element that holds children with fixed DOFs each (TOP3D_XL.m:961-971):
// Ks2_j = sum_c E_c T_sel(j,c) + F_j, where T_sel is the child's template or the template of its BC-modified Ke
// (uniqueKesFree_), and F_j collects the E-independent uniqueKesFixed_ parts.  The other blocks take ELEMS
// elements each, sharing every template entry that they read, and leave the flagged ones out.  Few elements: blocks
// of 2, so that small grids use more SMs, their 64 template rows prefetched (16 x 32 x 16 elements: 32 us as two
// launches, now 23; 50 x 100 x 50: 54, now 36; 64 x 128 x 64, in blocks of 16: 70, now 54).
constexpr int GL2_THREADS = 192;

template <int ELEMS>
__global__ void __launch_bounds__(GL2_THREADS) k_galerkin_l2(Grid gf, Grid gc, const double* __restrict__ Ef,
                                                             const double* __restrict__ Tm, int nflag,
                                                             const int32_t* __restrict__ fl_elem,
                                                             const int32_t* __restrict__ fl_tsel,
                                                             const double* __restrict__ fl_F,
                                                             const uint8_t* __restrict__ flagged,
                                                             double* __restrict__ Ks) {
  pdl_wait();
  __shared__ double sE[ELEMS][64];
  const int64_t nce = gc.nelems();
  const int fny = gf.nny(), fnx = gf.nnx(), tid = threadIdx.x;
  auto child = [&](int64_t j, int c) {
    const int gy = int(j % gc.ny), gx = int((j / gc.ny) % gc.nx), gz = int(j / (int64_t(gc.ny) * gc.nx));
    const int cy = c & 3, cx = (c >> 2) & 3, cz = c >> 4;
    return Ef[(4 * gy + cy) + int64_t(fny) * ((4 * gx + cx) + int64_t(fnx) * (4 * gz + cz))];
  };
  if (int(blockIdx.x) < nflag) {
    __shared__ int sT[64];
    const int f = blockIdx.x;
    const int64_t j = fl_elem[f];
    for (int c = tid; c < 64; c += GL2_THREADS) {
      sE[0][c] = child(j, c);
      sT[c] = fl_tsel[f * 64 + c];
    }
    __syncthreads();
    double a[3] = {0.0, 0.0, 0.0};
#pragma unroll 8
    for (int c = 0; c < 64; ++c) {
      const double* T = Tm + int64_t(sT[c]) * 576 + tid;
#pragma unroll
      for (int k = 0; k < 3; ++k) a[k] = fma(sE[0][c], __ldg(T + k * GL2_THREADS), a[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      Ks[j * 576 + tid + k * GL2_THREADS] = a[k] + fl_F[int64_t(f) * 576 + tid + k * GL2_THREADS];
    return;
  }
  const int64_t j0 = int64_t(int(blockIdx.x) - nflag) * ELEMS;
  bool any = false;
  for (int i = tid; i < ELEMS * 64; i += GL2_THREADS) {
    const int64_t j = j0 + i / 64;
    const double v = j < nce ? child(j, i % 64) : 0.0;
    sE[i / 64][i % 64] = v;
    any = any || v != 0.0;
  }
  // a group of coarse elements whose children are all void (E = 0) sums to zero: write it
  // without streaming the templates (irregular domains)
  if (!__syncthreads_or(any)) {
    for (int jj = 0; jj < ELEMS; ++jj) {
      const int64_t j = j0 + jj;
      if (j < nce && !(nflag && flagged[j]))
        for (int k = tid; k < 576; k += GL2_THREADS) Ks[j * 576 + k] = 0.0;
    }
    return;
  }
  double acc[ELEMS][3];
#pragma unroll
  for (int jj = 0; jj < ELEMS; ++jj) acc[jj][0] = acc[jj][1] = acc[jj][2] = 0.0;
#pragma unroll(ELEMS > 4 ? 2 : 8)
  for (int c = 0; c < 64; ++c) {
    const double t0 = __ldg(&Tm[c * 576 + tid]);
    const double t1 = __ldg(&Tm[c * 576 + tid + GL2_THREADS]);
    const double t2 = __ldg(&Tm[c * 576 + tid + 2 * GL2_THREADS]);
#pragma unroll
    for (int jj = 0; jj < ELEMS; ++jj) {
      const double e = sE[jj][c];
      acc[jj][0] = fma(e, t0, acc[jj][0]);
      acc[jj][1] = fma(e, t1, acc[jj][1]);
      acc[jj][2] = fma(e, t2, acc[jj][2]);
    }
  }
#pragma unroll
  for (int jj = 0; jj < ELEMS; ++jj) {
    const int64_t j = j0 + jj;
    if (j < nce && !(nflag && flagged[j])) {
      Ks[j * 576 + tid] = acc[jj][0];
      Ks[j * 576 + tid + GL2_THREADS] = acc[jj][1];
      Ks[j * 576 + tid + 2 * GL2_THREADS] = acc[jj][2];
    }
  }
}

void launch_galerkin_l2(cudaStream_t st, Grid gf, Grid gc, const double* Efine, const double* Tm, int nflag,
                        const int32_t* fl_elem, const int32_t* fl_tsel, const double* fl_F, const uint8_t* flagged,
                        double* Ks) {
  const int64_t n = gc.nelems();
  if (n < 148 * 16)
    launch_pdl(st, k_galerkin_l2<2>, unsigned(nflag + (n + 1) / 2), GL2_THREADS, 0, gf, gc, Efine, Tm, nflag, fl_elem,
               fl_tsel, fl_F, flagged, Ks);
  else
    launch_pdl(st, k_galerkin_l2<16>, unsigned(nflag + (n + 15) / 16), GL2_THREADS, 0, gf, gc, Efine, Tm, nflag, fl_elem,
               fl_tsel, fl_F, flagged, Ks);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Span-2 Galerkin operators of levels >= 3 (TOP3D_XL.m:979-995):
// Ks_J = sum_{c<8} P_c^T Ks_child(c) P_c.
// ---------------------------------------------------------------------------
// The child prolongators are P_c = W_c (x) I_3 (DOFs interleaved, 3 a + i), and W_c is itself a product of one 2x2
// matrix per axis: towards the child's side of the axis its far node is the midpoint of the coarse pair, its near node
// a coarse node.  A transform of the eight nodes' values is therefore four exact halvings and additions per axis
// (12 of each), from registers, instead of 64 multiply-adds with both operands from shared memory, whose loads
// bounded it (all levels of 128 x 256 x 128 elements: 328 us, now 110; 64 x 128 x 64: 49, now 20).
constexpr int GS2_THREADS = 192;

// v[a] (a: local node of the child) summed to the coarse nodes: out[b] = sum_a W_c[a][b] v[a]
__device__ __forceinline__ void gs2_to_coarse(double (&v)[8], int cy, int cx, int cz) {
  auto axis = [&](int lo, int hi, int side) {
    // child on the low side: its low node is the coarse low node, its high node the midpoint; high side: mirrored
    const double l = v[lo], h = v[hi], m = 0.5 * (side ? l : h);
    v[lo] = side ? m : l + m;
    v[hi] = side ? h + m : m;
  };
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int z = 0; z < 2; ++z) axis(hex_local(0, x, z), hex_local(1, x, z), cy);
#pragma unroll
  for (int y = 0; y < 2; ++y)
#pragma unroll
    for (int z = 0; z < 2; ++z) axis(hex_local(y, 0, z), hex_local(y, 1, z), cx);
#pragma unroll
  for (int y = 0; y < 2; ++y)
#pragma unroll
    for (int x = 0; x < 2; ++x) axis(hex_local(y, x, 0), hex_local(y, x, 1), cz);
}

__global__ void __launch_bounds__(GS2_THREADS) k_galerkin_span2(Grid gc, const double* __restrict__ Ksf,
                                                                const uint8_t* __restrict__ cpresent,
                                                                double* __restrict__ Ks) {
  pdl_wait();
  __shared__ double sK[8 * 576];  // the 8 children's operators, then T_c = K_c (W_c (x) I) in place
  const int64_t J = blockIdx.x;
  const int tid = threadIdx.x;
  if (!cpresent[J]) {  // the same for the whole CTA
    for (int k = tid; k < 576; k += GS2_THREADS) Ks[J * 576 + k] = 0.0;
    return;
  }
  const int gy = int(J % gc.ny), gx = int((J / gc.ny) % gc.nx), gz = int(J / (int64_t(gc.ny) * gc.nx));
  const int fny = 2 * gc.ny, fnx = 2 * gc.nx;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int cy = c & 1, cx = (c >> 1) & 1, cz = c >> 2;
    const int64_t f = (2 * gy + cy) + int64_t(fny) * ((2 * gx + cx) + int64_t(fnx) * (2 * gz + cz));
#pragma unroll
    for (int k = 0; k < 3; ++k) sK[c * 576 + tid + k * GS2_THREADS] = Ksf[f * 576 + tid + k * GS2_THREADS];
  }
  __syncthreads();
  // a thread per child, row and component of the columns (8 x 24 x 3): its eight entries, 3 apart
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    const int o = tid + u * GS2_THREADS, c = o / 72, rem = o - 72 * c, r = rem / 3, j = rem - 3 * r;
    double* K = sK + c * 576 + r * 24 + j;
    double v[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) v[a] = K[3 * a];
    gs2_to_coarse(v, c & 1, (c >> 1) & 1, c >> 2);
#pragma unroll
    for (int a = 0; a < 8; ++a) K[3 * a] = v[a];
  }
  __syncthreads();
  // the rows: a thread per column, component and half of the children (24 x 3 x 2); the halves meet in shared memory
  double s[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) s[a] = 0.0;
  const int half = tid / 72, rem = tid - 72 * half, col = rem / 3, i = rem - 3 * col;
  if (half < 2)
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) {
      const int c = 4 * half + c4;
      double v[8];
#pragma unroll
      for (int a = 0; a < 8; ++a) v[a] = sK[c * 576 + (3 * a + i) * 24 + col];
      gs2_to_coarse(v, c & 1, (c >> 1) & 1, c >> 2);
#pragma unroll
      for (int a = 0; a < 8; ++a) s[a] += v[a];
    }
  __syncthreads();
  if (half < 2)
#pragma unroll
    for (int a = 0; a < 8; ++a) sK[half * 576 + (3 * a + i) * 24 + col] = s[a];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int o = tid + k * GS2_THREADS;
    Ks[J * 576 + o] = sK[o] + sK[576 + o];
  }
}

void launch_galerkin_span2(cudaStream_t st, Grid gc, const double* Ksf, const uint8_t* cpresent, double* Ks) {
  launch_pdl(st, k_galerkin_span2, unsigned(gc.nelems()), GS2_THREADS, 0, gc, Ksf, cpresent, Ks);
  TOPX_CUDA_OK(cudaGetLastError());
}

// Jacobi diagonal of a coarse level from its element operators (TOP3D_XL.m:1000-1018),
// stored as its reciprocal (0 on absent nodes) so the smoother multiplies
template <typename T>
__global__ void k_diag_coarse(Grid g, const double* __restrict__ Ks, const uint8_t* __restrict__ present,
                              T* __restrict__ d) {
  pdl_wait();
  const int64_t N = g.nnodes();
  const int nny = g.ny + 1, nnx = g.nx + 1;
  for (int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; n < N; n += int64_t(gridDim.x) * blockDim.x) {
    double s[3] = {0.0, 0.0, 0.0};
    if (present[n]) {
      const int gy = int(n % nny), gx = int((n / nny) % nnx), gz = int(n / (int64_t(nny) * nnx));
      for (int a = 0; a < 8; ++a) {
        const int ey = gy - hex_ly(a), ex = gx - hex_lx(a), ez = gz - hex_lz(a);
        if (ey < 0 || ey >= g.ny || ex < 0 || ex >= g.nx || ez < 0 || ez >= g.nz) continue;
        const int64_t e = ey + int64_t(g.ny) * (ex + int64_t(g.nx) * ez);
        for (int c = 0; c < 3; ++c) s[c] += Ks[e * 576 + (3 * a + c) * 25];
      }
      for (int c = 0; c < 3; ++c) s[c] = 1.0 / s[c];
    }
    for (int c = 0; c < 3; ++c) d[n + c * g.stride] = T(s[c]);
  }
}

template <typename T>
void launch_diag_coarse(cudaStream_t st, Grid g, const double* Ks, const uint8_t* present, T* d) {
  launch_pdl(st, k_diag_coarse<T>, grid1d(g.nnodes(), 256), 256, 0, g, Ks, present, d);
  TOPX_CUDA_OK(cudaGetLastError());
}


template void launch_diag_coarse<double>(cudaStream_t, Grid, const double*, const uint8_t*, double*);
template void launch_diag_coarse<float>(cudaStream_t, Grid, const double*, const uint8_t*, float*);

}  // namespace topx
