// Level-1 elasticity kernels of the TOP3D_XL B200 path (the operator is in topx_ku.cu): Jacobi diagonal, PCG vector algebra, trilinear multigrid transfers, SIMP,
// unit compliance.  FP64 (plain path) and FP32 (mixed path) instantiations.
#include <algorithm>
#include <stdexcept>

#include "topx_kernels.cuh"
#include "topx_pcg.cuh"

namespace topx {

__constant__ double c_Ke64[576];

void upload_ke(const double* Ke576) {
  TOPX_CUDA_OK(cudaMemcpyToSymbol(c_Ke64, Ke576, sizeof(double) * 576));
}

static inline unsigned grid1d(int64_t n, int threads, int cap = 148 * 16) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return unsigned(b);
}

// ---------------------------------------------------------------------------
// Finest-level Jacobi diagonal (TOP3D_XL.m:1020-1050): sum over the node's
// hexes, in local-node order, of E_e * diag(Ke); fixed DOFs take cfix.  Stored
// as its reciprocal (0 on absent nodes) so the smoother multiplies.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_diag_l1(Grid g, const double* __restrict__ E, const uint8_t* __restrict__ fixbits,
                          const double* __restrict__ cfix, const uint8_t* __restrict__ present, T* __restrict__ d,
                          double* __restrict__ d0) {
  pdl_wait();
  const int64_t N = g.nnodes();
  const int nny = g.ny + 1, nnx = g.nx + 1;
  for (int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; n < N; n += int64_t(gridDim.x) * blockDim.x) {
    double v[3] = {0.0, 0.0, 0.0}, v0 = 0.0;
    if (present[n]) {
      const int gy = int(n % nny), gx = int((n / nny) % nnx), gz = int(n / (int64_t(nny) * nnx));
      double s[3] = {0.0, 0.0, 0.0};
      for (int a = 0; a < 8; ++a) {
        const int ey = gy - hex_ly(a), ex = gx - hex_lx(a), ez = gz - hex_lz(a);
        if (ey < 0 || ey >= g.ny || ex < 0 || ex >= g.nx || ez < 0 || ez >= g.nz) continue;
        const double Ee = E[ey + int64_t(nny) * (ex + int64_t(nnx) * ez)];
        for (int c = 0; c < 3; ++c) s[c] += c_Ke64[(3 * a + c) * 25] * Ee;
      }
      const uint8_t fb = fixbits[n];
      for (int c = 0; c < 3; ++c) v[c] = 1.0 / ((fb >> c) & 1 ? cfix[n] : s[c]);
      v0 = 1.0 / s[0];
    }
    for (int c = 0; c < 3; ++c) d[n + c * g.stride] = T(v[c]);
    d0[n] = double(T(v0));
  }
}

template <typename T>
void launch_diag_l1(cudaStream_t st, Grid g, const double* E, const uint8_t* fixbits, const double* cfix,
                    const uint8_t* present, T* d, double* d0) {
  launch_pdl(st, k_diag_l1<T>, grid1d(g.nnodes(), 256), 256, 0, g, E, fixbits, cfix, present, d, d0);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// PCG vector algebra (TOP3D_XL.m:613-622)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}
// The first V-cycle of a solve and every iteration run one pass over the level-1 residual: the update
// r -= lambda q (or r = b - q), the sums r'r and r'D r, and the y pass of the restriction from the new
// values.  A lane takes four nodes along y (32 bytes of every field, and a coarse node's own cell: rows hold a
// multiple of four nodes), sums their taps for the coarse node at its first one and for the next one, and hands
// the latter to the next lane; a warp takes whole lines, 32 cells at a time, so that nothing but that
// hand-over, from lane 31 to the next round's lane 0, crosses a round.  z'r needs no pass of its own:
// r'z = omega2 r'D r + (P'r)'xc.
template <int MODE, typename TC>
__global__ void __launch_bounds__(256) k_residual(const __grid_constant__ ResidualArgs a, int lines, int cy, FastDiv dcy) {
  pdl_wait();
  if (MODE == RES_UPDATE) {
    const int done = a.sc->done;
    if (a.parts.rr.n && blockIdx.x == 0 && threadIdx.x == 0) a.sc->ended = done;  // (pcg_ended)
    if (done) return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t S = a.g.stride, nlines = int64_t(a.g.nx + 1) * (a.g.nz + 1), ts = nlines * cy;
  double* __restrict__ const r = a.r;
  const double* __restrict__ const src = MODE == RES_INIT ? a.b : a.r;
  const double* __restrict__ const q = a.q;
  const double* __restrict__ const D = a.D;
  double lam = 0.0;
  int its = 0;
  if (MODE == RES_UPDATE) {
    its = a.sc->its;
    lam = a.sc->zr[its & 1] / (a.parts.pq.n ? parts_sum(a.parts.pq) : a.sc->pq);
  }
  double s0 = 0.0, rd = 0.0;  // b'b or r'r, and r'D r
  const int64_t line0 = (int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5)) * lines;
  const int cells = line0 < nlines ? int(min(int64_t(lines), nlines - line0)) * cy : 0;
  double carry[3] = {0.0, 0.0, 0.0};  // lane 31's part of the next cell's node
  for (int i0 = 0; i0 < cells; i0 += 32) {
    const int i = i0 + lane;
    const int64_t cell = line0 * cy + i, n = 4 * cell;
    double v[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c][0] = v[c][1] = v[c][2] = v[c][3] = 0.0;
    if (i < cells && chunk_active(a.act, n)) {
      double w[3][4], d[4];
      unsigned f = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        load4(src + n + c * S, v[c]);
        if (MODE != RES_KEEP) load4(q + n + c * S, w[c]);
      }
      if (MODE != RES_KEEP) {
        load4(D + n, d);
        f = *reinterpret_cast<const unsigned*>(a.flags + n) & 0x07070707u;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (MODE == RES_INIT) s0 = fma(v[c][k], v[c][k], s0);
            v[c][k] = MODE == RES_INIT ? v[c][k] - w[c][k] : v[c][k] - lam * w[c][k];
            if (MODE == RES_UPDATE) s0 = fma(v[c][k], v[c][k], s0);
          }
          *reinterpret_cast<double2*>(r + n + c * S) = make_double2(v[c][0], v[c][1]);
          *reinterpret_cast<double2*>(r + n + c * S + 2) = make_double2(v[c][2], v[c][3]);
        }
        if (f) {  // fixed DOFs have their own diagonal
          for (int k = 0; k < 4; ++k)
            for (int c = 0; c < 3; ++c)
              rd = fma(v[c][k] * v[c][k], f >> (8 * k + c) & 1u ? double(TC(a.icfix[n + k])) : d[k], rd);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            rd = fma(d[k], fma(v[2][k], v[2][k], fma(v[1][k], v[1][k], v[0][k] * v[0][k])), rd);
        }
      }
    }
    const bool begins = i - cy * int(dcy.div(uint32_t(i))) == 0;  // the line's first cell
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double own = fma(0.25, v[c][3], fma(0.5, v[c][2], fma(0.75, v[c][1], v[c][0])));
      const double next = fma(0.25, v[c][1], fma(0.5, v[c][2], 0.75 * v[c][3]));
      double prev = __shfl_up_sync(0xffffffffu, next, 1);
      if (lane == 0) prev = carry[c];
      carry[c] = __shfl_sync(0xffffffffu, next, 31);
      if (i < cells) a.tmp[cell + c * ts] = begins ? own : own + prev;
    }
  }
  if (MODE == RES_UPDATE && blockIdx.x == 0 && threadIdx.x == 0) {
    a.sc->lam = lam;
    a.sc->its_next = its + 1;
  }
  if (MODE != RES_KEEP && a.parts.rr.n) {  // the x and z passes' kernel sums them
    double t[2] = {s0, rd};
    parts_leave<2>(t, {a.parts.rr.part, a.parts.rd.part});
  } else if (MODE != RES_KEEP) {
    double t[2] = {s0, rd}, tot[2];
    if (reduce_publish<2>(t, a.rs, tot) && threadIdx.x == 0) {
      a.sc->rdr = tot[1];
      if (MODE == RES_INIT)
        pcg_start(a.sc, tot[0], a.tol, a.maxIT);
      else {
        a.sc->its = its + 1;
        pcg_stop_test(a.sc, tot[0], its + 1);
      }
    }
  }
}
// Lines of a warp: fewest rounds of 32 cells one after another, with 24 warps of an SM at a time; of those the fewest
// lines (the reduction at a CTA's end costs about a round)
static int residual_lines(int64_t nlines, int cy) {
  const int64_t slots = 148 * 24;
  int best = 1;
  int64_t bestCost = -1;
  for (int l = 1; l <= 64; ++l) {
    const int64_t warps = (nlines + l - 1) / l, waves = (warps + slots - 1) / slots;
    const int64_t cost = waves * ((int64_t(l) * cy + 31) / 32 + 1);
    if (bestCost < 0 || cost < bestCost) {
      bestCost = cost;
      best = l;
    }
  }
  return best;
}
int residual_blocks(Grid g, Grid gc) {
  const int64_t nlines = int64_t(g.nnx()) * g.nnz();
  const int lines = residual_lines(nlines, gc.nny());
  return int((nlines + 8 * lines - 1) / (8 * lines));
}
void launch_residual(cudaStream_t st, ResidualMode mode, const ResidualArgs& args, Grid gc) {
  const int cy = gc.nny();
  if (args.g.nny() != 4 * cy) throw std::runtime_error("level-1 rows do not hold four nodes per coarse node");
  const int64_t nlines = int64_t(args.g.nnx()) * args.g.nnz();
  const int lines = residual_lines(nlines, cy);
  const unsigned nb = unsigned(residual_blocks(args.g, gc));
  const FastDiv dcy{uint32_t(cy)};
  auto go = [&](auto kernel) { launch_pdl(st, kernel, nb, 256, 0, args, lines, cy, dcy); };
  if (mode == RES_KEEP)
    go(k_residual<RES_KEEP, double>);
  else if (mode == RES_INIT && args.pre32)
    go(k_residual<RES_INIT, float>);
  else if (mode == RES_INIT)
    go(k_residual<RES_INIT, double>);
  else if (args.pre32)
    go(k_residual<RES_UPDATE, float>);
  else
    go(k_residual<RES_UPDATE, double>);
  TOPX_CUDA_OK(cudaGetLastError());
}

// The 'Standard' V-cycle's own residual start and update (it restricts another vector)
__global__ void k_residual_init(Grid g, const double* __restrict__ b, const double* __restrict__ Ay,
                                double* __restrict__ r, PcgScalars* sc, RedScratch rs, double tol, int maxIT) {
  pdl_wait();
  const int64_t N = g.nnodes(), S = g.stride;
  double bb = 0.0;
  for (int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; n < N; n += int64_t(gridDim.x) * blockDim.x) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double bv = b[n + c * S];
      r[n + c * S] = bv - Ay[n + c * S];
      bb += bv * bv;
    }
  }
  double v[1] = {bb}, tot[1];
  if (reduce_publish<1>(v, rs, tot) && threadIdx.x == 0) pcg_start(sc, tot[0], tol, maxIT);
}

void launch_residual_init(cudaStream_t st, Grid g, const double* b, const double* Ay, double* r, PcgScalars* sc,
                          RedScratch rs, double tol, int maxIT) {
  launch_pdl(st, k_residual_init, grid1d(g.nnodes(), 256), 256, 0, g, b, Ay, r, sc, rs, tol, maxIT);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_pcg_update(Grid g, double* __restrict__ r, const double* __restrict__ q, PcgScalars* sc,
                             RedScratch rs, const uint32_t* __restrict__ act) {
  pdl_wait();
  if (sc->done) return;
  const double lam = sc->x1 / sc->pq;
  const int64_t S = g.stride;  // a multiple of 32, so node pairs are aligned
  const int64_t npair = (g.nnodes() + 1) / 2;
  double rr = 0.0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < npair; i += int64_t(gridDim.x) * blockDim.x) {
    if (!chunk_active(act, 2 * i)) continue;  // both nodes of the pair lie in one chunk
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t k = 2 * i + c * S;
      const double2 qv = *reinterpret_cast<const double2*>(q + k);
      double2 rv = *reinterpret_cast<const double2*>(r + k);
      rv.x = rv.x - lam * qv.x;
      rv.y = rv.y - lam * qv.y;
      *reinterpret_cast<double2*>(r + k) = rv;
      rr += rv.x * rv.x + rv.y * rv.y;
    }
  }
  double v[1] = {rr}, tot[1];
  if (reduce_publish<1>(v, rs, tot) && threadIdx.x == 0) {
    sc->lam = lam;
    sc->its += 1;
    pcg_stop_test(sc, tot[0], sc->its);
  }
}
void launch_pcg_update(cudaStream_t st, Grid g, double* r, const double* q, PcgScalars* sc, RedScratch rs,
                       const uint32_t* act) {
  launch_pdl(st, k_pcg_update, grid1d(g.nnodes(), 256), 256, 0, g, r, q, sc, rs, act);
  TOPX_CUDA_OK(cudaGetLastError());
}

// y += sc->lam * p over every node: the solution step of the last PCG iteration (an earlier one's is
// applied by the next K*u)
__global__ void k_pcg_flush(Grid g, double* __restrict__ y, const double* __restrict__ p, const PcgScalars* sc,
                            const uint32_t* __restrict__ act) {
  pdl_wait();
  const double lam = sc->lam;
  const int64_t S = g.stride;
  const int64_t npair = (g.nnodes() + 1) / 2;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < npair; i += int64_t(gridDim.x) * blockDim.x) {
    if (!chunk_active(act, 2 * i)) continue;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t k = 2 * i + c * S;
      const double2 pv = *reinterpret_cast<const double2*>(p + k);
      double2 yv = *reinterpret_cast<const double2*>(y + k);
      yv.x = fma(lam, pv.x, yv.x);
      yv.y = fma(lam, pv.y, yv.y);
      *reinterpret_cast<double2*>(y + k) = yv;
    }
  }
}

void launch_pcg_flush(cudaStream_t st, Grid g, double* y, const double* p, const PcgScalars* sc,
                      const uint32_t* act) {
  launch_pdl(st, k_pcg_flush, grid1d(g.nnodes(), 256), 256, 0, g, y, p, sc, act);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Trilinear restriction R = P^T (Solving_RestrictResidual, TOP3D_XL.m:783-798)
// as separable passes (y, x, z).  Weights (S-|d|)/S are exact in binary,
// equal to the reference's multiGridOperatorRI entries.
// ---------------------------------------------------------------------------
// x and z passes of the level-1 restriction in one launch: 32 neighbouring (y, x) nodes of a coarse plane per
// block, a warp per z tap; the x sums meet in shared memory.  tmp (6 B per level-1 node) comes from L2.
template <typename T>
__global__ void __launch_bounds__(32 * (2 * KU_SPAN - 1)) k_restrict_xz(const double* __restrict__ tmp, int inx, int inz,
                                                                       T* __restrict__ out, double* __restrict__ out64,
                                                                       int64_t ostr, int ony, int onx, FastDiv dy,
                                                                       PcgScalars* sc, PcgParts parts, int init,
                                                                       double tol, int maxIT) {
  pdl_wait();
  if (sc && !init && pcg_ended(sc, parts)) return;
  if (pcg_decide(sc, parts, init != 0, tol, maxIT)) return;
  constexpr int W = 2 * KU_SPAN - 1;
  __shared__ double sx[W][3][32];
  const int lane = threadIdx.x, dz = threadIdx.y, oz = blockIdx.y;
  const uint32_t m = blockIdx.x * 32 + lane, N = uint32_t(ony) * onx;
  const int64_t ts = int64_t(ony) * inx * inz;
  const int iz = KU_SPAN * oz + dz - (KU_SPAN - 1);
  double t[3] = {0.0, 0.0, 0.0};
  if (m < N && iz >= 0 && iz < inz) {
    const int ox = int(dy.div(m)), oy = int(m) - ox * ony;
#pragma unroll
    for (int dx = -(KU_SPAN - 1); dx <= KU_SPAN - 1; ++dx) {
      const int ix = KU_SPAN * ox + dx;
      if (ix < 0 || ix >= inx) continue;
      const double w = double(KU_SPAN - (dx < 0 ? -dx : dx)) / KU_SPAN;
      const int64_t k = oy + int64_t(ony) * (ix + int64_t(inx) * iz);
#pragma unroll
      for (int c = 0; c < 3; ++c) t[c] = fma(w, tmp[k + c * ts], t[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) sx[dz][c][lane] = t[c];
  __syncthreads();
  if (dz < 3 && m < N) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const int d = k - (KU_SPAN - 1);
      s = fma(double(KU_SPAN - (d < 0 ? -d : d)) / KU_SPAN, sx[k][dz][lane], s);
    }
    const int64_t n = m + int64_t(N) * oz + dz * ostr;
    out[n] = T(s);
    if (out64) out64[n] = s;
  }
}
template <typename T>
void launch_restrict_xz(cudaStream_t st, const double* tmp, Grid gf, T* out, double* out64, Grid gc, PcgScalars* sc,
                        const PcgParts* parts, bool init, double tol, int maxIT) {
  const int cy = gc.nny(), cx = gc.nnx();
  const dim3 nb(unsigned((cy * cx + 31) / 32), unsigned(gc.nnz()));
  launch_pdl(st, k_restrict_xz<T>, nb, dim3(32, 2 * KU_SPAN - 1), 0, tmp, gf.nnx(), gf.nnz(), out, out64, gc.stride, cy, cx,
             FastDiv{uint32_t(cy)}, sc, parts ? *parts : PcgParts{}, init ? 1 : 0, tol, maxIT);
  TOPX_CUDA_OK(cudaGetLastError());
}
template void launch_restrict_xz<double>(cudaStream_t, const double*, Grid, double*, double*, Grid, PcgScalars*,
                                         const PcgParts*, bool, double, int);
template void launch_restrict_xz<float>(cudaStream_t, const double*, Grid, float*, double*, Grid, PcgScalars*,
                                        const PcgParts*, bool, double, int);

template <typename T, int S, int AXIS>
__global__ void k_restrict_axis(const T* __restrict__ in, int64_t istr, int iny, int inx, int inz,
                                T* __restrict__ out, int64_t ostr, int ony, int onx, int onz, FastDiv fdy,
                                FastDiv fdx, const PcgScalars* sc) {
  pdl_wait();
  if (sc && sc->done) return;
  const uint32_t N = uint32_t(ony) * onx * onz;
  for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    const uint32_t q = fdy.div(n), oz = fdx.div(q);
    const int oy = int(n - q * uint32_t(ony)), ox = int(q - oz * uint32_t(onx));
    T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int d = -(S - 1); d <= S - 1; ++d) {
      int iy = oy, ix = ox, iz = int(oz);
      int lim;
      if (AXIS == 0) {
        iy = S * oy + d;
        lim = iny;
      } else if (AXIS == 1) {
        ix = S * ox + d;
        lim = inx;
      } else {
        iz = S * int(oz) + d;
        lim = inz;
      }
      const int ia = AXIS == 0 ? iy : (AXIS == 1 ? ix : iz);
      if (ia < 0 || ia >= lim) continue;
      const T w = T(S - (d < 0 ? -d : d)) / T(S);
      const int64_t k = iy + int64_t(iny) * (ix + int64_t(inx) * iz);
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] = fma(w, T(in[k + c * istr]), acc[c]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) out[n + c * ostr] = acc[c];
  }
}

// The restriction between coarse levels in one launch, for grids where launches count: 16 threads per coarse node, one
// per (x, z) column of its 27 fine taps.  Thread (dx, dz) forms the column's y sum as the first axis
// pass does, thread dz of the node the x sum of its columns as the second pass does, and thread 0
// the z sum as the third; each sum keeps the pass's element type and tap order, so the result
// equals the three passes bit for bit.
template <typename T>
__global__ void __launch_bounds__(256) k_restrict_coop(const T* __restrict__ in, int64_t istr, int iny, int inx,
                                                      int inz, T* __restrict__ out, int64_t ostr, int ony, int onx,
                                                      int onz, FastDiv fdy, FastDiv fdx, const PcgScalars* sc) {
  pdl_wait();
  if (sc && sc->done) return;
  constexpr int W = 3, L = 16, NODES = 256 / L;
  __shared__ T sy[NODES][W * W][3];  // y sums of the node's (dx, dz) columns
  __shared__ T sx[NODES][W][3];      // x sums per dz
  const int sub = threadIdx.x / L, lane = threadIdx.x % L;
  const uint32_t N = uint32_t(ony) * onx * onz;
  for (uint32_t base = blockIdx.x * uint32_t(NODES); base < N; base += gridDim.x * uint32_t(NODES)) {
    const uint32_t n = base + uint32_t(sub);
    const bool valid = n < N;
    const uint32_t q = valid ? fdy.div(n) : 0u, oz = valid ? fdx.div(q) : 0u;
    const int oy = int(n - q * uint32_t(ony)), ox = int(q - oz * uint32_t(onx));
    if (valid && lane < W * W) {
      const int ix = 2 * ox + lane % W - 1, iz = 2 * int(oz) + lane / W - 1;
      T t[3] = {T(0), T(0), T(0)};
      if (ix >= 0 && ix < inx && iz >= 0 && iz < inz) {
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy) {
          const int iy = 2 * oy + dy;
          if (iy < 0 || iy >= iny) continue;
          const T w = T(2 - (dy < 0 ? -dy : dy)) / T(2);
          const int64_t k = iy + int64_t(iny) * (ix + int64_t(inx) * iz);
#pragma unroll
          for (int c = 0; c < 3; ++c) t[c] = fma(w, in[k + c * istr], t[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) sy[sub][lane][c] = t[c];
    }
    __syncthreads();
    if (valid && lane < W) {
      T t[3] = {T(0), T(0), T(0)};
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        const int ix = 2 * ox + dx;
        if (ix < 0 || ix >= inx) continue;
        const T w = T(2 - (dx < 0 ? -dx : dx)) / T(2);
#pragma unroll
        for (int c = 0; c < 3; ++c) t[c] = fma(w, sy[sub][lane * W + dx + 1][c], t[c]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) sx[sub][lane][c] = t[c];
    }
    __syncthreads();
    if (valid && lane == 0) {
      T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
      for (int dz = -1; dz <= 1; ++dz) {
        const int iz = 2 * int(oz) + dz;
        if (iz < 0 || iz >= inz) continue;
        const T w = T(2 - (dz < 0 ? -dz : dz)) / T(2);
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] = fma(w, sx[sub][dz + 1][c], acc[c]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) out[n + c * ostr] = acc[c];
    }
    __syncthreads();  // the next nodes' sums reuse the shared arrays
  }
}

template <typename T>
void launch_restrict(cudaStream_t st, const T* in, Grid gf, T* tmp1, T* tmp2, T* out, Grid gc, const PcgScalars* sc) {
  const int fy = gf.nny(), fx = gf.nnx(), fz = gf.nnz();
  const int cy = gc.nny(), cx = gc.nnx(), cz = gc.nnz();
  const int64_t s1 = int64_t(cy) * fx * fz, s2 = int64_t(cy) * cx * fz;
  if (gf.nnodes() >= (int64_t(1) << 32)) throw std::runtime_error("grid too large for 32-bit node indices");
  const FastDiv dcy{uint32_t(cy)}, dfx{uint32_t(fx)}, dcx{uint32_t(cx)};
  if (gf.nnodes() <= kRestrictOneLaunch) {
    launch_pdl(st, k_restrict_coop<T>, grid1d(gc.nnodes() * 16, 256), 256, 0, in, gf.stride, fy, fx, fz, out,
               gc.stride, cy, cx, cz, dcy, dcx, sc);
  } else {
    launch_pdl(st, k_restrict_axis<T, 2, 0>, grid1d(s1, 256), 256, 0, in, gf.stride, fy, fx, fz, tmp1, s1, cy, fx, fz,
               dcy, dfx, sc);
    launch_pdl(st, k_restrict_axis<T, 2, 1>, grid1d(s2, 256), 256, 0, tmp1, s1, cy, fx, fz, tmp2, s2, cy, cx, fz, dcy,
               dcx, sc);
    launch_pdl(st, k_restrict_axis<T, 2, 2>, grid1d(gc.nnodes(), 256), 256, 0, tmp2, s2, cy, cx, fz, out, gc.stride,
               cy, cx, cz, dcy, dcx, sc);
  }
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Prolongation + Jacobi up-smoothing of the 'Adapted' V-cycle
// (TOP3D_XL.m:757-778, Solving_InterpolationDeviation 800-814):
//   x = omega*(r./d) + P*xc + (omega*r)./d   on present fine nodes.
// Inside the PCG the level-2 instance completes z'r (see k_residual) and updates beta/x1
// (TOP3D_XL.m:626-630); the level-1 prolongation itself is formed by the next K*u.
// ---------------------------------------------------------------------------
// SMOOTH = false (the 'Standard' V-cycle) stops after omega*(r/d) + P(xc); the Jacobi
// correction against K x follows in k_jacobi_correct.
template <typename TX, typename T, typename TD, int S, bool DOT, bool SMOOTH = true>
__global__ void __launch_bounds__(256) k_prolong_smooth(const TX* __restrict__ xc, Grid gc, const T* __restrict__ r,
                                                        const TD* __restrict__ dinv,
                                                        const uint8_t* __restrict__ present, T* __restrict__ x,
                                                        Grid gf, FastDiv dny, FastDiv dnx, T omega,
                                                        const double* __restrict__ rc, PcgScalars* sc, RedScratch rs,
                                                        Parts dot, double omega2, const uint32_t* __restrict__ act) {
  pdl_wait();
  if (sc && sc->done) return;
  const uint32_t fny = uint32_t(gf.nny()), fnx = uint32_t(gf.nnx());
  const uint32_t nn = uint32_t(gf.nnodes());  // < 2^32 (checked at launch)
  const int cny = gc.nny(), cnx = gc.nnx();
  double zr = 0.0;
  // grid-stride over the flattened fine grid: no idle lanes on odd extents, and one
  // reduction tail per CTA instead of one per 256 nodes
  for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += gridDim.x * blockDim.x) {
    if (!chunk_active(act, n)) continue;  // x is zero there and stays so
    T rv[3], di[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      rv[c] = r[n + c * gf.stride];
      di[c] = T(dinv[n + c * gf.stride]);
    }
    T v[3] = {T(0), T(0), T(0)};
    if (present[n]) {
      const uint32_t q = dny.div(n);
      const int fy = int(n - q * fny);
      const uint32_t fzu = dnx.div(q);
      const int fz = int(fzu);
      const int fx = int(q - fzu * fnx);
      const int Y = fy / S, X = fx / S, Z = fz / S;
      const int ty = fy - S * Y, tx = fx - S * X, tz = fz - S * Z;
      T pc[3] = {T(0), T(0), T(0)};
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        // corner a of the coarse hex, summed in the reference's local-node order
        const int oy = hex_ly(a), ox = hex_lx(a), oz = hex_lz(a);
        if ((oy && ty == 0) || (ox && tx == 0) || (oz && tz == 0)) continue;
        const T wy = oy ? T(ty) / T(S) : T(S - ty) / T(S);
        const T wx = ox ? T(tx) / T(S) : T(S - tx) / T(S);
        const T wz = oz ? T(tz) / T(S) : T(S - tz) / T(S);
        const T w = wy * wx * wz;
        const int64_t k = (Y + oy) + int64_t(cny) * ((X + ox) + int64_t(cnx) * (Z + oz));
#pragma unroll
        for (int c = 0; c < 3; ++c) pc[c] = fma(w, T(xc[k + c * gc.stride]), pc[c]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T t = omega * (rv[c] * di[c]);
        t = t + pc[c];
        if (SMOOTH) t = t + (omega * rv[c]) * di[c];
        v[c] = t;
        if (DOT) zr = fma(double(t), rc[n + c * gf.stride], zr);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) x[n + c * gf.stride] = v[c];
  }
  if (DOT && dot.n) {  // the next K*u sums them
    double vv[1] = {zr};
    parts_leave<1>(vv, {dot.part});
  } else if (DOT) {
    double vv[1] = {zr}, tot[1];
    if (reduce_publish<1>(vv, rs, tot) && threadIdx.x == 0) {
      const int its = sc->its;
      const double x2 = fma(omega2, sc->rdr, tot[0]);
      if (its > 0) sc->beta = x2 / sc->zr[(its - 1) & 1];
      sc->zr[its & 1] = x2;
    }
  }
}

int prolong_blocks(Grid gf) { return int(grid1d(gf.nnodes(), 256, 148 * 8)); }

template <typename TX, typename T, typename TD>
void launch_prolong_smooth(cudaStream_t st, int span, const TX* xc, Grid gc, const T* r, const TD* d,
                           const uint8_t* present, T* x, Grid gf, double omega, const double* rc, Parts dot,
                           PcgScalars* sc, RedScratch rs, const uint32_t* act) {
  if (gf.nnodes() >= (int64_t(1) << 32)) throw std::runtime_error("grid too large for 32-bit node indices");
  const unsigned nb = unsigned(prolong_blocks(gf));
  const FastDiv dny{uint32_t(gf.nny())}, dnx{uint32_t(gf.nnx())};
  auto go = [&](auto kernel) {
    launch_pdl(st, kernel, nb, 256, 0, xc, gc, r, d, present, x, gf, dny, dnx, T(omega), rc, sc, rs, dot,
               2.0 * omega, act);
  };
  if (span == 4)
    go(k_prolong_smooth<TX, T, TD, 4, false>);
  else if (rc)
    go(k_prolong_smooth<TX, T, TD, 2, true>);
  else
    go(k_prolong_smooth<TX, T, TD, 2, false>);
  TOPX_CUDA_OK(cudaGetLastError());
}

template <typename TX, typename T, typename TD>
void launch_prolong_add(cudaStream_t st, int span, const TX* xc, Grid gc, const T* r, const TD* d,
                        const uint8_t* present, T* x, Grid gf, double omega, PcgScalars* sc) {
  const unsigned nb = grid1d(gf.nnodes(), 256, 148 * 8);
  RedScratch none{nullptr, nullptr};
  if (gf.nnodes() >= (int64_t(1) << 32)) throw std::runtime_error("grid too large for 32-bit node indices");
  const FastDiv dny{uint32_t(gf.nny())}, dnx{uint32_t(gf.nnx())};
  auto go = [&](auto kernel) {
    launch_pdl(st, kernel, nb, 256, 0, xc, gc, r, d, present, x, gf, dny, dnx, T(omega), nullptr, sc, none,
               Parts{}, 0.0, nullptr);
  };
  if (span == 4)
    go(k_prolong_smooth<TX, T, TD, 4, false, false>);
  else
    go(k_prolong_smooth<TX, T, TD, 2, false, false>);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// 'Standard' V-cycle pieces (TOP3D_XL.m:758-763, 772-777): pre-smoothing from zero, the
// residual r - K x, and the Jacobi correction after the coarse-grid correction.  All return at
// once when the PCG has finished (sc->done), like the prolongation that writes the V-cycle
// output.
// ---------------------------------------------------------------------------
// x = omega*(r/d) on present nodes (the first line of the restriction loop, TX:757)
template <typename TR, typename T, typename TD>
__global__ void k_jacobi_pre(Grid g, const TR* __restrict__ r, const TD* __restrict__ dinv,
                             const uint8_t* __restrict__ present, T* __restrict__ x, T omega, const PcgScalars* sc) {
  pdl_wait();
  if (sc->done) return;
  const int64_t N = g.nnodes();
  for (int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; n < N; n += int64_t(gridDim.x) * blockDim.x) {
    const bool pres = present[n] != 0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      x[n + c * g.stride] = pres ? omega * (T(r[n + c * g.stride]) * T(dinv[n + c * g.stride])) : T(0);
  }
}
template <typename TR, typename T, typename TD>
void launch_jacobi_pre(cudaStream_t st, Grid g, const TR* r, const TD* d, const uint8_t* present, T* x, double omega,
                       const PcgScalars* sc) {
  launch_pdl(st, k_jacobi_pre<TR, T, TD>, grid1d(g.nnodes(), 256), 256, 0, g, r, d, present, x, T(omega), sc);
  TOPX_CUDA_OK(cudaGetLastError());
}

// q = r - q: the residual after pre-smoothing, restricted next (TX:761-762).  Zero on absent nodes: where the K*u's tiles
// leave some out, q keeps what stands there, a NaN of an earlier solve too.
template <typename TR, typename T>
__global__ void k_residual_inplace(Grid g, const TR* __restrict__ r, const uint8_t* __restrict__ present,
                                   T* __restrict__ q, const PcgScalars* sc) {
  pdl_wait();
  if (sc->done) return;
  const int64_t N = g.nnodes();
  for (int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; n < N; n += int64_t(gridDim.x) * blockDim.x) {
    const bool pres = present[n] != 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) q[n + c * g.stride] = pres ? T(r[n + c * g.stride]) - q[n + c * g.stride] : T(0);
  }
}
template <typename TR, typename T>
void launch_residual_inplace(cudaStream_t st, Grid g, const TR* r, const uint8_t* present, T* q, const PcgScalars* sc) {
  launch_pdl(st, k_residual_inplace<TR, T>, grid1d(g.nnodes(), 256), 256, 0, g, r, present, q, sc);
  TOPX_CUDA_OK(cudaGetLastError());
}

// x = x + omega*(r - q)/d on present nodes, q = K x (TX:775-776); the finest instance also
// reduces z'r and updates beta/x1 like the 'Adapted' prolongation (TX:626-630)
template <typename TR, typename T, typename TD, bool DOT>
__global__ void __launch_bounds__(256) k_jacobi_correct(Grid g, const TR* __restrict__ r, const T* __restrict__ q,
                                                        const TD* __restrict__ dinv,
                                                        const uint8_t* __restrict__ present, T* __restrict__ x,
                                                        T omega, PcgScalars* sc, RedScratch rs, int init) {
  pdl_wait();
  if (sc->done) return;
  const int64_t N = g.nnodes();
  double zr = 0.0;
  for (int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; n < N; n += int64_t(gridDim.x) * blockDim.x) {
    const bool pres = present[n] != 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = n + c * g.stride;
      const T rv = T(r[i]);
      const T t = pres ? x[i] + (omega * (rv - q[i])) * T(dinv[i]) : T(0);
      x[i] = t;
      if (DOT) zr += double(t) * double(rv);
    }
  }
  if (DOT) {
    double vv[1] = {zr}, tot[1];
    if (reduce_publish<1>(vv, rs, tot) && threadIdx.x == 0) {
      if (init) {
        sc->x1 = tot[0];
      } else {
        sc->beta = tot[0] / sc->x1;
        sc->x1 = tot[0];
      }
    }
  }
}
template <typename TR, typename T, typename TD>
void launch_jacobi_correct(cudaStream_t st, Grid g, const TR* r, const T* q, const TD* d, const uint8_t* present,
                           T* x, double omega, bool dot, bool init, PcgScalars* sc, RedScratch rs) {
  const unsigned nb = grid1d(g.nnodes(), 256, 148 * 8);
  if (dot)
    launch_pdl(st, k_jacobi_correct<TR, T, TD, true>, nb, 256, 0, g, r, q, d, present, x, T(omega), sc, rs,
               init ? 1 : 0);
  else
    launch_pdl(st, k_jacobi_correct<TR, T, TD, false>, nb, 256, 0, g, r, q, d, present, x, T(omega), sc, rs,
               init ? 1 : 0);
  TOPX_CUDA_OK(cudaGetLastError());
}

// K*u on a coarse level with its stored Galerkin matrices (Solving_KbyU_MatrixFree for
// iLevel > 1, TOP3D_XL.m:727-743).  One thread per node: for each hex around it, in
// local-node order (the order accumarray adds them), the product of the node's three rows of
// Ks_e with the hex's 24 DOFs, then the sum over hexes.  Deterministic, no atomics.  The
// reference forms u_e' Ks_e; the Galerkin matrices are symmetric, so rows serve for columns (up
// to the rounding of their assembly).
__global__ void __launch_bounds__(256) k_ku_coarse(Grid g, const double* __restrict__ Ks,
                                                   const uint8_t* __restrict__ epresent,
                                                   const uint8_t* __restrict__ present, const double* __restrict__ u,
                                                   double* __restrict__ y, const PcgScalars* sc) {
  pdl_wait();
  if (sc->done) return;
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
        if (!epresent[e]) continue;
        const double* K = Ks + e * 576 + (3 * a) * 24;  // rows 3a .. 3a + 2
        double t[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const int64_t m = (ey + hex_ly(b)) + int64_t(nny) * ((ex + hex_lx(b)) + int64_t(nnx) * (ez + hex_lz(b)));
          const double u0 = u[m], u1 = u[m + g.stride], u2 = u[m + 2 * g.stride];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            t[c] = fma(K[c * 24 + 3 * b], u0, t[c]);
            t[c] = fma(K[c * 24 + 3 * b + 1], u1, t[c]);
            t[c] = fma(K[c * 24 + 3 * b + 2], u2, t[c]);
          }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) s[c] += t[c];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) y[n + c * g.stride] = s[c];
  }
}
void launch_ku_coarse(cudaStream_t st, Grid g, const double* Ks, const uint8_t* epresent, const uint8_t* present,
                      const double* u, double* y, const PcgScalars* sc) {
  launch_pdl(st, k_ku_coarse, grid1d(g.nnodes(), 256), 256, 0, g, Ks, epresent, present, u, y, sc);
  TOPX_CUDA_OK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// conversions between the reference's compact numbering and the dense grid
// ---------------------------------------------------------------------------
template <typename TA, typename TB>
__global__ void k_convert(const TA* __restrict__ a, TB* __restrict__ b, int64_t n) {
  pdl_wait();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    b[i] = TB(a[i]);
}
template <typename TA, typename TB>
void launch_convert(cudaStream_t st, const TA* a, TB* b, int64_t n) {
  launch_pdl(st, k_convert<TA, TB>, grid1d(n, 256), 256, 0, a, b, n);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_index_nodes(const int32_t* __restrict__ nmb0, int64_t nn, int32_t* __restrict__ node_id) {
  pdl_wait();
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < nn; k += int64_t(gridDim.x) * blockDim.x)
    node_id[nmb0[k]] = int32_t(k);
}
void launch_index_nodes(cudaStream_t st, const int32_t* nodMapBack0, int64_t numNodes, int32_t* node_id, int64_t n) {
  TOPX_CUDA_OK(cudaMemsetAsync(node_id, 0xff, sizeof(int32_t) * size_t(n), st));
  launch_pdl(st, k_index_nodes, grid1d(numNodes, 256), 256, 0, nodMapBack0, numNodes, node_id);
  TOPX_CUDA_OK(cudaGetLastError());
}

__global__ void k_invert(int64_t n, const double* __restrict__ a, double* __restrict__ out) {
  pdl_wait();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = a[i] != 0.0 ? 1.0 / a[i] : 0.0;
}
void launch_invert(cudaStream_t st, int64_t n, const double* a, double* out) {
  launch_pdl(st, k_invert, grid1d(n, 256), 256, 0, n, a, out);
  TOPX_CUDA_OK(cudaGetLastError());
}

// interleaved compact DOF vector (3k+c) -> SoA dense grid field with unknown contents: every entry is written, zero
// where the domain has no node (node_id: compact id of a grid node or -1), so that the field needs no zeroing first.
__global__ void k_fill_grid_nodes(const double* __restrict__ src, double* __restrict__ dst, int64_t nnodes,
                                  int64_t stride, const int32_t* __restrict__ node_id) {
  pdl_wait();
  for (int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; n < stride; n += int64_t(gridDim.x) * blockDim.x) {
    const int64_t k = n < nnodes ? node_id[n] : -1;
    for (int c = 0; c < 3; ++c) dst[n + c * stride] = k >= 0 ? src[3 * k + c] : 0.0;
  }
}
void launch_fill_grid_nodes(cudaStream_t st, const double* src, double* dst, Grid g, const int32_t* node_id) {
  launch_pdl(st, k_fill_grid_nodes, grid1d(g.stride, 256), 256, 0, src, dst, g.nnodes(), g.stride, node_id);
  TOPX_CUDA_OK(cudaGetLastError());
}

// interleaved compact DOF vector (3k+c) -> SoA dense grid field
template <typename T>
__global__ void k_c2g_nodes(const double* __restrict__ src, T* __restrict__ dst, Grid g,
                            const int32_t* __restrict__ nmb0, int64_t nn) {
  pdl_wait();
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < nn; k += int64_t(gridDim.x) * blockDim.x) {
    const int64_t n = nmb0[k];
    for (int c = 0; c < 3; ++c) dst[n + c * g.stride] = T(src[3 * k + c]);
  }
}
template <typename T>
void launch_compact_to_grid_nodes(cudaStream_t st, const double* src, T* dst, Grid g, const int32_t* nodMapBack0,
                                  int64_t numNodes) {
  launch_pdl(st, k_c2g_nodes<T>, grid1d(numNodes, 256), 256, 0, src, dst, g, nodMapBack0, numNodes);
  TOPX_CUDA_OK(cudaGetLastError());
}
template <typename T>
__global__ void k_g2c_nodes(const T* __restrict__ src, double* __restrict__ dst, Grid g,
                            const int32_t* __restrict__ nmb0, int64_t nn) {
  pdl_wait();
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < nn; k += int64_t(gridDim.x) * blockDim.x) {
    const int64_t n = nmb0[k];
    for (int c = 0; c < 3; ++c) dst[3 * k + c] = double(src[n + c * g.stride]);
  }
}
template <typename T>
void launch_grid_to_compact_nodes(cudaStream_t st, const T* src, double* dst, Grid g, const int32_t* nodMapBack0,
                                  int64_t numNodes) {
  launch_pdl(st, k_g2c_nodes<T>, grid1d(numNodes, 256), 256, 0, src, dst, g, nodMapBack0, numNodes);
  TOPX_CUDA_OK(cudaGetLastError());
}

// SIMP moduli E = Emin + xPhys^p (E0 - Emin), compact -> dense (TOP3D_XL.m:107,116)
__global__ void k_simp_scatter(const double* __restrict__ x, const int32_t* __restrict__ emb0, int64_t Ne,
                               double Emin, double E0, double penal, double* __restrict__ Ed,
                               float* __restrict__ Ef) {
  pdl_wait();
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    const double v = Emin + pow(x[e], penal) * (E0 - Emin);
    const int64_t k = emb0[e];
    Ed[k] = v;
    if (Ef) Ef[k] = float(v);
  }
}
void launch_simp_scatter(cudaStream_t st, const double* xPhys, const int32_t* eleMapBack0, int64_t Ne, double Emin,
                         double E0, double penal, double* Ed, float* Ef) {
  launch_pdl(st, k_simp_scatter, grid1d(Ne, 256), 256, 0, xPhys, eleMapBack0, Ne, Emin, E0, penal, Ed, Ef);
  TOPX_CUDA_OK(cudaGetLastError());
}

// TopOpti_ComputeUnitCompliance (TOP3D_XL.m:579-598): ce_e = u_e^T Ke u_e with the
// unmodified Ke, one thread per element (compact order), FP64.
__global__ void k_unit_compliance(Grid g, const double* __restrict__ U, const int32_t* __restrict__ emb0,
                                  int64_t Ne, double w, int acc, double* __restrict__ ce) {
  pdl_wait();
  const int nny = g.ny + 1, nnx = g.nx + 1;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t id = emb0[e];  // the index of its lowest node
    double u[24];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int64_t n = id + hex_ly(a) + int64_t(nny) * (hex_lx(a) + int64_t(nnx) * hex_lz(a));
#pragma unroll
      for (int c = 0; c < 3; ++c) u[3 * a + c] = U[n + c * g.stride];
    }
    // Ke is symmetric: u^T Ke u = sum_j u_j (Ke_jj u_j + 2 sum_{i<j} Ke_ij u_i), 324 FMA for 600
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 24; ++j) {
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < j; ++i) t = fma(u[i], c_Ke64[i * 24 + j], t);
      s = fma(u[j], fma(2.0, t, c_Ke64[j * 24 + j] * u[j]), s);
    }
    ce[e] = acc ? ce[e] + w * s : w * s;
  }
}
void launch_unit_compliance(cudaStream_t st, Grid g, const double* U, const int32_t* eleMapBack0, int64_t Ne,
                            double weight, bool accumulate, double* ce) {
  launch_pdl(st, k_unit_compliance, grid1d(Ne, 128), 128, 0, g, U, eleMapBack0, Ne, weight, accumulate ? 1 : 0, ce);
  TOPX_CUDA_OK(cudaGetLastError());
}

// explicit instantiations
#define TOPX_INST(T)                                                                                             \
  template void launch_diag_l1<T>(cudaStream_t, Grid, const double*, const uint8_t*, const double*,              \
                                  const uint8_t*, T*, double*);                                                    \
  template void launch_restrict<T>(cudaStream_t, const T*, Grid, T*, T*, T*, Grid, const PcgScalars*);           \
  template void launch_prolong_smooth<T, T, T>(cudaStream_t, int, const T*, Grid, const T*, const T*,            \
                                               const uint8_t*, T*, Grid, double, const double*, Parts,           \
                                               PcgScalars*, RedScratch, const uint32_t*);
TOPX_INST(double)
TOPX_INST(float)
template void launch_compact_to_grid_nodes<double>(cudaStream_t, const double*, double*, Grid, const int32_t*, int64_t);
template void launch_grid_to_compact_nodes<double>(cudaStream_t, const double*, double*, Grid, const int32_t*, int64_t);
template void launch_prolong_smooth<float, double, float>(cudaStream_t, int, const float*, Grid, const double*,
                                                          const float*, const uint8_t*, double*, Grid, double,
                                                          const double*, Parts, PcgScalars*, RedScratch, const uint32_t*);
template void launch_prolong_add<double, double, double>(cudaStream_t, int, const double*, Grid, const double*,
                                                        const double*, const uint8_t*, double*, Grid, double,
                                                        PcgScalars*);
template void launch_jacobi_pre<double, double, double>(cudaStream_t, Grid, const double*, const double*,
                                                        const uint8_t*, double*, double, const PcgScalars*);
template void launch_residual_inplace<double, double>(cudaStream_t, Grid, const double*, const uint8_t*, double*,
                                                      const PcgScalars*);
template void launch_jacobi_correct<double, double, double>(cudaStream_t, Grid, const double*, const double*,
                                                            const double*, const uint8_t*, double*, double, bool,
                                                            bool, PcgScalars*, RedScratch);
template void launch_convert<double, float>(cudaStream_t, const double*, float*, int64_t);
template void launch_convert<float, double>(cudaStream_t, const float*, double*, int64_t);
template void launch_convert<double, double>(cudaStream_t, const double*, double*, int64_t);

}  // namespace topx

namespace topx {

// E = val on every solid element (compact -> dense); the solid-domain solve of
// TOP3D_XL.m:94-104 uses repmat(modulus_) rather than SIMP(1).
__global__ void k_fill_scatter(const int32_t* __restrict__ emb0, int64_t Ne, double val, double* __restrict__ Ed,
                               float* __restrict__ Ef) {
  pdl_wait();
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    Ed[emb0[e]] = val;
    if (Ef) Ef[emb0[e]] = float(val);
  }
}
void launch_fill_scatter(cudaStream_t st, const int32_t* eleMapBack0, int64_t Ne, double val, double* Ed, float* Ef) {
  launch_pdl(st, k_fill_scatter, grid1d(Ne, 256), 256, 0, eleMapBack0, Ne, val, Ed, Ef);
  TOPX_CUDA_OK(cudaGetLastError());
}

}  // namespace topx
