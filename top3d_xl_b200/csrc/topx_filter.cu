// The PDE (Helmholtz) density filter of the TOP3D_XL B200 path (TOP3D_XL.m:816-917): a Jacobi-preconditioned CG on
// the nodes of the solid domain, matrix-free.
//
// A cube's scalar element matrix is diagonal in the basis of sums and differences of its corner values along the
// three axes (a Walsh transform), with four values by the number of differences: 8 products instead of 64, and
// the transforms are shared between neighbours as in the elasticity operator (topx_ku.cu), whose tiles and TMA
// pipeline this one has too.  The inverse diagonal depends only on a node's number of solid elements, so one byte per
// node holds it and the solid flag of the element above.  A CG iteration is two launches: the operator forms
// p = D r + beta p, so z is not stored, and takes the previous step of y; the update needs r and q only.  Per
// node of 8 bytes a value: r, p, y read and p, q, y written, then r, q read and r written.
// Measured on a B200, operator and update of an iteration: 128x256x128 elements 30 and 14 us, a 96x192x96 box with a
// third solid 18 and 15 us; with the 64 entries, synchronous plane loads and z, p stored by the update 46 and 26,
// and 38 and 21 us.  The operator is bound by its two barriers a plane (0.6 of HBM at 128x256x128).
#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <vector>

#include "topx_kernels.cuh"
#include "topx_opt.cuh"
#include "topx_tma.cuh"

namespace topx {

namespace {

constexpr int FK_NT = 256;
constexpr int FK_CTAS = 4;  // CTAs of an SM
constexpr int FK_PAD = 64;  // reach of a neighbour index (PY + 1)
constexpr int FK_ROW = FK_NT + FK_PAD;

template <typename T>
struct FilterSmem {
  T su[2][FK_ROW];    // a plane's values, and those of the plane below, read by their own threads
  T cor[3][FK_ROW];   // face values for the corners (y+1, x), (y, x+1), (y+1, x+1)
  uint64_t bar[2];
};
struct FilterMaps {
  CUtensorMap r, p, y;
};

// One element layer between two transformed faces, as ku_layer: [ss, sd, ds, dd]; G enters as the layer below's part of
// the lower plane and leaves complete, Bn is this layer's part of the upper plane.
template <typename T>
__device__ __forceinline__ void filter_layer(const FilterKe<T>& K, bool solid, const T (&W0)[4], const T (&W1)[4],
                                             T (&G)[4], T (&Bn)[4]) {
  const T h0 = solid ? K.h[0] : T(0), h1 = solid ? K.h[1] : T(0), h2 = solid ? K.h[2] : T(0), h3 = solid ? K.h[3] : T(0);
  const T hs[4] = {h0, h1, h1, h2}, hd[4] = {h1, h2, h2, h3};
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const T fs = hs[m] * (W0[m] + W1[m]), fd = hd[m] * (W1[m] - W0[m]);
    G[m] += fs - fd;
    Bn[m] = fs + fd;
  }
}

template <typename T>
__global__ void __launch_bounds__(FK_NT, FK_CTAS)
    k_filter_ku(const __grid_constant__ FilterArgs<T> a, const __grid_constant__ FilterMaps maps, const int box,
                const int ybox, const unsigned bytes) {
  constexpr int HB = 16 / int(sizeof(T));  // rows before the tile: a copy starts on a 16-byte boundary
  extern __shared__ __align__(128) unsigned char fk_smem[];  // two planes' boxes of r, p, y, then the rest
  const int len = 2 * box + ybox;  // of a stage, in values
  T* const stages = reinterpret_cast<T*>(fk_smem);
  FilterSmem<T>& sm = *reinterpret_cast<FilterSmem<T>*>(stages + 2 * len);
  const int t = threadIdx.x, PY = a.sh.PY;
  const int nny = a.g.ny + 1, nnx = a.g.nx + 1, nnz = a.g.nz + 1;
  int tyi = blockIdx.x, txi = blockIdx.y, tzi = blockIdx.z;
  if (a.active) {
    const uint32_t e = a.active[blockIdx.x];
    tyi = int(e & 1023u);
    txi = int((e >> 10) & 1023u);
    tzi = int(e >> 20);
  }
  int zc0 = tzi * a.sh.zc, zend = min(zc0 + a.sh.zc, nnz);
  if (a.active && a.zr) {
    const uint32_t r = a.zr[blockIdx.x];
    zc0 = int(r & 0xffffu);
    zend = int(r >> 16);
  }
  const int lx = t / PY, ly = t - lx * PY;
  const int y0 = tyi * a.sh.TY, x0 = txi * a.sh.TX;
  const int gy = y0 - 1 + ly, gx = x0 - 1 + lx;
  const bool in_tile = lx < a.sh.PX;
  const bool inb = in_tile && gy >= 0 && gy < nny && gx >= 0 && gx < nnx;
  const bool own = inb && ly >= 1 && ly <= a.sh.TY && lx >= 1 && lx <= a.sh.TX;
  const int o = in_tile ? lx * (a.sh.TY + 2 * HB) + ly + HB - 1 : 0, oy = own ? (lx - 1) * a.sh.TY + ly - 1 : 0;
  const int64_t n0 = inb ? gy + int64_t(nny) * gx : 0, np = int64_t(nny) * nnx;
  bool ok = true;  // no wait of this thread gave up
  auto issue = [&](int zp, int s) {
    if (t == 0 && ok) {
      T* d = stages + s * len;
      mbar_expect(&sm.bar[s], bytes);
      tma_load(d, &maps.r, y0 - HB, x0 - 1, zp, &sm.bar[s]);
      tma_load(d + box, &maps.p, y0 - HB, x0 - 1, zp, &sm.bar[s]);
      tma_load(d + 2 * box, &maps.y, y0, x0, zp, &sm.bar[s]);
    }
  };
  if (t == 0) {
    tma_prefetch(&maps.r);
    tma_prefetch(&maps.p);
    tma_prefetch(&maps.y);
    mbar_init(&sm.bar[0]);
    mbar_init(&sm.bar[1]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  issue(zc0 - 1, 0);
  issue(zc0, 1);
  auto flags_at = [&](int zp) -> unsigned {
    return inb && zp >= 0 && zp < nnz ? unsigned(a.flags[n0 + np * zp]) : 0u;
  };
  unsigned f = flags_at(zc0 - 1);
  const int its = a.sc->its;  // steps done: none (p = z), one (y starts), more
  const T beta = T(a.sc->beta), lam = T(a.sc->lam);
  if (a.sc->done) {  // the same for the whole launch
    ok = plane_wait(sm.bar, 0, 1, t == 0) && plane_wait(sm.bar, 1, 1, t == 0);
    if (!ok) report_copy_wait(a.err);
    return;
  }
  double dot = 0.0;
  bool solid = false;  // of the layer below plane zp
  T W0[4], Bq[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) W0[m] = Bq[m] = T(0);
#pragma unroll 1
  for (int zp = zc0 - 1; zp <= zend; ++zp) {
    const int s = (zp - zc0 + 1) & 1;
    const T* st = stages + s * len;
    const int64_t n = n0 + np * zp;
    if (ok) ok = plane_wait(sm.bar, zp - zc0 + 1, zend - zc0 + 1, t == 0);
    T v = a.ke.dp[f & 15u] * st[o];  // D r; 0 off the domain
    const T po = st[box + o];
    if (its > 0) v = v + beta * po;
    if (own && zp >= zc0 && zp < zend) {
      a.pout[n] = v;
      if (its > 0) a.y[n] = its > 1 ? st[2 * box + oy] + lam * po : lam * po;
    }
    sm.su[s][t] = v;
    const unsigned fn = flags_at(zp + 1);
    __syncthreads();
    if (zp + 2 <= zend) issue(zp + 2, s);  // every thread has read the stage
    const T* u = sm.su[s] + t;
    const T u10 = u[1], u01 = u[PY], u11 = u[PY + 1];
    const T s0 = v + u10, d0 = v - u10, s1 = u01 + u11, d1 = u01 - u11;
    const T W1[4] = {s0 + s1, s1 - s0, d0 + d1, d1 - d0};
    T Bn[4] = {T(0), T(0), T(0), T(0)};
    if (zp >= zc0) {
      filter_layer(a.ke, solid, W0, W1, Bq, Bn);  // Bq: plane zp - 1 complete, in face modes
      if (zp > zc0) {
        const T lo_s = Bq[0] + Bq[2], hi_s = Bq[0] - Bq[2], lo_d = Bq[1] + Bq[3], hi_d = Bq[1] - Bq[3];
        sm.cor[0][FK_PAD + t] = hi_s - hi_d;
        sm.cor[1][FK_PAD + t] = lo_s + lo_d;
        sm.cor[2][FK_PAD + t] = hi_s + hi_d;
        __syncthreads();
        if (own) {
          const T qv = (((lo_s - lo_d) + sm.cor[0][FK_PAD + t - 1]) + sm.cor[1][FK_PAD + t - PY]) +
                       sm.cor[2][FK_PAD + t - PY - 1];
          a.q[n - np] = qv;
          dot = fma(double(sm.su[s ^ 1][t]), double(qv), dot);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      W0[m] = W1[m];
      Bq[m] = Bn[m];
    }
    solid = (f & 128u) != 0u;
    f = fn;
  }
  if (!ok) report_copy_wait(a.err);
  double r[1] = {dot}, tot[1];
  if (reduce_publish<1>(r, a.rs, tot) && t == 0) a.sc->pq = tot[0];
}

// element -> node: sum over the node's hexes (local-node order) of src_e*(1/8)  (TOP3D_XL.m:880-886)
template <typename T>
__global__ void k_filter_start(const __grid_constant__ FilterArgs<T> a, const T* __restrict__ srcE, FastDiv dny, FastDiv dnx) {
  pdl_wait();
  const uint32_t N = uint32_t(a.g.nnodes());  // < 2^32 (checked at launch)
  const int nny = a.g.ny + 1, nnx = a.g.nx + 1;
  double bb = 0.0, rz = 0.0;
  for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    if (!chunk_active(a.act, n)) continue;  // no solid element around these nodes: zero
    const uint32_t q = dny.div(n), qz = dnx.div(q);
    const int gy = int(n - q * uint32_t(nny)), gx = int(q - qz * uint32_t(nnx)), gz = int(qz);
    T s = T(0);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int ey = gy - hex_ly(c), ex = gx - hex_lx(c), ez = gz - hex_lz(c);
      if (ey < 0 || ex < 0 || ez < 0) continue;
      s = s + srcE[ey + int64_t(nny) * (ex + int64_t(nnx) * ez)] * T(0.125);
    }
    a.r[n] = s;
    bb += double(s) * double(s);
    rz += double(a.ke.dp[a.flags[n] & 15u] * s) * double(s);
  }
  double v[2] = {bb, rz}, tot[2];
  if (reduce_publish<2>(v, a.rs, tot) && threadIdx.x == 0) {
    a.sc->normB = sqrt(tot[0]);
    a.sc->x1 = tot[1];
    a.sc->tol = a.tol;
    a.sc->maxIT = a.maxIT;
    a.sc->its = 0;
    a.sc->done = 0;
    a.sc->first = 1;
    a.sc->beta = 0.0;
  }
}

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct Vec4<double> {
  static __device__ __forceinline__ void load(const double* p, double (&v)[4]) {
    const double2 x = *reinterpret_cast<const double2*>(p), y = *reinterpret_cast<const double2*>(p + 2);
    v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
  }
  static __device__ __forceinline__ void store(double* p, const double (&v)[4]) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
  }
};

// four nodes a thread (rows hold a multiple of four)
template <typename T>
__global__ void __launch_bounds__(256) k_filter_update(const __grid_constant__ FilterArgs<T> a) {
  pdl_wait();
  if (a.sc->done) return;
  const double lam = a.sc->x1 / a.sc->pq;
  const T lamT = T(lam);
  const int64_t N4 = a.g.nnodes() / 4;
  double rr = 0.0, rz = 0.0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < N4; i += int64_t(gridDim.x) * blockDim.x) {
    if (!chunk_active(a.act, 4 * i)) continue;  // zero there and stays so
    T r[4], q[4];
    Vec4<T>::load(a.r + 4 * i, r);
    Vec4<T>::load(a.q + 4 * i, q);
    const unsigned f = *reinterpret_cast<const unsigned*>(a.flags + 4 * i);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      r[k] = r[k] - lamT * q[k];
      rr = fma(double(r[k]), double(r[k]), rr);
      rz = fma(double(a.ke.dp[f >> (8 * k) & 15u] * r[k]), double(r[k]), rz);
    }
    Vec4<T>::store(a.r + 4 * i, r);
  }
  double v[2] = {rr, rz}, tot[2];
  if (reduce_publish<2>(v, a.rs, tot) && threadIdx.x == 0) {
    a.sc->rr = tot[0];
    a.sc->resnorm = sqrt(tot[0]) / a.sc->normB;
    a.sc->its += 1;
    a.sc->first = 0;
    a.sc->lam = lam;
    if (a.sc->resnorm < a.sc->tol) {
      a.sc->done = 1;
    } else if (a.sc->its >= a.sc->maxIT) {
      a.sc->done = 2;
    } else {
      a.sc->beta = tot[1] / a.sc->x1;
      a.sc->x1 = tot[1];
    }
  }
}

// node -> element mean (TOP3D_XL.m:894-901) of the solution, its last step included; compact element order
template <typename T>
__global__ void k_filter_n2e(const __grid_constant__ FilterArgs<T> a, const int32_t* __restrict__ emb0, int64_t Ne,
                             double* __restrict__ out) {
  pdl_wait();
  const int64_t nny = a.g.ny + 1, nnx = a.g.nx + 1;
  const int its = a.sc->its;
  const T lam = its > 0 ? T(a.sc->lam) : T(0);
  const T* p = its & 1 ? a.pout : a.pin;  // step k writes pout (k even) or pin (k odd)
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < Ne; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t id = emb0[e];  // the index of its lowest node
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int64_t n = id + hex_ly(c) + nny * (hex_lx(c) + nnx * hex_lz(c));
      T v = T(0);
      if (its > 0) v = its > 1 ? a.y[n] + lam * p[n] : lam * p[n];
      s += double(v);
    }
    out[e] = s * (1.0 / 8);
  }
}

inline unsigned blocks(int64_t n) { return unsigned(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16))); }

template <typename T>
void filter_attr() {
  TOPX_CUDA_OK(cudaFuncSetAttribute(k_filter_ku<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024 / FK_CTAS));
}

}  // namespace

void prepare_filter_kernels() {
  filter_attr<double>();
  filter_attr<float>();
}

template <typename T>
FilterKe<T> filter_ke(const double* KF64) {
  FilterKe<T> k;
  for (int d = 0; d < 4; ++d) {  // differences along the first d of y, x, z
    double s = 0.0;
    for (int a = 0; a < 8; ++a)
      for (int b = 0; b < 8; ++b) {
        double w = KF64[8 * a + b];
        if (d > 0 && hex_ly(a) != hex_ly(b)) w = -w;
        if (d > 1 && hex_lx(a) != hex_lx(b)) w = -w;
        if (d > 2 && hex_lz(a) != hex_lz(b)) w = -w;
        s += w;
      }
    k.h[d] = T(s / 64.0);
  }
  double s = 0.0;
  for (int c = 0; c <= 8; ++c) {
    k.dp[c] = c ? T(1.0 / s) : T(0);
    s += KF64[0];
  }
  return k;
}
template FilterKe<double> filter_ke<double>(const double*);
template FilterKe<float> filter_ke<float>(const double*);

// As ku_shape: planes formed and written, the warps of a plane, and the waves of FK_CTAS CTAs per SM.
FilterShape filter_shape(Grid g, int rows, int bytes) {
  const int nnx = g.nnx(), nnz = g.nnz(), HB = 16 / bytes;
  const double slots = double(FK_CTAS) * num_sms();
  FilterShape best{};
  double bestCost = -1;
  for (int nty = 1; nty <= rows; ++nty) {
    const int TY = ((rows + nty - 1) / nty + HB - 1) / HB * HB, PY = TY + 2;
    if (PY > FK_PAD - 2 || (rows + TY - 1) / TY != nty || PY * 3 > FK_NT) continue;
    if (TY < 6 && rows >= 6) break;
    const int TXmax = std::min(FK_NT / PY - 2, nnx);
    const int ntx = (nnx + TXmax - 1) / TXmax, TX = (nnx + ntx - 1) / ntx, PX = TX + 2;
    const double plane_cost = (PY * PX + 31) / 32 * (1.0 + 3.0 / PY) / 8.0 + 0.4;
    for (int zc = 1; zc <= 64 && zc <= nnz + 1; ++zc) {
      const double ctas = double(nty) * ntx * ((nnz + zc - 1) / zc);
      const double waves = ctas / slots, w = waves <= 1.0 ? 1.0 : 0.5 * (waves + std::ceil(waves));
      const double cost = (w + 0.3) * (zc + 4) * (1.0 + 0.003 * zc) * plane_cost;
      if (bestCost < 0 || cost < bestCost) {
        bestCost = cost;
        best = FilterShape{PY, PX, TY, TX, zc, dim3(unsigned(nty), unsigned(ntx), unsigned((nnz + zc - 1) / zc))};
      }
    }
  }
  if (bestCost < 0) throw std::runtime_error("no filter tile for this grid");
  return best;
}

std::vector<uint32_t> filter_active_tiles(Grid g, int rows, const FilterShape& f, const std::vector<uint8_t>& present,
                                          std::vector<uint32_t>& zranges) {
  KuShape k{f.PY, f.PX, f.TY, f.TX, f.zc, f.grid};
  return ku_active_tiles(g, rows, k, present, &zranges);
}

template <typename T>
void launch_filter_start(cudaStream_t st, const FilterArgs<T>& a, const T* srcE) {
  if (a.g.nnodes() >= (int64_t(1) << 32)) throw std::runtime_error("grid too large for 32-bit node indices");
  const FastDiv dny{uint32_t(a.g.nny())}, dnx{uint32_t(a.g.nnx())};
  launch_pdl(st, k_filter_start<T>, blocks(a.g.nnodes()), 256, 0, a, srcE, dny, dnx);
}
template <typename T>
void launch_filter_ku(cudaStream_t st, const FilterArgs<T>& a) {
  const dim3 grd = a.active ? dim3(unsigned(a.ntiles)) : a.sh.grid;
  if (grd.x == 0) return;
  constexpr int HB = 16 / int(sizeof(T)), line = 128 / int(sizeof(T));
  auto up = [](int n) { return (n + line - 1) / line * line; };  // boxes start on 128-byte boundaries
  const int PB = a.sh.TY + 2 * HB, full = PB * a.sh.PX, own = a.sh.TY * a.sh.TX;
  FilterMaps m;
  m.r = field_map(a.r, a.g, 1, PB, a.sh.PX);
  m.p = field_map(a.pin, a.g, 1, PB, a.sh.PX);
  m.y = field_map(a.y, a.g, 1, a.sh.TY, a.sh.TX);
  const size_t smem = sizeof(T) * 2 * size_t(2 * up(full) + up(own)) + sizeof(FilterSmem<T>);
  launch_pdl(st, k_filter_ku<T>, grd, FK_NT, smem, a, m, up(full), up(own), unsigned(sizeof(T) * (2 * full + own)));
}
template <typename T>
void launch_filter_update(cudaStream_t st, const FilterArgs<T>& a) {
  launch_pdl(st, k_filter_update<T>, blocks(a.g.nnodes() / 4), 256, 0, a);
}
template <typename T>
void launch_filter_n2e(cudaStream_t st, const FilterArgs<T>& a, const int32_t* eleMapBack0, int64_t Ne, double* out) {
  launch_pdl(st, k_filter_n2e<T>, blocks(Ne), 256, 0, a, eleMapBack0, Ne, out);
}
#define TOPX_INST(T)                                                                                        \
  template void launch_filter_start<T>(cudaStream_t, const FilterArgs<T>&, const T*);                       \
  template void launch_filter_ku<T>(cudaStream_t, const FilterArgs<T>&);                                    \
  template void launch_filter_update<T>(cudaStream_t, const FilterArgs<T>&);                                \
  template void launch_filter_n2e<T>(cudaStream_t, const FilterArgs<T>&, const int32_t*, int64_t, double*);
TOPX_INST(double)
TOPX_INST(float)

}  // namespace topx
