// Level-1 stiffness operator of the TOP3D_XL B200 path, matrix-free (Solving_KbyU_MatrixFree,
// TOP3D_XL.m:684-725), and the PCG step that is fused with it.
//
// The reference's per-element BC matrices (uniqueKesFree_/uniqueKesFixed_) reduce exactly to
//     y = m .* K_E (m .* u) + (1-m) .* cfix .* u
// with m the free-DOF mask and cfix(node) = sum over its hexes of 1/nAdj.
//
// Sums and differences instead of Ke.  A cube is symmetric under its three reflections, so in the basis
// of sums and differences of the eight corner values along y, x and z (a Walsh transform per
// component) its 24x24 stiffness matrix falls into blocks of at most 3x3 with eight different values
// (KuModes).  An element takes 41 operations there instead of 576, and the transforms are separable:
// the y and x stages of a face (12 values) serve the element layers above and below it.  Per node the
// operator takes about 160 FP64 operations, 600 with Ke itself.  Differences of neighbouring values
// come first, so a smooth field cancels exactly at the start instead of at the end of long sums.
//
// Tiles.  A CTA of 256 threads marches a z-chunk of a PY x PX tile of node columns (y fastest), one
// thread per column; the outer ring is halo.  A thread copies the values of its own node two
// planes ahead, asynchronously, into slots that only it reads, forms the operator's input
// there (masked u, or the PCG direction), and exchanges through shared memory twice per plane: its
// value with the other corners of its face, and its face's forces with the nodes at those corners.  The
// transformed face of the plane below and the forces from the layer below stay in registers.  A
// node takes no separate launch for the last row of a grid.  No atomics: the result is deterministic.
//
// Measured on a B200, one PCG-mode launch (128x256x128, 64x128x64 and 50x100x50 elements): 185, 36
// and 27 us, with Ke's 576 entries in a 32 x 8 tile and a launch for the last row 280, 54 and 32 us.
// Bound by the shared-memory and load/store pipe (71 % of its wavefronts; the FP64 pipe 31 %,
// DRAM 37 %): 8-byte accesses, since rows of an odd number of nodes start at odd addresses.  What was
// slower there: three planes in flight (257 us: the slots take the L1 cache that serves the halo),
// two planes per barrier (275), loads into registers one plane ahead (386), CTAs of 128 threads (203)
// or 512 (190), three CTAs per SM with spills (319).
#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <type_traits>
#include <vector>

#include "topx_ke_classes.h"
#include "topx_kernels.cuh"

namespace topx {

namespace {

constexpr int KU_NT = 256;  // threads of a CTA
constexpr int KU_CTAS = 2;  // CTAs of an SM
constexpr int KU_PAD = 64;  // reach of a neighbour index (PY + 1)
constexpr int KU_ROW = KU_NT + KU_PAD;

template <int BYTES>
__device__ __forceinline__ void cp_async_el(void* smem, const void* gmem, bool pred) {
  static_assert(BYTES == 4 || BYTES == 8, "element copy size");
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int n = pred ? BYTES : 0;  // 0: fill with zeros, read nothing
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// an array element at a 32-bit byte offset from a uniform base
template <typename T>
__device__ __forceinline__ T* at(T* base, uint32_t bytes) {
  using C = typename std::conditional<std::is_const<T>::value, const char, char>::type;
  return reinterpret_cast<T*>(reinterpret_cast<C*>(base) + bytes);
}

template <int MODE>
struct KuSmem {
  static constexpr int NF = MODE == KU_PLAIN ? 4 : 10;
  double stage[2][NF][KU_NT];  // of two planes: a[3], E, then (PCG) p_in[3], y[3]
  double su[2][3][KU_ROW];     // a plane's masked values, and those of the plane below, read by their own threads
  double cor[3][3][KU_ROW];    // face forces for the corners (y+1, x), (y, x+1), (y+1, x+1)
};

// One element layer between two transformed faces: W0 (below) and W1 (above), faces [component x, y, z]
// [ss, sd, ds, dd] with s/d the sum or difference along (y, x).  G enters as the layer below's part of the lower
// plane's forces and leaves complete; Bn is this layer's part of the upper plane's.
__device__ __forceinline__ void ku_layer(const KuModes& K, double E, double (&W0)[3][4], const double (&W1)[3][4],
                                         double (&G)[3][4], double (&Bn)[3][4]) {
  enum { SS = 0, SD = 1, DS = 2, DD = 3 };
  auto sum = [&](int c, int m) { return W0[c][m] + W1[c][m]; };
  auto dif = [&](int c, int m) { return W1[c][m] - W0[c][m]; };
  // F of a mode that is a sum along z adds to both planes, of a difference to the upper and from the lower
  auto first_s = [&](int c, int m, double f) {
    G[c][m] += f;
    Bn[c][m] = f;
  };
  auto then_d = [&](int c, int m, double f) {
    G[c][m] -= f;
    Bn[c][m] += f;
  };
  auto only_d = [&](int c, int m, double f) {
    G[c][m] -= f;
    Bn[c][m] = f;
  };
  {  // normal strains: x (sd, s), y (ds, s), z (ss, d)
    const double ex = sum(0, SD), ey = sum(1, DS), ez = dif(2, SS);
    const double eb = E * K.b * (ex + ey + ez), ea = E * K.a_b;
    first_s(0, SD, fma(ea, ex, eb));
    first_s(1, DS, fma(ea, ey, eb));
    only_d(2, SS, fma(ea, ez, eb));
  }
  {  // shear strains xy, xz, yz
    const double eg = E * K.g;
    const double fxy = eg * (sum(0, DS) + sum(1, SD));
    first_s(0, DS, fxy);
    first_s(1, SD, fxy);
    const double fxz = eg * (dif(0, SS) + sum(2, SD));
    only_d(0, SS, fxz);
    first_s(2, SD, fxz);
    const double fyz = eg * (dif(1, SS) + sum(2, DS));
    only_d(1, SS, fyz);
    first_s(2, DS, fyz);
  }
  const double ep = E * K.p, eq = E * K.q;
  {  // bending about z: x (sd, d) with y (ds, d)
    const double u = dif(0, SD), v = dif(1, DS);
    then_d(0, SD, fma(ep, u, eq * v));
    then_d(1, DS, fma(ep, v, eq * u));
  }
  {  // x (dd, s) with z (ds, d), y (dd, s) with z (sd, d)
    const double u = sum(0, DD), v = dif(2, DS);
    first_s(0, DD, fma(ep, u, eq * v));
    then_d(2, DS, fma(ep, v, eq * u));
    const double w = sum(1, DD), t = dif(2, SD);
    first_s(1, DD, fma(ep, w, eq * t));
    then_d(2, SD, fma(ep, t, eq * w));
  }
  {  // torsion: x (ds, d), y (sd, d), z (dd, s)
    const double u = dif(0, DS), v = dif(1, SD), w = sum(2, DD);
    const double es = E * K.s * (u + v + w), er = E * K.r_s;
    then_d(0, DS, fma(er, u, es));
    then_d(1, SD, fma(er, v, es));
    first_s(2, DD, fma(er, w, es));
  }
  const double eh = E * K.h;  // the triple differences
  then_d(0, DD, eh * dif(0, DD));
  then_d(1, DD, eh * dif(1, DD));
  then_d(2, DD, eh * dif(2, DD));
}

// MODE KU_PLAIN: out = K in.  KU_P_UPDATE: p = z + beta p_in (p = z on the first step) for a given z.
// It stores p, reduces p'q into sc->pq and applies the previous iteration's solution step y += lam p_in.
template <int MODE>
__global__ void __launch_bounds__(KU_NT, KU_CTAS) k_ku(const __grid_constant__ KuArgs a) {
  constexpr bool PCG = MODE != KU_PLAIN;
  extern __shared__ __align__(16) unsigned char ku_dyn_smem[];
  KuSmem<MODE>& sm = *reinterpret_cast<KuSmem<MODE>*>(ku_dyn_smem);
  const int t = threadIdx.x, PY = a.sh.PY;
  const int nny = a.g.ny + 1, nnx = a.g.nx + 1, nnz = a.g.nz + 1;
  const int64_t S = a.g.stride;
  int tyi = blockIdx.x, txi = blockIdx.y, tzi = blockIdx.z;
  if (a.active) {
    const uint32_t e = a.active[blockIdx.x];
    tyi = int(e & 1023u);
    txi = int((e >> 10) & 1023u);
    tzi = int(e >> 20);
  }
  int zc0 = tzi * a.sh.zc, zend = min(zc0 + a.sh.zc, nnz);
  if (a.active && a.zr) {  // only the planes of the chunk that hold a present node
    const uint32_t r = a.zr[blockIdx.x];
    zc0 = int(r & 0xffffu);
    zend = int(r >> 16);
  }
  const int lx = t / PY, ly = t - lx * PY;
  const int y0 = tyi * a.sh.TY, x0 = txi * a.sh.TX;  // first own node
  const int gy = y0 - 1 + ly, gx = x0 - 1 + lx;      // this thread's node, and the lower corner of its face
  const bool in_tile = lx < a.sh.PX;
  const bool inb = in_tile && gy >= 0 && gy < nny && gx >= 0 && gx < nnx;
  const bool einb = in_tile && gy >= 0 && gy < a.g.ny && gx >= 0 && gx < a.g.nx;
  const bool own = inb && ly >= 1 && ly <= a.sh.TY && lx >= 1 && lx <= a.sh.TX;
  // byte offsets of the node on plane 0 and of a plane (an array has less than 4 GB: checked at launch)
  const uint32_t n0 = inb ? 8u * uint32_t(gy + nny * gx) : 0u, np = 8u * uint32_t(nny) * uint32_t(nnx);
  const uint32_t e0 = einb ? 8u * uint32_t(gy + a.g.ny * gx) : 0u, ep = 8u * uint32_t(a.g.ny) * uint32_t(a.g.nx);
  const double* const araw = MODE == KU_P_UPDATE ? a.z : a.in;

  auto issue = [&](int zp, int s) {
    const bool ok = inb && zp >= 0 && zp < nnz && zp <= zend;
    const uint32_t n = ok ? n0 + np * uint32_t(zp) : 0u;
    const bool yok = PCG && own && zp >= zc0 && zp < zend;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      cp_async_el<8>(&sm.stage[s][c][t], at(araw + c * S, n), ok);
      if (PCG) {
        cp_async_el<8>(&sm.stage[s][4 + c][t], at(a.pin + c * S, n), ok);
        cp_async_el<8>(&sm.stage[s][7 + c][t], at(a.yacc + c * S, yok ? n : 0u), yok);
      }
    }
    const bool eok = einb && zp >= zc0 && zp >= 1 && zp <= a.g.nz && zp <= zend;  // the layer between zp - 1 and zp
    cp_async_el<8>(&sm.stage[s][3][t], at(a.E, eok ? e0 + ep * uint32_t(zp - 1) : 0u), eok);
  };
  issue(zc0 - 1, 0);
  cp_async_commit();
  issue(zc0, 1);
  cp_async_commit();
  auto flags_at = [&](int zp) -> unsigned {
    return inb && zp >= 0 && zp < nnz && zp <= zend ? unsigned(a.flags[(n0 + np * uint32_t(zp)) / 8u]) : 0u;
  };
  unsigned f = flags_at(zc0 - 1), fo = 0;  // of the plane, and of the one below
  const bool first = PCG && a.sc->first;
  const double beta = PCG ? a.sc->beta : 0.0, lam = PCG ? a.sc->lam : 0.0;
  if (PCG && a.sc->done) {
    cp_async_wait_all();
    return;
  }
  double dot = 0.0;
  // Plane zp in slot s, and the element layer below it (between the faces Wp and W): plane zp - 1 is then
  // complete.  G holds its forces in face modes, Bn takes the layer's part of plane zp's.
  auto step = [&](int zp, int s, double (&Wp)[3][4], double (&W)[3][4], double (&G)[3][4], double (&Bn)[3][4]) {
    const uint32_t n = n0 + np * uint32_t(zp);
    const bool mine = own && zp >= zc0 && zp < zend;
    cp_async_wait_all_but_one();
    const double E = sm.stage[s][3][t];
    double v[3], y[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v[c] = sm.stage[s][c][t];
      if (PCG) {
        const double po = sm.stage[s][4 + c][t];
        if (!first) v[c] = fma(beta, po, v[c]);
        if (mine) {
          *at(a.pout + c * S, n) = v[c];
          if (!first) *at(a.yacc + c * S, n) = fma(lam, po, sm.stage[s][7 + c][t]);
        }
      }
      if (f & (1u << c)) v[c] = 0.0;
      sm.su[s][c][t] = v[c];
    }
    if (zp + 2 <= zend) issue(zp + 2, s);
    cp_async_commit();
    const unsigned fn = flags_at(zp + 1);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double* u = sm.su[s][c] + t;
      const double u00 = v[c], u10 = u[1], u01 = u[PY], u11 = u[PY + 1];
      const double s0 = u00 + u10, d0 = u00 - u10, s1 = u01 + u11, d1 = u01 - u11;
      W[c][0] = s0 + s1;
      W[c][1] = s1 - s0;
      W[c][2] = d0 + d1;
      W[c][3] = d1 - d0;
    }
    if (zp >= zc0) {
      ku_layer(a.K, E, Wp, W, G, Bn);
      if (zp > zc0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double lo_s = G[c][0] + G[c][2], hi_s = G[c][0] - G[c][2];
          const double lo_d = G[c][1] + G[c][3], hi_d = G[c][1] - G[c][3];
          y[c] = lo_s - lo_d;
          sm.cor[0][c][KU_PAD + t] = hi_s - hi_d;
          sm.cor[1][c][KU_PAD + t] = lo_s + lo_d;
          sm.cor[2][c][KU_PAD + t] = hi_s + hi_d;
        }
        __syncthreads();
        if (own) {
          const uint32_t m = n - np;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            double yv = ((y[c] + sm.cor[0][c][KU_PAD + t - 1]) + sm.cor[1][c][KU_PAD + t - PY]) +
                        sm.cor[2][c][KU_PAD + t - PY - 1];
            double p = sm.su[s ^ 1][c][t];
            if (fo & (1u << c)) {  // a fixed DOF: its own value, unmasked
              p = PCG ? *at(a.pout + c * S, m) : *at(a.in + c * S, m);
              yv = *at(a.cfix, m) * p;
            }
            *at(a.out + c * S, m) = yv;
            if (PCG) dot = fma(p, yv, dot);
          }
        }
      }
    }
    fo = f;
    f = fn;
  };
  double W0[3][4], Bq[3][4];  // the transformed face of the plane below, and its forces from the layer below
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int m = 0; m < 4; ++m) W0[c][m] = Bq[c][m] = 0.0;
  double W1[3][4], Bn[3][4];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int m = 0; m < 4; ++m) Bn[c][m] = 0.0;
#pragma unroll 1
  for (int zp = zc0 - 1; zp <= zend; ++zp) {
    step(zp, (zp - zc0 + 1) & 1, W0, W1, Bq, Bn);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        W0[c][m] = W1[c][m];
        Bq[c][m] = Bn[c][m];
      }
  }
  cp_async_wait_all();
  if (PCG) {
    double r[1] = {dot}, tot[1];
    if (reduce_publish<1>(r, a.rs, tot) && t == 0) a.sc->pq = tot[0];
  }
}

template <int MODE>
void ku_smem_attr() {
  TOPX_CUDA_OK(cudaFuncSetAttribute(k_ku<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int(sizeof(KuSmem<MODE>))));
}

int ku_num_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 148;
  return n > 0 ? n : 148;
}

}  // namespace

void prepare_ku_kernels() {
  ku_smem_attr<KU_PLAIN>();
  ku_smem_attr<KU_P_UPDATE>();
}

// Sign of corner a in mode (sy, sx, sz); the y difference runs from the upper to the lower row, along the y axis.
static double mode_sign(int a, int sy, int sx, int sz) {
  double v = 1.0;
  if (sy) v *= hex_ly(a) ? -1.0 : 1.0;
  if (sx) v *= hex_lx(a) ? 1.0 : -1.0;
  if (sz) v *= hex_lz(a) ? 1.0 : -1.0;
  return v;
}
// Entry of Kh between component ci in mode (sy, sx, sz) and component cj in mode (ty, tx, tz).
static long double mode_entry(const double* Ke, int ci, int sy, int sx, int sz, int cj, int ty, int tx, int tz) {
  long double s = 0.0L;
  for (int a = 0; a < 8; ++a)
    for (int b = 0; b < 8; ++b)
      s += (long double)(mode_sign(a, sy, sx, sz) * mode_sign(b, ty, tx, tz)) * Ke[(3 * a + ci) * 24 + 3 * b + cj];
  return s / 64.0L;
}

// The eight values of Ke in the basis of sums and differences: Kh = H Ke H^T / 64.  Checks that Ke has the
// cube's value classes (which is what makes every other entry of Kh vanish).
KuModes ku_modes(const double* Ke576) {
  double first[kKeClasses];
  bool seen[kKeClasses] = {};
  for (int i = 0; i < 576; ++i) {
    const int code = ke_class_code(i), c = (code > 0 ? code : -code) - 1;
    const double v = code > 0 ? Ke576[i] : -Ke576[i];
    if (!seen[c]) {
      first[c] = v;
      seen[c] = true;
    } else if (!(std::fabs(v - first[c]) <= 1e-13 * std::fabs(first[c]))) {
      throw std::runtime_error("element stiffness does not have the hex8 value classes");
    }
  }
  const long double a = mode_entry(Ke576, 0, 0, 1, 0, 0, 0, 1, 0), b = mode_entry(Ke576, 0, 0, 1, 0, 1, 1, 0, 0), g = mode_entry(Ke576, 0, 1, 0, 0, 1, 0, 1, 0),
                    p = mode_entry(Ke576, 0, 0, 1, 1, 0, 0, 1, 1), q = mode_entry(Ke576, 0, 0, 1, 1, 1, 1, 0, 1),
                    r = mode_entry(Ke576, 0, 1, 0, 1, 0, 1, 0, 1), s = mode_entry(Ke576, 0, 1, 0, 1, 1, 0, 1, 1),
                    h = mode_entry(Ke576, 0, 1, 1, 1, 0, 1, 1, 1);
  KuModes K;
  K.a_b = double(a - b);
  K.b = double(b);
  K.g = double(g);
  K.p = double(p);
  K.q = double(q);
  K.r_s = double(r - s);
  K.s = double(s);
  K.h = double(h);
  return K;
}

// Tile and z-chunk of the launch.  A CTA's time goes with its planes (zc + 2 formed for zc written, and
// about two planes' worth of start and end), each plane's with its warps and with the
// 32-byte sectors its unaligned rows of PY nodes touch.  Every tile height whose tiles come out
// even, with the widest tile that then fits the CTA, and every chunk length are compared; past six
// waves the last one's share is small.  In a sweep of tiles and chunks at the three sizes above no
// other choice was more than 8 % faster than the one taken.
KuShape ku_shape(Grid g) {
  const int nny = g.nny(), nnx = g.nnx(), nnz = g.nnz();
  if (g.nnodes() >= (int64_t(1) << 29)) throw std::runtime_error("grid too large for 32-bit byte offsets");
  const double slots = double(KU_CTAS) * ku_num_sms();
  KuShape best{};
  double bestCost = -1;
  for (int nty = 1; nty <= nny; ++nty) {
    const int TY = (nny + nty - 1) / nty, PY = TY + 2;
    if (PY > KU_PAD - 2 || (nny + TY - 1) / TY != nty) continue;
    if (PY * 3 > KU_NT) continue;
    if (TY < 6 && nny >= 6) break;
    const int TXmax = std::min(KU_NT / PY - 2, nnx);
    const int ntx = (nnx + TXmax - 1) / TXmax, TX = (nnx + ntx - 1) / ntx, PX = TX + 2;
    const double plane_cost = (PY * PX + 31) / 32 * (1.0 + 3.0 / PY) / 8.0 + 0.4;
    for (int zc = 1; zc <= 64 && zc <= nnz + 1; ++zc) {
      const double ctas = double(nty) * ntx * ((nnz + zc - 1) / zc);
      const double waves = ctas / slots, w = waves > 6 ? waves + 0.5 : std::ceil(waves);
      const double cost = w * (zc + 4) * plane_cost;
      if (bestCost < 0 || cost < bestCost) {
        bestCost = cost;
        best = KuShape{PY, PX, TY, TX, zc, dim3(unsigned(nty), unsigned(ntx), unsigned((nnz + zc - 1) / zc))};
      }
    }
  }
  if (bestCost < 0) throw std::runtime_error("no K*u tile for this grid");
  return best;
}

std::vector<uint32_t> ku_active_tiles(Grid g, const KuShape& k, const std::vector<uint8_t>& present,
                                      std::vector<uint32_t>* zranges) {
  const int nny = g.nny(), nnx = g.nnx(), nnz = g.nnz();
  if (k.grid.x > 1024 || k.grid.y > 1024 || k.grid.z > 4095 || nnz > 65535) return {};
  std::vector<uint32_t> list;
  if (zranges) zranges->clear();
  for (unsigned tz = 0; tz < k.grid.z; ++tz)
    for (unsigned tx = 0; tx < k.grid.y; ++tx)
      for (unsigned ty = 0; ty < k.grid.x; ++ty) {
        int lo = -1, hi = -1;
        for (int z = int(tz) * k.zc; z < std::min(nnz, int(tz + 1) * k.zc); ++z) {
          bool any = false;
          for (int x = int(tx) * k.TX; x < std::min(nnx, int(tx + 1) * k.TX) && !any; ++x)
            for (int y = int(ty) * k.TY; y < std::min(nny, int(ty + 1) * k.TY) && !any; ++y)
              any = present[size_t(y + int64_t(nny) * (x + int64_t(nnx) * z))] != 0;
          if (any) {
            if (lo < 0) lo = z;
            hi = z + 1;
          }
        }
        if (lo >= 0) {
          list.push_back(ty | (tx << 10) | (tz << 20));
          if (zranges) zranges->push_back(uint32_t(lo) | (uint32_t(hi) << 16));
        }
      }
  return list;
}

void launch_ku(cudaStream_t st, KuMode mode, const KuArgs& args, int ntiles) {
  const dim3 grd = args.active ? dim3(unsigned(ntiles)) : args.sh.grid;
  if (grd.x == 0) return;
  if (mode == KU_PLAIN)
    (k_ku<KU_PLAIN><<<grd, KU_NT, sizeof(KuSmem<KU_PLAIN>), st>>>(args), topx::count_launch());
  else
    (k_ku<KU_P_UPDATE><<<grd, KU_NT, sizeof(KuSmem<KU_P_UPDATE>), st>>>(args), topx::count_launch());
  TOPX_CUDA_OK(cudaGetLastError());
}

}  // namespace topx
