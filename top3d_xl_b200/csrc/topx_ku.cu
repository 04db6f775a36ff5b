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
// come first, so a smooth field cancels exactly at the start instead of at the end of long sums: error against long
// double 1.1e-15 (Ke's entries: 3.8e-15), on a large offset 8.4e-13 (4.5e-12), for random fields 2.21e-16 (2.24e-16).
//
// Tiles.  A CTA of 256 threads marches a z-chunk of a PY x PX tile of node columns (y fastest), one
// thread per column; the outer ring is halo.  One thread copies the boxes of a plane's fields two planes ahead by
// TMA (out-of-grid entries arrive as zeros); every thread forms the operator's input at its own node
// there (masked u, or the PCG direction), and exchanges through shared memory twice per plane: its
// value with the other corners of its face, and its face's forces with the nodes at those corners.  The
// transformed face of the plane below and the forces from the layer below stay in registers.  No
// atomics: the result is deterministic.
//
// Measured on a B200, one PCG-mode launch (128x256x128, 64x128x64 and 50x100x50 elements), the direction formed
// from the residual and the level-2 correction included: 188, 40 and 29 us.  With z read from memory 185, 36 and
// 27 us, to which the prolongation that wrote z added 80, 25 and 21 us.  With Ke's 576 entries in a 32 x 8 tile and
// a launch for the last row, z read: 280, 54 and 32 us.  What bounds it is the number of instructions an SM issues
// (0.5 per cycle and scheduler with its 16 warps, a third of them FP64; DRAM 35 %), then the two barriers of a plane.  What was slower:
// 8-byte asynchronous copies by every thread instead of TMA (300 us: they need L1 lines, of which little is left
// beside the shared memory), a spilled register (local memory goes to L2 for the same reason: 240 to 320), two
// planes per barrier, loads into registers one plane ahead, CTAs of 128 or 512 threads, three CTAs per SM.
#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <type_traits>
#include <vector>

#include "topx_ke_classes.h"
#include "topx_kernels.cuh"
#include "topx_tma.cuh"

namespace topx {

namespace {

constexpr int KU_NT = 256;  // threads of a CTA
constexpr int KU_CTAS = 2;  // CTAs of an SM
constexpr int KU_PAD = 64;  // reach of a neighbour index (PY + 1)
constexpr int KU_ROW = KU_NT + KU_PAD;
constexpr int KU_COARSE = 64;  // coarse nodes of a tile per plane

template <int BYTES>
__device__ __forceinline__ void cp_async_el(void* smem, const void* gmem, bool pred) {
  static_assert(BYTES == 4 || BYTES == 8, "element copy size");
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int n = pred ? BYTES : 0;  // 0: fill with zeros, read nothing
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Maps of the arrays that a launch reads through TMA, and the places of their boxes in a stage
struct KuMaps {
  CUtensorMap a, E, p, y, D;  // u, z or r; (PCG) p_in, y; (fused) the Jacobi diagonal
};
// Offsets in doubles of a stage's boxes, and its length; boxes start on 128-byte boundaries
struct KuStage {
  int E, p, y, D, len;
};

template <int MODE>
struct KuSmem {
  static constexpr bool FUSED = MODE == KU_FUSED;
  double su[2][3][KU_ROW];   // a plane's masked values, and those of the plane below, read by their own threads
  double cor[3][3][KU_ROW];  // face forces for the corners (y+1, x), (y, x+1), (y+1, x+1)
  double xc[FUSED ? 3 : 1][FUSED ? 3 : 1][FUSED ? KU_COARSE : 1];  // ring of level-2 planes under the tile
  int at[FUSED ? 3 : 1][FUSED ? KU_NT : 1];  // the thread's level-2 copy (element, slot) and its node's place in a cell
  double zc[FUSED ? 2 : 1][FUSED ? 3 : 1][FUSED ? KU_NT : 1];  // xc at the node's (y, x) on the planes that end its cell
  uint64_t bar[2];
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
// KU_FUSED: z = omega2 (r D) + P xc is formed here from the residual r, the inverse diagonal D (one
// value per node: the diagonal entries of its free DOFs are equal) and the level-2 correction xc, so no
// pass over the level-1 grid writes or reads z.  TC: the preconditioner's type.
// Both store p, reduce p'q into sc->pq and apply the previous iteration's solution step y += lam p_in.
// OFF: the type of a node's byte offset.
template <int MODE, typename TC, typename OFF>
__global__ void __launch_bounds__(KU_NT, KU_CTAS)
    k_ku(const __grid_constant__ KuArgs a, const __grid_constant__ KuMaps maps, const KuStage sg, const unsigned bytes) {
  constexpr bool PCG = MODE != KU_PLAIN;
  extern __shared__ __align__(128) double ku_stages[];  // two planes' boxes, then the rest
  KuSmem<MODE>& sm = *reinterpret_cast<KuSmem<MODE>*>(ku_stages + 2 * sg.len);
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
  const bool own = inb && ly >= 1 && ly <= a.sh.TY && lx >= 1 && lx <= a.sh.TX;
  // byte offsets of the node on plane 0 and of a plane
  const OFF n0 = inb ? 8u * OFF(gy + nny * gx) : 0u, np = 8u * OFF(nny) * OFF(nnx);
  // the node's place in a box of TY + 4 rows from y0 - 2, and (own nodes) in y's box of the tile itself
  const int PB = a.sh.TY + 4, bx = PB * a.sh.PX, o = in_tile ? lx * PB + ly + 1 : 0;
  const int oy = own ? (lx - 1) * a.sh.TY + ly - 1 : 0, by = a.sh.TY * a.sh.TX;
  const TC* const xc = static_cast<const TC*>(a.xc);

  // level-2 nodes under the tile (fused), copied by the threads t < 3 cn; kept in shared memory, since the loop
  // needs every register
  const int Zfirst = max(zc0 - 1, 0) / KU_SPAN;
  if (MODE == KU_FUSED) {
    const int Yc0 = max(y0 - 1, 0) / KU_SPAN, Xc0 = max(x0 - 1, 0) / KU_SPAN;
    const int cny = min((y0 + a.sh.TY) / KU_SPAN + 1, a.gc.ny) - Yc0 + 1;
    const int cn = cny * (min((x0 + a.sh.TX) / KU_SPAN + 1, a.gc.nx) - Xc0 + 1);
    const int c = t / cn, r = t - c * cn, xx = r / cny, yy = r - xx * cny;
    sm.at[0][t] = c < 3 ? int((Yc0 + yy) + (a.gc.ny + 1) * (Xc0 + xx) + c * a.gc.stride) : -1;
    sm.at[1][t] = c * KU_COARSE + r;
    const int Y = gy / KU_SPAN, X = gx / KU_SPAN;
#pragma unroll
    for (int i = 0; i < 3; ++i) sm.zc[0][i][t] = sm.zc[1][i][t] = 0.0;  // stays so off the level-2 grid (weight 0)
    sm.at[2][t] = inb && gy <= KU_SPAN * a.gc.ny ? (Y - Yc0) + cny * (X - Xc0) + (gy % KU_SPAN << 8) + (gx % KU_SPAN << 10) + (cny << 12) : -1;
  }
  auto issue_coarse = [&](int Z) {
    const int e = sm.at[0][t];
    if (e >= 0) {
      const bool ok = Z <= a.gc.nz;
      TC* dst = reinterpret_cast<TC*>(&sm.xc[Z % 3][0][0]) + sm.at[1][t];
      cp_async_el<int(sizeof(TC))>(dst, xc + (ok ? int64_t(e) + int64_t(a.gc.ny + 1) * (a.gc.nx + 1) * Z : 0), ok);
    }
  };
  bool ok = true;  // no wait of this thread gave up
  // one thread issues the copies of plane zp and of the layer below it
  auto issue = [&](int zp, int s) {
    if (t == 0 && ok) {
      double* d = ku_stages + s * sg.len;
      mbar_expect(&sm.bar[s], bytes);
      tma_load(d, &maps.a, y0 - 2, x0 - 1, zp, &sm.bar[s]);
      tma_load(d + sg.E, &maps.E, y0 - 2, x0 - 1, zp - 1, &sm.bar[s]);
      if (PCG) {
        tma_load(d + sg.p, &maps.p, y0 - 2, x0 - 1, zp, &sm.bar[s]);
        tma_load(d + sg.y, &maps.y, y0, x0, zp, &sm.bar[s]);
      }
      if (MODE == KU_FUSED) tma_load(d + sg.D, &maps.D, y0 - 2, x0 - 1, zp, &sm.bar[s]);
    }
    // the far end of the cell that begins on plane zp, whose readers are past a barrier by then
    if (MODE == KU_FUSED && zp % KU_SPAN == 0) issue_coarse(zp / KU_SPAN + 1);
  };
  if (t == 0) {
    tma_prefetch(&maps.a);
    tma_prefetch(&maps.E);
    if (PCG) tma_prefetch(&maps.p);
    if (PCG) tma_prefetch(&maps.y);
    if (MODE == KU_FUSED) tma_prefetch(&maps.D);
    mbar_init(&sm.bar[0]);
    mbar_init(&sm.bar[1]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  if (MODE == KU_FUSED) {
    for (int Z = 0; Z < 3; ++Z) issue_coarse(Zfirst + Z);
  }
  issue(zc0 - 1, 0);
  issue(zc0, 1);
  auto flags_at = [&](int zp) -> unsigned {
    return inb && zp >= 0 && zp < nnz ? unsigned(a.flags[(n0 + np * OFF(zp)) / 8u]) : 0u;
  };
  unsigned f = flags_at(zc0 - 1), fo = 0;  // of the plane, and of the one below
  const bool first = PCG && (MODE == KU_FUSED ? a.sc->its == 0 : a.sc->first != 0);
  const double lam = PCG ? a.sc->lam : 0.0;
  double beta = PCG ? a.sc->beta : 0.0;
  if (PCG && a.sc->done) {  // the same for the whole launch
    cp_async_wait_all();
    ok = plane_wait(sm.bar, 0, 1, t == 0) && plane_wait(sm.bar, 1, 1, t == 0);
    if (!ok) report_copy_wait(a.err);
    return;
  }
  if (MODE == KU_FUSED && a.parts.dot.n) {  // z'r, whose level-2 part the prolongation left in parts
    const int its = a.sc->its;
    const double zr = fma(a.omega2, a.sc->rdr, parts_sum(a.parts.dot));
    if (its > 0) beta = zr / a.sc->zr[(its - 1) & 1];
    if (blockIdx.x + blockIdx.y + blockIdx.z == 0 && t == 0) a.sc->zr[its & 1] = zr;
  }
  // xc interpolated to the node's (y, x) on level-2 plane Z (fused)
  auto coarse = [&](int Z) {
    const int e = sm.at[2][t];
    if (e < 0) return;
    const int c0 = e & 255, wy = e >> 8 & 3, wx = e >> 10 & 3, dy = wy ? 1 : 0, dx = wx ? e >> 12 : 0;
    const TC* p = reinterpret_cast<const TC*>(&sm.xc[Z % 3][0][0]) + c0;
    const double fy = double(wy) / KU_SPAN, fx = double(wx) / KU_SPAN;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const TC* q = p + c * KU_COARSE;
      double s = (1.0 - fy) * (1.0 - fx) * double(q[0]);
      s = fma(fy * (1.0 - fx), double(q[dy]), s);
      s = fma((1.0 - fy) * fx, double(q[dx]), s);
      sm.zc[Z & 1][c][t] = fma(fy * fx, double(q[dx + dy]), s);
    }
  };
  double dot = 0.0;
  // Plane zp in slot s, and the element layer below it (between the faces Wp and W): plane zp - 1 is then
  // complete.  G holds its forces in face modes, Bn takes the layer's part of plane zp's.
  auto step = [&](int zp, int s, double (&Wp)[3][4], double (&W)[3][4], double (&G)[3][4], double (&Bn)[3][4]) {
    const OFF n = n0 + np * OFF(zp);
    const bool mine = own && zp >= zc0 && zp < zend;
    const double* st = ku_stages + s * sg.len;
    if (ok) ok = plane_wait(sm.bar, zp - zc0 + 1, zend - zc0 + 1, t == 0);
    if (MODE == KU_FUSED) cp_async_wait_all();  // level-2 planes, a plane ahead of their use
    const double E = st[sg.E + o];
    double v[3], y[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = st[c * bx + o];
    if (MODE == KU_FUSED) {
      const int Z = zp / KU_SPAN, tz = zp & (KU_SPAN - 1);
      if (zp < zc0) {
        __syncthreads();  // the first level-2 planes, copied by other threads
        coarse(Zfirst);
        coarse(Zfirst + 1);
      } else if (tz == 0 && zp > 0) {
        coarse(Z + 1);
      }
      const double D = st[sg.D + o];
      // z is zero off the domain: no correction there, and r is zero
      const double wz = f & 8u ? tz * (1.0 / KU_SPAN) : 0.0, wa = f & 8u ? 1.0 - tz * (1.0 / KU_SPAN) : 0.0;
      double d[3] = {D, D, D};
      if (f & 7u)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (f & (1u << c)) d[c] = double(TC(*at(a.icfix, n)));  // a fixed DOF's diagonal
#pragma unroll
      for (int c = 0; c < 3; ++c)
        v[c] = fma(a.omega2 * v[c], d[c], fma(wz, sm.zc[(Z + 1) & 1][c][t], wa * sm.zc[Z & 1][c][t]));
    }
    if (PCG) {
      if (!first) {
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = fma(beta, st[sg.p + c * bx + o], v[c]);
      }
      if (mine) {
#pragma unroll
        for (int c = 0; c < 3; ++c) *at(a.pout + c * S, n) = v[c];
        if (!first)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            *at(a.yacc + c * S, n) = fma(lam, st[sg.p + c * bx + o], st[sg.y + c * by + oy]);
      }
    }
    if (f & 7u)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        if (f & (1u << c)) v[c] = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) sm.su[s][c][t] = v[c];
    const unsigned fn = flags_at(zp + 1);
    __syncthreads();
    if (zp + 2 <= zend) issue(zp + 2, s);  // every thread has read the stage
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
          const OFF m = n - np;
          double p[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            y[c] = (y[c] + sm.cor[1][c][KU_PAD + t - PY]) +
                   (sm.cor[0][c][KU_PAD + t - 1] + sm.cor[2][c][KU_PAD + t - PY - 1]);
            if (PCG) p[c] = sm.su[s ^ 1][c][t];
          }
          if (fo & 7u) {  // a fixed DOF: its own value, unmasked
            const double cf = *at(a.cfix, m);
#pragma unroll
            for (int c = 0; c < 3; ++c)
              if (fo & (1u << c)) {
                p[c] = PCG ? *at(a.pout + c * S, m) : *at(a.in + c * S, m);
                y[c] = cf * p[c];
              }
          }
          if (MODE == KU_PLAIN && a.compact) {
            const int k = a.compact[m / 8u];
            if (k >= 0)
#pragma unroll
              for (int c = 0; c < 3; ++c) a.out[3 * int64_t(k) + c] = y[c];
          } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) *at(a.out + c * S, m) = y[c];
          }
          if (PCG)
#pragma unroll
            for (int c = 0; c < 3; ++c) dot = fma(p[c], y[c], dot);
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
  if (!ok) report_copy_wait(a.err);
  if (MODE == KU_FUSED && a.parts.pq.n) {  // the residual pass sums them
    double r[1] = {dot};
    parts_leave<1>(r, {a.parts.pq.part});
  } else if (PCG) {
    double r[1] = {dot}, tot[1];
    if (reduce_publish<1>(r, a.rs, tot) && t == 0) a.sc->pq = tot[0];
  }
}

// Grids below this many nodes have fields of less than 4 GB, whose offsets fit 32 bits and cost no instruction;
// beyond, the same kernel with 64-bit offsets.
constexpr int64_t kOffset32Nodes = int64_t(1) << 29;

template <int MODE, typename TC>
void ku_smem_attr() {
  for (auto kernel : {k_ku<MODE, TC, uint32_t>, k_ku<MODE, TC, uint64_t>})
    TOPX_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024 / KU_CTAS));
}

}  // namespace

// the give-up path of the operator's waits: two barriers that no copy completes
__global__ void k_copy_wait_selftest(int* err) {
  pdl_wait();
  __shared__ uint64_t bar[2];
  if (threadIdx.x == 0) {
    mbar_init(&bar[0]);
    mbar_init(&bar[1]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (!plane_wait(bar, 0, 1, threadIdx.x == 0)) report_copy_wait(err);
}
void launch_copy_wait_selftest(cudaStream_t st, int* err) {
  launch_pdl(st, k_copy_wait_selftest, 1, 32, 0, err);
  TOPX_CUDA_OK(cudaGetLastError());
}

void prepare_ku_kernels() {
  ku_smem_attr<KU_PLAIN, double>();
  ku_smem_attr<KU_P_UPDATE, double>();
  ku_smem_attr<KU_FUSED, double>();
  ku_smem_attr<KU_FUSED, float>();
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
// about two planes' worth of start and end), each plane's with its warps and the sectors that its rows touch;
// two CTAs fit an SM, a last wave that is nearly empty costs about half a wave, and long chunks drift apart
// and lose the halo planes that neighbours share in L2.  Every even tile height whose tiles come out
// even, with the widest tile that then fits the CTA, and every chunk length are compared.  Sweeps of tiles and
// chunks at the sizes above found at most 5 % more.
KuShape ku_shape(Grid g, int rows) {
  const int nny = rows, nnx = g.nnx(), nnz = g.nnz();
  const double slots = double(KU_CTAS) * num_sms();
  KuShape best{};
  double bestCost = -1;
  for (int nty = 1; nty <= nny; ++nty) {
    const int TY = (((nny + nty - 1) / nty) + 1) & ~1, PY = TY + 2;  // even: a box starts on a 16-byte boundary
    if (PY > KU_PAD - 2 || (nny + TY - 1) / TY != nty) continue;
    if (PY * 3 > KU_NT) continue;
    if (TY < 6 && nny >= 6) break;
    const int TXmax = std::min(KU_NT / PY - 2, nnx);
    const int ntx = (nnx + TXmax - 1) / TXmax, TX = (nnx + ntx - 1) / ntx, PX = TX + 2;
    if (((PY + 2) / KU_SPAN + 2) * ((PX + 2) / KU_SPAN + 2) > KU_COARSE) continue;
    const double plane_cost = (PY * PX + 31) / 32 * (1.0 + 3.0 / PY) / 8.0 + 0.4;
    for (int zc = 1; zc <= 64 && zc <= nnz + 1; ++zc) {
      const double ctas = double(nty) * ntx * ((nnz + zc - 1) / zc);
      const double waves = ctas / slots, w = waves <= 1.0 ? 1.0 : 0.5 * (waves + std::ceil(waves));
      const double cost = (w + 0.3) * (zc + 4) * (1.0 + 0.003 * zc) * plane_cost;
      if (bestCost < 0 || cost < bestCost) {
        bestCost = cost;
        best = KuShape{PY, PX, TY, TX, zc, dim3(unsigned(nty), unsigned(ntx), unsigned((nnz + zc - 1) / zc))};
      }
    }
  }
  if (bestCost < 0) throw std::runtime_error("no K*u tile for this grid");
  return best;
}

std::vector<uint32_t> ku_active_tiles(Grid g, int rows, const KuShape& k, const std::vector<uint8_t>& present,
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
            for (int y = int(ty) * k.TY; y < std::min(rows, int(ty + 1) * k.TY) && !any; ++y)
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

template <int MODE, typename TC>
static void launch(cudaStream_t st, const KuArgs& a, dim3 grd) {
  const int PB = a.sh.TY + 4, PX = a.sh.PX, box = PB * PX, own = a.sh.TY * a.sh.TX;
  auto up = [](int doubles) { return (doubles + 15) / 16 * 16; };
  KuMaps m{};
  KuStage sg{};
  int at = up(3 * box), used = 4 * box;
  m.a = field_map(a.in, a.g, 3, PB, PX);
  m.E = field_map(a.E, a.g, 1, PB, PX);
  sg.E = at;
  at += up(box);
  if (MODE != KU_PLAIN) {
    m.p = field_map(a.pin, a.g, 3, PB, PX);
    sg.p = at;
    at += up(3 * box);
    m.y = field_map(a.yacc, a.g, 3, a.sh.TY, a.sh.TX);
    sg.y = at;
    at += up(3 * own);
    used += 3 * box + 3 * own;
  }
  if (MODE == KU_FUSED) {
    m.D = field_map(a.D, a.g, 1, PB, PX);
    sg.D = at;
    at += up(box);
    used += box;
  }
  sg.len = at;
  const size_t smem = sizeof(double) * 2 * size_t(at) + sizeof(KuSmem<MODE>);
  launch_pdl(st, a.g.nnodes() < kOffset32Nodes ? k_ku<MODE, TC, uint32_t> : k_ku<MODE, TC, uint64_t>, grd, KU_NT, smem, a, m,
             sg, unsigned(8 * used));
}
void launch_ku(cudaStream_t st, KuMode mode, const KuArgs& args, int ntiles) {
  const dim3 grd = args.active ? dim3(unsigned(ntiles)) : args.sh.grid;
  if (grd.x == 0) return;
  if (mode == KU_PLAIN)
    launch<KU_PLAIN, double>(st, args, grd);
  else if (mode == KU_P_UPDATE)
    launch<KU_P_UPDATE, double>(st, args, grd);
  else if (args.pre32)
    launch<KU_FUSED, float>(st, args, grd);
  else
    launch<KU_FUSED, double>(st, args, grd);
  TOPX_CUDA_OK(cudaGetLastError());
}

}  // namespace topx
