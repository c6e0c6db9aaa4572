// K6: force and potential gather (de2, sfac.cpp:409-483; potl,
// sfac.cpp:497-545).
//
// One thread per point, 8 lanes per point (few points) or a CTA per brick of
// the grid (many): every output has exactly one writer, and the sum order is
// fixed and the same in all three.  The stencil origin is computed in FP64 exactly as the
// reference does (u = scale(x)*K, k1 = ceil(u), k0 = (k1 - order/2) mod K);
// the B-spline weights and the order^3 sum are FP32, factorised as
// sum_i wx_i sum_j wy_j sum_k wz_k Q  (one pass gives phi and all three
// derivatives).  The chain rule through iL and the scaling are FP64.
#include <algorithm>
#include <cmath>

#include "reduce.cuh"
#include "spme_kernels.hpp"

namespace spme {

SPME_CHECK_READER(gather)

constexpr int kCellWords = 16;  // 9 used: sum_a s_a,i (dE/dr_a)_j

// idx[i] = (o + i) mod K for 0 <= o < K, without a division when K >= P.
template <int P>
__device__ __forceinline__ void wrap_run(int o, int K, int (&idx)[P]) {
  if (K >= P) {
#pragma unroll
    for (int i = 0; i < P; i++) {
      const int v = o + i;
      idx[i] = v >= K ? v - K : v;
    }
  } else {
#pragma unroll
    for (int i = 0; i < P; i++) idx[i] = (o + i) % K;
  }
}

// Sums of one x plane of the stencil, sy = sum_j wy_j sum_k wz_k Q and the two
// with a derivative: pl points at the plane's first value of the run in z.
// WRAP false: the z indices are 0 .. P - 1; true: iz[k].
template <int P, bool WRAP>
__device__ __forceinline__ void plane_sum(const float *__restrict__ grid, const Geom &g, const float *pl,
                                          const int (&iy)[P], const int (&iz)[P], const float (&wy)[P],
                                          const float (&dwy)[P], const float (&wz)[P], const float (&dwz)[P], float &sy,
                                          float &dy, float &dz) {
  sy = dy = dz = 0.f;
#pragma unroll
  for (int j = 0; j < P; j++) {
    const float *col = pl + (long)iy[j] * g.K2;
    float sz = 0.f, dzz = 0.f;
#pragma unroll
    for (int k = 0; k < P; k++) {
      const float q = SPME_IN(col + (WRAP ? iz[k] : k) - grid, (long)g.K0 * g.K1 * g.K2, CK_GATHER_GRID)
                          ? __ldg(col + (WRAP ? iz[k] : k))
                          : 0.f;
      sz = fmaf(wz[k], q, sz);
      dzz = fmaf(dwz[k], q, dzz);
    }
    sy = fmaf(wy[j], sz, sy);
    dy = fmaf(dwy[j], sz, dy);
    dz = fmaf(wy[j], dzz, dz);
  }
}

// Vector width of the row loads: each z run of P values is read as W / kVW
// aligned float2 loads from zb = o2 rounded down to even (W = P + 2 values,
// the weights shifted by o2 - zb with zeros around the run).  4 loads instead
// of 6 per row at order 6 (fewer L1 requests); the extra terms are exact
// zeros, so the sums are bit-identical to the scalar ones.  float4 windows
// (3 loads of 12 values) measured no faster.
constexpr int kVW = 2;  // float2
template <int P> struct VecWin { static constexpr int W = (P + kVW - 1 + kVW - 1) / kVW * kVW; };

// The same from aligned vector loads: the window of W values at pl holds the
// run, the weights are pre-shifted (zeros outside the run).
template <int P>
__device__ __forceinline__ void plane_sum_vec(const float *__restrict__ grid, const Geom &g, const float *pl,
                                              const int (&iy)[P], const float (&wy)[P], const float (&dwy)[P],
                                              const float (&wz)[VecWin<P>::W], const float (&dwz)[VecWin<P>::W],
                                              float &sy, float &dy, float &dz) {
  sy = dy = dz = 0.f;
#pragma unroll
  for (int j = 0; j < P; j++) {
    const float *col = pl + (long)iy[j] * g.K2;
    float sz = 0.f, dzz = 0.f;
#pragma unroll
    for (int v = 0; v < VecWin<P>::W / kVW; v++) {
      const float2 q = SPME_IN(col + 2 * v + 1 - grid, (long)g.K0 * g.K1 * g.K2, CK_GATHER_GRID)
                           ? __ldg(reinterpret_cast<const float2 *>(col) + v)
                           : make_float2(0.f, 0.f);
      sz = fmaf(wz[2 * v], q.x, sz); dzz = fmaf(dwz[2 * v], q.x, dzz);
      sz = fmaf(wz[2 * v + 1], q.y, sz); dzz = fmaf(dwz[2 * v + 1], q.y, dzz);
    }
    sy = fmaf(wy[j], sz, sy);
    dy = fmaf(dwy[j], sz, dy);
    dz = fmaf(wy[j], dzz, dz);
  }
}

// Order-P stencil sum of the grid around one point, factorised per axis:
// pot = sum_i wx_i sum_j wy_j sum_k wz_k Q, and the three derivatives, the
// planes in order.  plane(xi, sy, dy, dz): the sums of grid plane xi.
template <int P, class F>
__device__ __forceinline__ void stencil_sum(const Geom &g, int o0, const float (&wx)[P], const float (&dwx)[P],
                                            F &&plane, float &pot, float &gx, float &gy, float &gz) {
  int xi = o0;  // (o0 + i) mod K0
#pragma unroll 1
  for (int i = 0; i < P; i++, xi = (xi + 1 == g.K0) ? 0 : xi + 1) {
    float sy, dy, dz;
    plane(xi, sy, dy, dz);
    pot = fmaf(wx[i], sy, pot);
    gx = fmaf(dwx[i], sy, gx);
    gy = fmaf(wx[i], dy, gy);
    gz = fmaf(wx[i], dz, gz);
  }
}

// Calls f with the plane sums of a point whose z run starts at o2, as a
// function of the plane: f([](xi, sy, dy, dz)).  The choice between vector
// loads, plain loads and wrapped indices is warp-uniform (no divergent second
// copy of the stencil); it depends on nothing but the active lanes' o2.
template <int P, class F>
__device__ __forceinline__ void with_planes(const float *__restrict__ grid, const Geom &g, const int (&iy)[P], int o2,
                                            const float (&wy)[P], const float (&dwy)[P], const float (&wz)[P],
                                            const float (&dwz)[P], F &&f) {
  const long plane = (long)g.K1 * g.K2;
  int iz[P];
  const int sh = o2 & (kVW - 1), zb = o2 - sh;
  if ((g.K2 % kVW) == 0 && __all_sync(__activemask(), zb + VecWin<P>::W <= g.K2)) {
    constexpr int W = VecWin<P>::W;
    float wzv[W], dwzv[W];
#pragma unroll
    for (int k = 0; k < W; k++) {
      float v = 0.f, d = 0.f;
#pragma unroll
      for (int t = 0; t < kVW; t++)
        if (k - t >= 0 && k - t < P) {
          v = (sh == t) ? wz[k - t] : v;
          d = (sh == t) ? dwz[k - t] : d;
        }
      wzv[k] = v;
      dwzv[k] = d;
    }
    f([&](int xi, float &sy, float &dy, float &dz) {
      plane_sum_vec<P>(grid, g, grid + xi * plane + zb, iy, wy, dwy, wzv, dwzv, sy, dy, dz);
    });
  } else if (__all_sync(__activemask(), o2 + P <= g.K2)) {
    f([&](int xi, float &sy, float &dy, float &dz) {
      plane_sum<P, false>(grid, g, grid + xi * plane + o2, iy, iz, wy, dwy, wz, dwz, sy, dy, dz);
    });
  } else {
    wrap_run<P>(o2, g.K2, iz);
    f([&](int xi, float &sy, float &dy, float &dz) {
      plane_sum<P, true>(grid, g, grid + xi * plane, iy, iz, wy, dwy, wz, dwz, sy, dy, dz);
    });
  }
}

// Cell-sorted view of the points (from the cell sort of the same solve):
// sorted rank r is point perm[r], in cell key[r] with in-cell fractions
// rec[r].xyz.  Consecutive threads then read neighbouring grid points.
struct SortedView {
  const uint32_t *perm, *key;
  const float4 *rec;
  FastDiv K2d, K12d;  // division by K2 and by K1*K2
};

// A point's input index, stencil origin (wrapped) and B-spline arguments; see
// gather_kernel for SORTED.
struct PointAt {
  int a, o0, o1, o2;
  float t0, t1, t2;
};
template <int P, bool SORTED>
__device__ __forceinline__ PointAt point_at(const Geom &g, int r, int n, const double *__restrict__ x,
                                            const SortedView &sv) {
  PointAt p;
  if (SORTED) {
    p.a = (int)sv.perm[r];
    uint32_t key = sv.key[r];
    // a failed check substitutes atom 0 / key 0 (the run is flagged already)
    if (!SPME_IN(p.a, n, CK_GATHER_ATOM)) p.a = 0;
    if (!SPME_IN(key, (long)g.K0 * g.K1 * g.K2, CK_GATHER_KEY)) key = 0;
    const float4 u = sv.rec[r];
    const uint32_t n0 = sv.K12d.div(key), rem = key - n0 * (uint32_t)(g.K1 * g.K2);
    const uint32_t n1 = sv.K2d.div(rem), n2 = rem - n1 * (uint32_t)g.K2;
    p.o0 = imod((int)n0 + 1 - P / 2, g.K0);
    p.o1 = imod((int)n1 + 1 - P / 2, g.K1);
    p.o2 = imod((int)n2 + 1 - P / 2, g.K2);
    p.t0 = 1.f - u.x;
    p.t1 = 1.f - u.y;
    p.t2 = 1.f - u.z;
  } else {
    const CellConst cc = *g.cell;
    p.a = r;
    double s0, s1, s2;
    frac_coords(cc, x[3 * r + 0], x[3 * r + 1], x[3 * r + 2], s0, s1, s2);
    const double u0 = __dmul_rn(s0, (double)g.K0), u1 = __dmul_rn(s1, (double)g.K1), u2 = __dmul_rn(s2, (double)g.K2);
    const int c0 = (int)ceil(u0), c1 = (int)ceil(u1), c2 = (int)ceil(u2);
    p.t0 = (float)((double)c0 - u0);
    p.t1 = (float)((double)c1 - u1);
    p.t2 = (float)((double)c2 - u2);
    p.o0 = imod(c0 - P / 2, g.K0);
    p.o1 = imod(c1 - P / 2, g.K1);
    p.o2 = imod(c2 - P / 2, g.K2);
  }
  return p;
}

// Stencil sums of a point by one thread.
template <int P>
__device__ __forceinline__ void point_sums(const Geom &g, const Spline &S, const float *__restrict__ grid,
                                           const PointAt &pt, float &pot, float &gx, float &gy, float &gz) {
  float wx[P], dwx[P], wy[P], dwy[P], wz[P], dwz[P];
#pragma unroll
  for (int i = 0; i < P; i++) {
    dbspl_eval(S, P, pt.t0, i, wx[i], dwx[i]);
    dbspl_eval(S, P, pt.t1, i, wy[i], dwy[i]);
    dbspl_eval(S, P, pt.t2, i, wz[i], dwz[i]);
  }
  int iy[P];
  wrap_run<P>(pt.o1, g.K1, iy);
  with_planes<P>(grid, g, iy, pt.o2, wy, dwy, wz, dwz, [&](auto &&plane) {
    stencil_sum<P>(g, pt.o0, wx, dwx, plane, pot, gx, gy, gz);
  });
}

// CELL: also the per-block sums of s_i (dE/dr)_j over the block's points
// (s = iL^T x, unwrapped), written to cellp[block][9] in a fixed order.
// SORTED: thread r handles point perm[r], with the stencil origin from its
// cell (k1 = n + 1, argument 1 - f; for f = 0 this is the reference's
// origin shifted by one cell, whose extra weight M(0) = 0 -- the same sum);
// otherwise the origin comes from x in FP64 exactly as de2/potl compute it.
template <int P, bool GRAD, bool POT, bool CELL, bool SORTED>
__global__ void __launch_bounds__(256, CELL ? 2 : 3) gather_kernel(Geom g, Spline S, int n, const double *__restrict__ x,
                                                     const double *__restrict__ w,
                                                     const float *__restrict__ grid, double *__restrict__ dx,
                                                     double *__restrict__ phi, double *__restrict__ cellp,
                                                     SortedView sv) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  double cacc[9];
  if (CELL) {
#pragma unroll
    for (int c = 0; c < 9; c++) cacc[c] = 0.0;
  }
  if (r < n) {
    const CellConst cc = *g.cell;
    const PointAt pt = point_at<P, SORTED>(g, r, n, x, sv);
    const int a = pt.a;
    float pot = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
    point_sums<P>(g, S, grid, pt, pot, gx, gy, gz);
    if (GRAD) {
      const double f = -w[a] * cc.iV;
      const double G0 = (double)gx * f * g.K0, G1 = (double)gy * f * g.K1, G2 = (double)gz * f * g.K2;
      const double d0 = cc.iL00 * G0;
      const double d1 = cc.iL10 * G0 + cc.iL11 * G1;
      const double d2 = cc.iL20 * G0 + cc.iL21 * G1 + cc.iL22 * G2;
      dx[3 * a + 0] = d0;
      dx[3 * a + 1] = d1;
      dx[3 * a + 2] = d2;
      if (CELL) {
        const double x0 = x[3 * a + 0], x1 = x[3 * a + 1], x2 = x[3 * a + 2];
        const double v0 = x0 * cc.iL00 + x1 * cc.iL10 + x2 * cc.iL20;  // unwrapped s
        const double v1 = x1 * cc.iL11 + x2 * cc.iL21;
        const double v2 = x2 * cc.iL22;
        cacc[0] = v0 * d0; cacc[1] = v0 * d1; cacc[2] = v0 * d2;
        cacc[3] = v1 * d0; cacc[4] = v1 * d1; cacc[5] = v1 * d2;
        cacc[6] = v2 * d0; cacc[7] = v2 * d1; cacc[8] = v2 * d2;
      }
    }
    if (POT) phi[a] = (double)pot * cc.iV;
  }
  if (CELL) {
    __shared__ double red[8][9];
    block_reduce_n<9>(cacc, red, cellp + (long)blockIdx.x * kCellWords);
  }
}

// dE/dL (6: [ax, by, cz, bx, cx, cy]) at fixed Cartesian positions:
//   D = -V iL^T Pi - sum_a s_a (dE/dr_a)^T,  dE/dL = lower triangle of D,
// Pi the virial (symmetric, from ev[1..6]); the first term is dE/dL at fixed
// fractional coordinates (notes.tex: V Pi = -(dE/dL)^T L).
__global__ void cell_grad_kernel(Geom g, const double *__restrict__ cellp, int nblocks,
                                 const double *__restrict__ ev, double *__restrict__ dEdL) {
  __shared__ double P9[9];
  sum_partials<9>(cellp, nblocks, kCellWords, P9);
  if (threadIdx.x != 0) return;
  const CellConst c = *g.cell;
  const double iL[3][3] = {{c.iL00, 0.0, 0.0}, {c.iL10, c.iL11, 0.0}, {c.iL20, c.iL21, c.iL22}};
  const double Pi[3][3] = {{ev[1], ev[4], ev[5]}, {ev[4], ev[2], ev[6]}, {ev[5], ev[6], ev[3]}};
  const double V = 1.0 / c.iV;
  double D[3][3];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      double gs = 0.0;
      for (int k = 0; k < 3; k++) gs += iL[k][i] * Pi[k][j];
      D[i][j] = -V * gs - P9[3 * i + j];
    }
  dEdL[0] = D[0][0];
  dEdL[1] = D[1][1];
  dEdL[2] = D[2][2];
  dEdL[3] = D[1][0];
  dEdL[4] = D[2][0];
  dEdL[5] = D[2][1];
}

// The same for few points: 8 lanes per point, lane i < P sums plane i, and the
// point's first lane adds the planes in order (the same sums, so the same
// bits).  With few points the thread-per-point kernel is one thread's chain of
// P^2 row loads long while most of the chip idles.
template <int P, bool GRAD, bool POT>
__global__ void __launch_bounds__(128) gather_split_kernel(Geom g, Spline S, int n, const double *__restrict__ w,
                                                           const float *__restrict__ grid, double *__restrict__ dx,
                                                           double *__restrict__ phi, SortedView sv) {
  const int r = blockIdx.x * (blockDim.x / 8) + threadIdx.x / 8, i = threadIdx.x & 7;
  const bool live = r < n;
  const PointAt pt = point_at<P, true>(g, live ? r : n - 1, n, nullptr, sv);
  const int a = pt.a, o2 = pt.o2;
  int xi = pt.o0 + min(i, P - 1);
  if (xi >= g.K0) xi %= g.K0;
  float wx = 0.f, dwx = 0.f, wy[P], dwy[P], wz[P], dwz[P];
#pragma unroll
  for (int k = 0; k < P; k++) {
    float b, d;
    dbspl_eval(S, P, pt.t0, k, b, d);
    if (k == i) {
      wx = b;
      dwx = d;
    }
    dbspl_eval(S, P, pt.t1, k, wy[k], dwy[k]);
    dbspl_eval(S, P, pt.t2, k, wz[k], dwz[k]);
  }
  int iy[P];
  wrap_run<P>(pt.o1, g.K1, iy);
  float sy = 0.f, dy = 0.f, dz = 0.f;
  if (i < P)
    with_planes<P>(grid, g, iy, o2, wy, dwy, wz, dwz, [&](auto &&plane) { plane(xi, sy, dy, dz); });
  __syncwarp();
  float pot = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
  for (int k = 0; k < P; k++) {  // every lane of the point adds the planes in order
    const float wk = __shfl_sync(0xffffffffu, wx, k, 8), sk = __shfl_sync(0xffffffffu, sy, k, 8);
    if (POT) pot = fmaf(wk, sk, pot);
    if (GRAD) {
      gx = fmaf(__shfl_sync(0xffffffffu, dwx, k, 8), sk, gx);
      gy = fmaf(wk, __shfl_sync(0xffffffffu, dy, k, 8), gy);
      gz = fmaf(wk, __shfl_sync(0xffffffffu, dz, k, 8), gz);
    }
  }
  if (!live) return;
  const CellConst cc = *g.cell;
  if (GRAD && i < 3) {  // lane i writes component i
    const double f = -w[a] * cc.iV;
    const double G0 = (double)gx * f * g.K0, G1 = (double)gy * f * g.K1, G2 = (double)gz * f * g.K2;
    dx[3 * a + i] = i == 0 ? cc.iL00 * G0
                           : (i == 1 ? cc.iL10 * G0 + cc.iL11 * G1 : cc.iL20 * G0 + cc.iL21 * G1 + cc.iL22 * G2);
  }
  if (POT && i == 3) phi[a] = (double)pot * cc.iV;
}

// ---------------------------------------------------------------------------
// Gather by bricks: the grid block of a brick in shared memory.
//
// One CTA takes the points of a brick of TX x TY x 32 cells (whole buckets of
// the cell sort, so the points are TX TY contiguous runs of the sorted order)
// and copies the brick's grid block with its stencil halo, rows of 40 values
// from 4 below the brick, to shared memory with cp.async (periodic images row
// by row).  One thread then takes one point, reads its P^3 values with
// constant offsets from one address, and no load passes the L1 tag stage,
// which bounds the thread-per-point kernel above.
//
// Shared-memory wavefronts bound it instead (23 M at 1M points, order 6; 61%
// of the pipe's peak).  32 lanes at unrelated places cost about 3.4
// wavefronts per load.  All lanes add the same offset for the same tap, so
// the lanes of a warp are conflict-free on every load when their origins
// differ modulo 32: the brick's points are ordered by (rank within their
// origin's class modulo 32, class), which brings it to 2.0.  The order only
// decides which thread computes a point, never a result, so the ranks may
// come from shared-memory atomics.  1M points, order 6, 256^3: 183 -> 135 us.
template <int P, int TX, int TY, int NT_>
struct TileCfg {
  static constexpr int NT = NT_;  // threads
  static constexpr int RX = TX + P - 1, RY = TY + P - 1, PITCH = 40, Z0 = 4;
  static constexpr int ROWS = RX * RY, CELLROWS = TX * TY;
  static constexpr int ITEMS = (TX * TY * 4 + NT - 1) / NT < 2 ? 2 : (TX * TY * 4 + NT - 1) / NT;
  static constexpr int CAP = ITEMS * NT;             // points ordered at a time
  static constexpr int LEVELS = 64;                  // ranks that get an exact place; later ones follow in any order
};
template <int P, int TX, int TY, int NT>
struct TileSmem {
  using C = TileCfg<P, TX, TY, NT>;
  __align__(16) float tile[C::ROWS * C::PITCH];
  float4 rec[C::CAP];  // fractions of the points in the conflict-free order
  uint2 list[C::CAP];  // their input index and origin
  int rowidx[C::ROWS]; // grid row (x K1 + y) of every tile row
  int start[C::CELLROWS], pref[C::CELLROWS + 1];
  uint32_t lmask[C::LEVELS];
  int lbase[C::LEVELS + 1];
  __align__(16) int hist[32];
  int wsum[32], extra;
};

struct TileArgs {
  Geom g;
  const int *cs;        // bucket offsets of the cell sort
  const uint32_t *perm, *key;
  const float4 *rec;
  const double *w;
  const float *grid;
  double *dx, *phi;
  int n, nty, nzb;
  long nb;
  const uint32_t *crowd;  // the sort's crowd word
};

// Enqueues the copies of the brick's tile rows in pieces of V values.
template <int P, int TX, int TY, int NT, int V>
__device__ __forceinline__ void tile_copy(const TileArgs &A, TileSmem<P, TX, TY, NT> &sm, int z0) {
  using C = TileCfg<P, TX, TY, NT>;
  constexpr int PQ = C::PITCH / V;
  const int K2 = A.g.K2, nq = K2 / V;
  const int zq0 = imod(z0 - C::Z0, K2) / V;
  for (int e = threadIdx.x; e < C::ROWS * PQ; e += NT) {
    const int r = e / PQ, c = e - r * PQ;
    int zq = zq0 + c;
    if (zq >= nq) zq = nq >= PQ ? zq - nq : zq % nq;
    const long src = (long)sm.rowidx[r] * K2 + V * zq;
    if (!SPME_IN(src, (long)A.g.K0 * A.g.K1 * K2 - (V - 1), CK_GATHER_GRID)) continue;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(sm.tile + r * C::PITCH + V * c);
    if (V == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(A.grid + src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(A.grid + src), "n"(4 * V) : "memory");
  }
}

template <int P, int TX, int TY, int NT, bool GRAD, bool POT>
__global__ void __launch_bounds__(NT, 768 / NT) gather_tile_kernel(TileArgs A, Spline S) {
  using C = TileCfg<P, TX, TY, NT>;
  extern __shared__ __align__(16) unsigned char gt_smem[];
  TileSmem<P, TX, TY, NT> &sm = *reinterpret_cast<TileSmem<P, TX, TY, NT> *>(gt_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Geom &g = A.g;
  if (__ldg(A.crowd)) return;  // gather_crowded_kernel takes all points
  const int tz = (int)(blockIdx.x % (unsigned)A.nzb), bxy = (int)(blockIdx.x / (unsigned)A.nzb);
  const int x0 = (bxy / A.nty) * TX, y0 = (bxy % A.nty) * TY, z0 = tz * 32;
  const bool near = g.K0 >= C::RX && g.K1 >= C::RY;
  for (int r = tid; r < C::ROWS; r += C::NT) {
    int xi = x0 + r / C::RY + 1 - P / 2, yi = y0 + r % C::RY + 1 - P / 2;
    if (near) {
      xi += xi < 0 ? g.K0 : (xi >= g.K0 ? -g.K0 : 0);
      yi += yi < 0 ? g.K1 : (yi >= g.K1 ? -g.K1 : 0);
    } else {
      xi = imod(xi, g.K0);
      yi = imod(yi, g.K1);
    }
    sm.rowidx[r] = xi * g.K1 + yi;
  }
  // the brick's points: one run of the sorted order per cell row
  int cnt = 0;
  if (tid < C::CELLROWS) {
    const int gx = x0 + tid / TY, gy = y0 + tid % TY;
    if (gx < g.K0 && gy < g.K1) {
      const long b = ((long)gx * g.K1 + gy) * A.nzb + tz;
      if (SPME_IN(b, A.nb, CK_GATHER_ROW)) {
        const int s = __ldg(A.cs + b);
        cnt = __ldg(A.cs + b + 1) - s;
        sm.start[tid] = s;
        if (!SPME_IN(s, A.n + 1, CK_GATHER_ROW) || !SPME_IN(cnt, A.n - s + 1, CK_GATHER_ROW)) cnt = 0;
      }
    }
  }
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) sm.wsum[warp] = incl;
  __syncthreads();
  int wpre = 0, total = 0;
#pragma unroll
  for (int k = 0; k < C::NT / 32; k++) {
    const int v = sm.wsum[k];
    wpre += k < warp ? v : 0;
    total += v;
  }
  if (total == 0) return;  // an empty brick
  if (tid < C::CELLROWS) sm.pref[tid + 1] = wpre + incl;
  if (tid == 0) sm.pref[0] = 0;
  // the grid block in the widest pieces that divide a row (then no piece
  // crosses the periodic boundary)
  if ((g.K2 & 3) == 0) tile_copy<P, TX, TY, NT, 4>(A, sm, z0);
  else if ((g.K2 & 1) == 0) tile_copy<P, TX, TY, NT, 2>(A, sm, z0);
  else tile_copy<P, TX, TY, NT, 1>(A, sm, z0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int c0 = 0; c0 < total; c0 += C::CAP) {
    const int m = min(C::CAP, total - c0);
    if (tid < 32) sm.hist[tid] = 0;
    if (tid == 32) sm.extra = 0;
    __syncthreads();
    int ploc[C::ITEMS], prank[C::ITEMS];
    uint32_t pa[C::ITEMS];
    float4 pr[C::ITEMS];
#pragma unroll
    for (int it = 0; it < C::ITEMS; it++) {
      const int t = tid + it * C::NT;
      prank[it] = -1;
      if (t < m) {
        int lo = 0;  // largest row with pref[row] <= c0 + t
#pragma unroll
        for (int step = C::CELLROWS / 2; step > 0; step >>= 1)
          if (sm.pref[lo + step] <= c0 + t) lo += step;
        const int a = sm.start[lo] + (c0 + t - sm.pref[lo]);
        if (SPME_IN(a, A.n, CK_GATHER_ATOM)) {
          const int rx = lo / TY, ry = lo - rx * TY;
          const int row = sm.rowidx[(rx + P / 2 - 1) * C::RY + ry + P / 2 - 1];
          pr[it] = __ldg(A.rec + a);
          pa[it] = __ldg(A.perm + a);
          if (!SPME_IN(pa[it], A.n, CK_GATHER_ATOM)) pa[it] = 0;
          int zl = (int)(__ldg(A.key + a) - (uint32_t)row * (uint32_t)g.K2) - z0;
          if (!SPME_IN(zl, 32, CK_GATHER_KEY)) zl = 0;
          ploc[it] = (rx * C::RY + ry) * C::PITCH + zl + C::Z0 + 1 - P / 2;
          prank[it] = atomicAdd(&sm.hist[ploc[it] & 31], 1);
        }
      }
    }
    __syncthreads();
    if (warp == 0) {  // places of the ranks: rank r holds the classes with more than r points
      uint32_t m0 = 0, m1 = 0;
#pragma unroll
      for (int c = 0; c < 32; c += 4) {
        const int4 h = *reinterpret_cast<const int4 *>(sm.hist + c);
        m0 |= (h.x > lane ? 1u : 0u) << c | (h.y > lane ? 2u : 0u) << c | (h.z > lane ? 4u : 0u) << c |
              (h.w > lane ? 8u : 0u) << c;
        m1 |= (h.x > lane + 32 ? 1u : 0u) << c | (h.y > lane + 32 ? 2u : 0u) << c |
              (h.z > lane + 32 ? 4u : 0u) << c | (h.w > lane + 32 ? 8u : 0u) << c;
      }
      int s0 = __popc(m0), s1 = __popc(m1);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u0 = __shfl_up_sync(0xffffffffu, s0, o), u1 = __shfl_up_sync(0xffffffffu, s1, o);
        if (lane >= o) {
          s0 += u0;
          s1 += u1;
        }
      }
      const int tot0 = __shfl_sync(0xffffffffu, s0, 31);
      sm.lmask[lane] = m0;
      sm.lmask[lane + 32] = m1;
      sm.lbase[lane + 1] = s0;
      sm.lbase[lane + 33] = tot0 + s1;
      if (lane == 0) sm.lbase[0] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < C::ITEMS; it++) {
      if (prank[it] < 0) continue;
      const int c = ploc[it] & 31;
      const int pos = prank[it] < C::LEVELS
                          ? sm.lbase[prank[it]] + __popc(sm.lmask[prank[it]] & ((1u << c) - 1u))
                          : sm.lbase[C::LEVELS] + atomicAdd(&sm.extra, 1);
      if (SPME_IN(pos, C::CAP, CK_GATHER_ATOM)) {
        sm.list[pos] = make_uint2(pa[it], (uint32_t)ploc[it]);
        sm.rec[pos] = pr[it];
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int p = tid; p < m; p += C::NT) {
      const uint2 e = sm.list[p];
      const float4 u = sm.rec[p];
      const uint32_t a = e.x;
      const double qa = GRAD ? __ldg(A.w + a) : 0.0;
      const float *q = sm.tile + e.y;
      float wx[P], dwx[P], wy[P], dwy[P], wz[P], dwz[P];
#pragma unroll
      for (int i = 0; i < P; i++) {
        dbspl_eval(S, P, 1.f - u.x, i, wx[i], dwx[i]);
        dbspl_eval(S, P, 1.f - u.y, i, wy[i], dwy[i]);
        dbspl_eval(S, P, 1.f - u.z, i, wz[i], dwz[i]);
      }
      // the sums of stencil_sum, term by term in the same order
      float pot = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
      for (int i = 0; i < P; i++) {
        float sy = 0.f, dy = 0.f, dz = 0.f;
#pragma unroll
        for (int j = 0; j < P; j++) {
          float sz = 0.f, dzz = 0.f;
#pragma unroll
          for (int k = 0; k < P; k++) {
            const float v = q[(i * C::RY + j) * C::PITCH + k];
            sz = fmaf(wz[k], v, sz);
            if (GRAD) dzz = fmaf(dwz[k], v, dzz);
          }
          sy = fmaf(wy[j], sz, sy);
          if (GRAD) {
            dy = fmaf(dwy[j], sz, dy);
            dz = fmaf(wy[j], dzz, dz);
          }
        }
        if (POT) pot = fmaf(wx[i], sy, pot);
        if (GRAD) {
          gx = fmaf(dwx[i], sy, gx);
          gy = fmaf(wx[i], dy, gy);
          gz = fmaf(wx[i], dz, gz);
        }
      }
      const CellConst &cc = *g.cell;
      if (GRAD) {
        const double f = -qa * cc.iV;
        const double G0 = (double)gx * f * g.K0, G1 = (double)gy * f * g.K1,
                     G2 = (double)gz * f * g.K2;
        A.dx[3 * (long)a + 0] = cc.iL00 * G0;
        A.dx[3 * (long)a + 1] = cc.iL10 * G0 + cc.iL11 * G1;
        A.dx[3 * (long)a + 2] = cc.iL20 * G0 + cc.iL21 * G1 + cc.iL22 * G2;
      }
      if (POT) A.phi[a] = (double)pot * cc.iV;
    }
    __syncthreads();
  }
}

// After the bricks: zeroes the count words for the next sort (in place of a
// memset, so that it costs no launch more), and in a crowded system takes all
// points, one thread each at a time.
constexpr int kCrowdThreads = 128, kCrowdPerSM = 6;
template <int P, bool GRAD, bool POT>
__global__ void __launch_bounds__(kCrowdThreads, kCrowdPerSM) gather_crowded_kernel(TileArgs A, Spline S, SortedView sv,
                                                                                    ZeroWords zw) {
  zero_words(zw);
  if (!__ldg(A.crowd)) return;
  const Geom &g = A.g;
  const int step = gridDim.x * kCrowdThreads;
  for (long r = (long)blockIdx.x * kCrowdThreads + threadIdx.x; r < A.n; r += step) {
    const CellConst cc = *g.cell;
    const PointAt pt = point_at<P, true>(g, (int)r, A.n, nullptr, sv);
    float pot = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
    point_sums<P>(g, S, A.grid, pt, pot, gx, gy, gz);
    const long a = pt.a;
    if (GRAD) {
      const double f = -A.w[a] * cc.iV;
      const double G0 = (double)gx * f * g.K0, G1 = (double)gy * f * g.K1, G2 = (double)gz * f * g.K2;
      A.dx[3 * a + 0] = cc.iL00 * G0;
      A.dx[3 * a + 1] = cc.iL10 * G0 + cc.iL11 * G1;
      A.dx[3 * a + 2] = cc.iL20 * G0 + cc.iL21 * G1 + cc.iL22 * G2;
    }
    if (POT) A.phi[a] = (double)pot * cc.iV;
  }
}

template <int P, int TX, int TY, int NT, bool GRAD, bool POT>
static void gather_tile_launch(const TileArgs &A, const Spline &S, const SortedView &sv, const ZeroWords &zw,
                               cudaStream_t st) {
  const unsigned blocks = (unsigned)(((A.g.K0 + TX - 1) / TX) * (long)A.nty * A.nzb);
  gather_tile_kernel<P, TX, TY, NT, GRAD, POT><<<blocks, NT, sizeof(TileSmem<P, TX, TY, NT>), st>>>(A, S);
  gather_crowded_kernel<P, GRAD, POT><<<kCrowdPerSM * 148, kCrowdThreads, 0, st>>>(A, S, sv, zw);
}

template <int P, int TX, int TY, int NT>
static void gather_tile_attr() {
  const int bytes = (int)sizeof(TileSmem<P, TX, TY, NT>);
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaFuncSetAttribute(gather_tile_kernel<P, TX, TY, NT, true, true>, attr, bytes);
  cudaFuncSetAttribute(gather_tile_kernel<P, TX, TY, NT, true, false>, attr, bytes);
  cudaFuncSetAttribute(gather_tile_kernel<P, TX, TY, NT, false, true>, attr, bytes);
}

template <int P, int TX, int TY, int NT>
static void gather_tile_t(TileArgs A, const Spline &S, const SortedView &sv, const ZeroWords &zw, cudaStream_t st) {
  A.nty = (A.g.K1 + TY - 1) / TY;
  if (A.dx && A.phi) gather_tile_launch<P, TX, TY, NT, true, true>(A, S, sv, zw, st);
  else if (A.dx) gather_tile_launch<P, TX, TY, NT, true, false>(A, S, sv, zw, st);
  else gather_tile_launch<P, TX, TY, NT, false, true>(A, S, sv, zw, st);
}

// The brick shape: 16 x 8 x 32 cells and 256 threads, 3 CTAs per SM.  A
// smaller brick copies more halo per point and has more unequal classes, a
// larger one leaves fewer CTAs to overlap their copies (1M points, order 6,
// 256^3: 137 us; 8 x 8 with 128 threads 143, 16 x 16 with 256 or 384 threads
// 147 / 145, 16 x 8 with 128 threads 147).
constexpr int kTileX = 16, kTileY = 8, kTileThreads = 256;

static void gather_tile(const TileArgs &A, const Spline &S, const SortedView &sv, const ZeroWords &zw,
                        cudaStream_t st) {
  if (A.g.order == 6) gather_tile_t<6, kTileX, kTileY, kTileThreads>(A, S, sv, zw, st);
  else gather_tile_t<8, kTileX, kTileY, kTileThreads>(A, S, sv, zw, st);
}

// Where bricks are the faster gather (sorted points).  A brick copies its halo
// block and orders its points whatever their number, and one CTA walks through
// them, kTileThreads at a time: with few points per brick the copy is longer
// than the points' own loads, with few bricks the SMs have little to overlap,
// and with many points in few bricks the longest CTA decides.  Evenly filled
// cubic grids, thread per point / bricks, us (mean: points per 4096 cells):
//   order 6   70k 256^3 (mean 16) 38.9 / 80.9   260k 256^3 (63) 85.0 / 89.1
//             195k 200^3 (100) 55.3 / 58.3      274k 224^3 (100) 76.7 / 68.6
//             105k 120^3 (250) 26.7 / 29.7      110k 144^3 (150) 29.7 / 29.7
//             150k 160^3 (150) 43.0 / 35.8      520k 256^3 (127) 118.8 / 97.2
//             1M 256^3 (244) 173.0 / 132.1      1.6M 160^3 (1600) 174.1 / 166.9
//     384 to 767 bricks: 128k 128^3 (a brick 250) 36.9 / 33.8, 169k 120^3 (352)
//             36.9 / 31.7, 205k 128^3 (400) 39.9 / 42.1, 512k 128^3 65.6 / 70.7
//     fewer:  130k 48^3 24.6 / 87.1, 260k 72^3 36.9 / 58.4, 165k 104^3 32.8 / 33.9
//   order 8   66k 256^3 (16) 63.5 / 97.2        82k 224^3 (30) 69.7 / 74.8
//             66k 192^3 (38) 56.3 / 52.2        130k 256^3 (32) 140.3 / 103.4
//             1M 256^3 (244) 347.3 / 207.9      2.1M 176^3 (1600) 405.5 / 357.3
//     384 to 767 bricks: 512k 128^3 (1000) 122.9 / 105.5, 675k 120^3 (1600) 142.3 /
//             117.8, 819k 128^3 (1600) 166.0 / 175.1, 1M 128^3 (1953) 190.5 / 179.2
//     two per SM or fewer: 66k 96^3 (a brick 306) 32.8 / 29.8, 130k 96^3 (602)
//             51.2 / 42.0, 260k 90^3 (1204) 65.6 / 72.7, 130k 48^3 38.9 / 126.0
//     between: 69k 104^3 (189) 34.8 / 37.9, 274k 104^3 (754) 72.7 / 78.8
// Odd rows are copied value by value and need twice the points: order 6, 271k
// 195^3 (150) 70.6 / 72.7, 327k 175^3 (250) 66.5 / 62.5; order 8, 109k 195^3 (60)
// 75.8 / 85.0, 262k 225^3 (94) 163.8 / 132.1.  Order 4: 100k on 96^3 14.3 / 16.4, 1M
// on 200^3 77.8 / 79.9 (not taken).
constexpr int kTileCells = kTileX * kTileY * 32;
constexpr int kTileMinPointsOdd = 262144;
static bool use_tiles(const Geom &g, int n) {
  if (g.order < 6) return false;
  const bool p6 = g.order == 6, odd = g.K2 & 1;
  const double mean = (double)n * kTileCells / ((double)g.K0 * g.K1 * g.K2);
  const long bricks = (long)((g.K0 + kTileX - 1) / kTileX) * ((g.K1 + kTileY - 1) / kTileY) * ((g.K2 + 31) / 32);
  const double per = (double)n / (double)bricks;
  if (n < (odd ? kTileMinPointsOdd : (p6 ? 122880 : 65536))) return false;
  if (mean < (p6 ? (odd ? 200.0 : 96.0) : (odd ? 90.0 : 31.0)) || mean > (p6 ? 1600.0 : 2000.0)) return false;
  if (p6) return bricks >= 768 || (bricks >= 384 && per <= 384.0);
  return bricks >= 384 || (bricks >= 208 && bricks <= 2 * 148 && per <= 640.0);
}

// A brick's CTA takes its points in series, so in a small droplet or a cluster
// the fullest brick takes longer than one thread per point does for the whole
// system.  This is the largest bucket of systems that bricks still serve: the
// one to expect (at 4.5 sigma) where bricks of a dense region hold 512 points
// and one more per 400 of the system, or 1.5 times the mean.  Beyond it the
// solve's gather is one thread per point, decided on the device.  Order 6, cubes
// of a share of the box, thread per point / bricks / this rule, us: 1M on 256^3,
// 0.1 of the box 117.8 / 103.3 / 103.4, 0.03 113.7 / 238.6 / 111.6, 0.001 93.2 / 3125 /
// 101.4; 260k on 192^3, 0.3 50.1 / 50.1 / 48.1, 0.1 44.0 / 60.4 / 44.0; 130k on 128^3,
// 0.3 31.7 / 35.8 / 35.9, 0.1 28.7 / 66.7 / 27.7.  Order 8, 1M on 256^3, 0.1 191.5 /
// 173.0 / 171.2, 0.03 179.2 / 451.6 / 209.9.  (In one kernel, bricks for the first
// points of each bucket and CTAs behind them for the others: 0.3 of 256^3 175.1, 260k
// in 0.1 of 192^3 56.3; the points of full bricks alone one thread each: 72.7 there.)
int gather_crowd_most(const Geom &g, int n) {
  const double mean = (double)n * kTileCells / ((double)g.K0 * g.K1 * g.K2);
  const double bucket = std::max(512.0 + n / 400.0, 1.5 * mean) / (kTileX * kTileY);
  return (int)(bucket + 4.5 * std::sqrt(bucket) + 2.0);
}

bool gather_uses_buckets(const Geom &g, int n, bool dx, bool phi) { return n > 0 && (dx || phi) && use_tiles(g, n); }

void gather_prepare() {
  gather_tile_attr<6, kTileX, kTileY, kTileThreads>();
  gather_tile_attr<8, kTileX, kTileY, kTileThreads>();
}

// Threads per CTA of the thread-per-point kernel: 128 rather than 256 spread
// the CTAs of mid-size systems more evenly over the SMs (solves of 50k points,
// order 8: 98.5 -> 94.3 us; 50k, order 4: 61.6 -> 59.6; 64 threads the same,
// but 4000 points at order 6 55.4 -> 57.5).
constexpr int kGatherThreads = 128;

// Points below which 8 lanes share one (orders 6 and 8).  Solves, thread per
// point / 8 lanes, us: order 6, 500 points 43.1 / 35.0, 4000 55.4 / 49.0, 16k
// 63.6 / 55.6, 32k 73.8 / 68.5, 50k 73.8 / 73.8; order 8, 4000 61.6 / 55.4, 16k
// 69.7 / 65.7, 32k 84.1 / 84.0, 50k 90.2 / 92.4; order 4, 4000 43.1 / 43.1, 16k
// 45.2 / 46.0 (not taken).  Sorted points only: de2 of 24k points in input order
// took 134 us with 8 lanes against 127, its lanes computing the FP64 origin 8 times.
// One line for both orders, where order 8 stops gaining.  A server with 32 such
// requests in flight serves the same number either way (order 6,
// 1000 points 86.8k / 87.5k solves/s, 16k 40.1k / 40.0k).
constexpr int kSplitMaxPoints = 24576;

int gather_route(const Geom &g, int n) {
  if (use_tiles(g, n)) return 2;
  return g.order >= 6 && n <= kSplitMaxPoints ? 1 : 0;
}

template <int P, bool SORTED>
static int gather_p(const Geom &g, const Spline &S, int n, const double *x, const double *w, const float *grid,
                    double *dx, double *phi, double *cellp, const SortedView &sv, cudaStream_t st) {
  if (cellp) {
    gather_kernel<P, true, true, true, SORTED>
        <<<(n + 255) / 256, 256, 0, st>>>(g, S, n, x, w, grid, dx, phi, cellp, sv);
    return 1;
  }
  if constexpr (P >= 6 && SORTED) {
    if (n <= kSplitMaxPoints && (dx || phi)) {
      const int blocks = (n + 15) / 16;
      if (dx && phi)
        gather_split_kernel<P, true, true><<<blocks, 128, 0, st>>>(g, S, n, w, grid, dx, phi, sv);
      else if (dx)
        gather_split_kernel<P, true, false><<<blocks, 128, 0, st>>>(g, S, n, w, grid, dx, phi, sv);
      else
        gather_split_kernel<P, false, true><<<blocks, 128, 0, st>>>(g, S, n, w, grid, dx, phi, sv);
      return 1;
    }
  }
  constexpr int threads = kGatherThreads;
  const int blocks = (n + threads - 1) / threads;
  if (dx && phi)
    gather_kernel<P, true, true, false, SORTED><<<blocks, threads, 0, st>>>(g, S, n, x, w, grid, dx, phi, nullptr, sv);
  else if (dx)
    gather_kernel<P, true, false, false, SORTED><<<blocks, threads, 0, st>>>(g, S, n, x, w, grid, dx, phi, nullptr, sv);
  else if (phi)
    gather_kernel<P, false, true, false, SORTED><<<blocks, threads, 0, st>>>(g, S, n, x, w, grid, dx, phi, nullptr, sv);
  else return 0;
  return 1;
}

template <bool SORTED>
static int gather_any(const Geom &g, const Spline &S, int n, const double *x, const double *w, const float *grid,
                      double *dx, double *phi, double *cellp, const SortedView &sv, cudaStream_t st) {
  switch (g.order) {
    case 2: return gather_p<2, SORTED>(g, S, n, x, w, grid, dx, phi, cellp, sv, st);
    case 4: return gather_p<4, SORTED>(g, S, n, x, w, grid, dx, phi, cellp, sv, st);
    case 6: return gather_p<6, SORTED>(g, S, n, x, w, grid, dx, phi, cellp, sv, st);
    case 8: return gather_p<8, SORTED>(g, S, n, x, w, grid, dx, phi, cellp, sv, st);
    default: return 0;
  }
}

static SortedView make_view(const Geom &g, const uint32_t *perm, const uint32_t *keys, const float4 *rec) {
  SortedView sv{perm, keys, rec, FastDiv((uint32_t)g.K2), FastDiv((uint32_t)g.K1 * (uint32_t)g.K2)};
  return sv;
}

int launch_gather(const Geom &g, const Spline &S, int n, const double *x, const double *w,
                  const float *grid, double *dx, double *phi, cudaStream_t st, const uint32_t *perm,
                  const uint32_t *keys, const float4 *rec, const int *cs, const uint32_t *crowd,
                  const ZeroWords &zw) {
  if (n <= 0 || (!dx && !phi)) return 0;
  if (cs && use_tiles(g, n)) {
    gather_tile(TileArgs{g, cs, perm, keys, rec, w, grid, dx, phi, n, 0, (g.K2 + 31) / 32,
                         sort_buckets(g, kSpreadZShift), crowd},
                S, make_view(g, perm, keys, rec), zw, st);
    return 2;
  }
  if (perm) return gather_any<true>(g, S, n, x, w, grid, dx, phi, nullptr, make_view(g, perm, keys, rec), st);
  return gather_any<false>(g, S, n, x, w, grid, dx, phi, nullptr, SortedView{}, st);
}

// Gather of dE/dx and phi (phi may be null) plus dE/dL; ev must already hold
// the energy and virial of this solve.  cellp: ceil(n/256) x kCellWords.
int launch_gather_cell(const Geom &g, const Spline &S, int n, const double *x, const double *w,
                       const float *grid, double *dx, double *phi, double *cellp, const double *ev, double *dEdL,
                       cudaStream_t st, const uint32_t *perm, const uint32_t *keys, const float4 *rec) {
  int k = 0;
  if (n > 0) {
    if (perm) k = gather_any<true>(g, S, n, x, w, grid, dx, phi, cellp, make_view(g, perm, keys, rec), st);
    else k = gather_any<false>(g, S, n, x, w, grid, dx, phi, cellp, SortedView{}, st);
  }
  cell_grad_kernel<<<1, 9 * 32, 0, st>>>(g, cellp, (n + 255) / 256, ev, dEdL);
  return k + 1;
}

size_t gather_cell_words(int cap) { return (size_t)((cap + 255) / 256 + 1) * kCellWords; }

}  // namespace spme
