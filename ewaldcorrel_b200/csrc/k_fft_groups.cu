// FFT passes by groups of Stockham stages, for lengths without an n1 n2 split
// into two register transforms of at most 16 (125, 162, 200, 216, 243, 250 and
// so on) and for the z/y passes beside such a length.
//
// The radix stages of the shared-memory engine (fft_engine.cuh) are taken in
// two groups, each run in registers: stages 1..s by the n2 tasks j2, which
// hold the elements j2 + n2 m (m < n1), stages s+1.. by the n1 tasks k1, which
// hold the elements k1 + n1 j2 of the first group's result.  n1 and n2 are the
// products of the groups' radices, one exchange lies between them, and every
// stage multiplies by the same table entries and runs the same butterfly as
// the engine's, so the results have the same bits.  The engine took one
// shared-memory round trip, a barrier and an index computation per stage: the
// FFT passes of a solve on 216^3 took 596 us with it and take 311 (200^3 481 ->
// 268, 243^3 840 -> 412, 162^3 295 -> 167, 125^3 132 -> 128).
#include <type_traits>

#include "fft_engine.cuh"
#include "influence.cuh"

namespace spme {

SPME_CHECK_READER(fft_groups)

template <int... R>
struct Radices {
  static constexpr int N = (R * ... * 1);
};

// Stage of radix R with NsL as the product of the group's earlier radices.
// FIRST: the group begins the transform (Ns0 = 1, k0 = 0), S = n2; else Ns0 =
// n1, k0 = the task's k1, S = 1.  Twiddle index of input r: r k n / (Ns R)
// with k = k0 + Ns0 (j mod NsL), Ns = Ns0 NsL.
template <int SIGN, bool FIRST, int N, int NsL>
__device__ __forceinline__ void group_stages(float2 (&)[N], const float2 *, int, int, int, int) {}
template <int SIGN, bool FIRST, int N, int NsL, int R, int... Rest>
__device__ __forceinline__ void group_stages(float2 (&v)[N], const float2 *tw, int n, int k0, int Ns0, int S) {
  constexpr int m = N / R;
  const int st = S * (N / (NsL * R));
  float2 o[N];
#pragma unroll
  for (int j = 0; j < m; j++) {
    const int q = j / NsL, kl = j % NsL;
    const int k = k0 + Ns0 * kl;
    float2 t[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      t[r] = v[j + r * m];
      if (r > 0 && !(FIRST && NsL == 1)) t[r] = cmul(t[r], twid<SIGN>(tw, r * k * st));
    }
    Bfly<R, SIGN>::run(t, tw, n);
#pragma unroll
    for (int r = 0; r < R; r++) o[q * NsL * R + kl + r * NsL] = t[r];
  }
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = o[i];
  group_stages<SIGN, FIRST, N, NsL * R, Rest...>(v, tw, n, k0, Ns0, S);
}
template <int SIGN, bool FIRST, int... R>
__device__ __forceinline__ void group_run(Radices<R...>, float2 (&v)[Radices<R...>::N], const float2 *tw, int n, int k0,
                                          int Ns0, int S) {
  group_stages<SIGN, FIRST, Radices<R...>::N, 1, R...>(v, tw, n, k0, Ns0, S);
}

// The groups with a compiled form; ids index kGroups.
constexpr int kGroupCount = 16, kGroupStages = 3;
static const int kGroups[kGroupCount][kGroupStages] = {
    {3, 0, 0}, {4, 0, 0}, {5, 0, 0}, {7, 0, 0}, {2, 3, 0}, {4, 2, 0}, {3, 3, 0}, {2, 5, 0}, {4, 3, 0},
    {3, 5, 0}, {4, 4, 0}, {2, 3, 3}, {4, 5, 0}, {3, 7, 0}, {5, 5, 0}, {3, 3, 3}};
template <class F>
__device__ __forceinline__ void with_group(int id, F &&f) {
  switch (id) {
    case 0: f(Radices<3>{}); break;
    case 1: f(Radices<4>{}); break;
    case 2: f(Radices<5>{}); break;
    case 3: f(Radices<7>{}); break;
    case 4: f(Radices<2, 3>{}); break;
    case 5: f(Radices<4, 2>{}); break;
    case 6: f(Radices<3, 3>{}); break;
    case 7: f(Radices<2, 5>{}); break;
    case 8: f(Radices<4, 3>{}); break;
    case 9: f(Radices<3, 5>{}); break;
    case 10: f(Radices<4, 4>{}); break;
    case 11: f(Radices<2, 3, 3>{}); break;
    case 12: f(Radices<4, 5>{}); break;
    case 13: f(Radices<3, 7>{}); break;
    case 14: f(Radices<5, 5>{}); break;
    case 15: f(Radices<3, 3, 3>{}); break;
    default: break;
  }
}

static int group_id(const int *rad, int count) {
  if (count < 1 || count > kGroupStages) return -1;
  for (int g = 0; g < kGroupCount; g++) {
    bool same = true;
    for (int i = 0; i < kGroupStages; i++) same = same && kGroups[g][i] == (i < count ? rad[i] : 0);
    if (same) return g;
  }
  return -1;
}

// Splits a length's stages into two compiled groups with the smallest larger
// factor; false when there is none.
bool fft_group_split(const FftLen &L, FftGroups &G) {
  bool found = false;
  for (int s = 1; s < L.nst; s++) {
    const int a = group_id(L.rad, s), b = group_id(L.rad + s, L.nst - s);
    if (a < 0 || b < 0) continue;
    int n1 = 1;
    for (int i = 0; i < s; i++) n1 *= L.rad[i];
    const int n2 = L.n / n1, big = n1 > n2 ? n1 : n2;
    if (found && big >= (G.n1 > G.n2 ? G.n1 : G.n2)) continue;
    G = FftGroups{L.n, n1, n2, a, b, L.tw};
    found = true;
  }
  return found;
}

__device__ __forceinline__ void load_tw(float2 *tw, const FftGroups &F) {
  for (int i = threadIdx.x; i < F.n; i += blockDim.x) tw[i] = F.tw[i];
}

// z passes: one line, row[2b] + i row[2b+1], per G lanes (8, 16 or 32, the
// power of two that holds both factors), as the two-level z passes.  Rows are
// paired within planes of rpp rows (lpp lines each), the last row of an odd
// plane alone.
constexpr int kGzWarps = 4;

template <int G>
__global__ void __launch_bounds__(32 * kGzWarps) fft_gz_r2c_kernel(FftGroups F, const float *__restrict__ rin,
                                                                   float2 *__restrict__ cout, int nlines, int rpp,
                                                                   FastDiv lpp, ZeroWords zw) {
  zero_words(zw);
  extern __shared__ float2 sm[];
  constexpr int LW = 32 / G;
  const int n = F.n, n1 = F.n1, n2 = F.n2, ldim = n / 2 + 1, ep = n2 | 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & (G - 1);
  const int line = (blockIdx.x * (blockDim.x >> 5) + warp) * LW + lane / G;
  float2 *tw = sm, *ex = sm + n + (warp * LW + lane / G) * n1 * ep;
  uint32_t pl, pr;  // line pr of the plane pl
  lpp.divmod((uint32_t)min(line, nlines - 1), pl, pr);
  const int ra = (int)pl * rpp + 2 * (int)pr;
  const bool va = line < nlines, vb = va && 2 * (int)pr + 1 < rpp;  // the rows there are
  const bool la = va && t < n2, lb = vb && t < n2;
  const float *pa = rin + (long)ra * n + t, *pb = pa + n;
  load_tw(tw, F);
  with_group(F.g1, [&](auto RL) {
    constexpr int N = decltype(RL)::N;
    float2 u[N];
#pragma unroll
    for (int m = 0; m < N; m++) {
      u[m].x = la && SPME_IN(t + n2 * m, n, CK_FFT_LINE) ? __ldg(pa + n2 * m) : 0.f;
      u[m].y = lb && SPME_IN(t + n2 * m, n, CK_FFT_LINE) ? __ldg(pb + n2 * m) : 0.f;
    }
    __syncthreads();
    if (t < n2) {
      group_run<-1, true>(RL, u, tw, n, 0, 1, n2);
#pragma unroll
      for (int k1 = 0; k1 < N; k1++) ex[k1 * ep + t] = u[k1];
    }
  });
  __syncwarp();
  const int t1 = min(t, n1 - 1);
  const int mirror = lane - t + (t1 == 0 ? 0 : n1 - t1);
  with_group(F.g2, [&](auto RL) {
    constexpr int N = decltype(RL)::N;
    float2 w[N];
#pragma unroll
    for (int j2 = 0; j2 < N; j2++) w[j2] = ex[t1 * ep + j2];
    group_run<-1, false>(RL, w, tw, n, t1, n1, 1);
#pragma unroll
    for (int k2 = 0; k2 <= N / 2; k2++) {
      float2 v;
      v.x = __shfl_sync(0xffffffffu, w[N - 1 - k2].x, mirror);
      v.y = __shfl_sync(0xffffffffu, w[N - 1 - k2].y, mirror);
      if (t1 == 0) v = w[(N - k2) % N];
      const float2 u = w[k2];
      const int k = t + n1 * k2;
      if (t < n1 && k < ldim) {
        if (va) cout[(long)ra * ldim + k] = make_float2(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));
        if (vb) cout[(long)(ra + 1) * ldim + k] = make_float2(0.5f * (u.y + v.y), -0.5f * (u.x - v.x));
      }
    }
  });
}

template <int G>
__global__ void __launch_bounds__(32 * kGzWarps) fft_gz_c2r_kernel(FftGroups F, const float2 *__restrict__ cin,
                                                                   float *__restrict__ rout, int nlines, int rpp,
                                                                   FastDiv lpp) {
  extern __shared__ float2 sm[];
  constexpr int LW = 32 / G;
  const int n = F.n, n1 = F.n1, n2 = F.n2, ldim = n / 2 + 1, ep = n2 | 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & (G - 1);
  const int line = (blockIdx.x * (blockDim.x >> 5) + warp) * LW + lane / G;
  float2 *tw = sm, *ex = sm + n + (warp * LW + lane / G) * n1 * ep;
  uint32_t pl, pr;  // line pr of the plane pl
  lpp.divmod((uint32_t)min(line, nlines - 1), pl, pr);
  const int ra = (int)pl * rpp + 2 * (int)pr;
  const bool va = line < nlines, vb = va && 2 * (int)pr + 1 < rpp;  // the rows there are
  const bool la = va && t < n2, lb = vb && t < n2;
  const float2 *pa = cin + (long)ra * ldim, *pb = pa + ldim;
  load_tw(tw, F);
  with_group(F.g1, [&](auto RL) {
    constexpr int N = decltype(RL)::N;
    float2 u[N];
#pragma unroll
    for (int m = 0; m < N; m++) {
      const int k = t + n2 * m;
      const bool lo = k < ldim;
      const int kk = lo ? k : n - k;
      float2 a = make_float2(0.f, 0.f), c = make_float2(0.f, 0.f);
      if (la && SPME_IN(kk, ldim, CK_FFT_LINE)) a = __ldg(pa + kk);
      if (lb && SPME_IN(kk, ldim, CK_FFT_LINE)) c = __ldg(pb + kk);
      if (kk == 0 || 2 * kk == n) {
        a.y = 0.f;
        c.y = 0.f;
      }
      u[m] = lo ? make_float2(a.x - c.y, a.y + c.x) : make_float2(a.x + c.y, c.x - a.y);
    }
    __syncthreads();
    if (t < n2) {
      group_run<+1, true>(RL, u, tw, n, 0, 1, n2);
#pragma unroll
      for (int k1 = 0; k1 < N; k1++) ex[k1 * ep + t] = u[k1];
    }
  });
  __syncwarp();
  if (t >= n1) return;
  with_group(F.g2, [&](auto RL) {
    constexpr int N = decltype(RL)::N;
    float2 w[N];
#pragma unroll
    for (int j2 = 0; j2 < N; j2++) w[j2] = ex[t * ep + j2];
    group_run<+1, false>(RL, w, tw, n, t, n1, 1);
    float *qa = rout + (long)ra * n + t, *qb = qa + n;
#pragma unroll
    for (int k2 = 0; k2 < N; k2++) {
      if (va && SPME_IN(t + n1 * k2, n, CK_FFT_LINE)) qa[n1 * k2] = w[k2].x;
      if (vb && SPME_IN(t + n1 * k2, n, CK_FFT_LINE)) qb[n1 * k2] = w[k2].y;
    }
  });
}

// Lines along y of every x-plane, B = 2^lgB per CTA, b fastest in the thread
// index; with `partials`, CTA 0 (one more than the lines need) reduces the
// energy/virial partials of the preceding x pass.
template <int SIGN>
__global__ void __launch_bounds__(512) fft_gy_kernel(FftGroups F, float2 *__restrict__ data, int nlines, FastDiv lpp,
                                                     long pstride, int es, int lgB,
                                                     const double *__restrict__ partials, int nblocks,
                                                     const CellConst *__restrict__ cell, double *__restrict__ raw,
                                                     double *__restrict__ ev) {
  if (partials && blockIdx.x == 0) {
    finish_partials(partials, nblocks, cell, raw, ev);
    return;
  }
  extern __shared__ float2 sm[];
  const int n = F.n, n1 = F.n1, n2 = F.n2, B = 1 << lgB;
  float2 *tw = sm, *ex = sm + n;
  load_tw(tw, F);
  const int b = threadIdx.x & (B - 1), t = threadIdx.x >> lgB;
  const int l = (int)(blockIdx.x - (partials ? 1 : 0)) * B + b;
  const bool live = l < nlines;
  uint32_t pl = 0, r = 0;
  if (live) lpp.divmod((uint32_t)l, pl, r);
  float2 *p = data + (long)pl * pstride + r;
  __syncthreads();
  if (t < n2)
    with_group(F.g1, [&](auto RL) {
      constexpr int N = decltype(RL)::N;
      float2 u[N];
#pragma unroll
      for (int m = 0; m < N; m++)
        u[m] = live && SPME_IN(t + n2 * m, n, CK_FFT_LINE) ? p[(long)(t + n2 * m) * es] : make_float2(0.f, 0.f);
      group_run<SIGN, true>(RL, u, tw, n, 0, 1, n2);
#pragma unroll
      for (int k1 = 0; k1 < N; k1++) ex[(k1 * n2 + t) * B + b] = u[k1];
    });
  __syncthreads();
  if (t < n1 && live)
    with_group(F.g2, [&](auto RL) {
      constexpr int N = decltype(RL)::N;
      float2 w[N];
#pragma unroll
      for (int j2 = 0; j2 < N; j2++) w[j2] = ex[(t * n2 + j2) * B + b];
      group_run<SIGN, false>(RL, w, tw, n, t, n1, 1);
#pragma unroll
      for (int k2 = 0; k2 < N; k2++)
        if (SPME_IN(t + n1 * k2, n, CK_FFT_LINE)) p[(long)(t + n1 * k2) * es] = w[k2];
    });
}

// x pass with the pointwise reciprocal step: the modes and results of
// fft_x_kernel (k_fft.cu).  The inverse transform begins from natural order
// like the forward one, so it takes an exchange of its own before it.
template <int MODE, int IM>
__global__ void __launch_bounds__(512) fft_gx_kernel(FftGroups F, Geom g, Influence inf, const double *__restrict__ iB0,
                                                     const double *__restrict__ iB1, const double *__restrict__ iB2,
                                                     float2 *__restrict__ data, int lgB,
                                                     double *__restrict__ partials, FastDiv ldd) {
  extern __shared__ float2 sm[];
  __shared__ double red[16][7];
  const int n = F.n, n1 = F.n1, n2 = F.n2, B = 1 << lgB;
  float2 *tw = sm, *ex = sm + n;
  load_tw(tw, F);
  const int nlines = g.K1 * g.ldim;
  const int b = threadIdx.x & (B - 1), t = threadIdx.x >> lgB;
  const int line = blockIdx.x * B + b;
  const bool live = line < nlines;
  uint32_t uy = 0, uz = 0;
  if (live) ldd.divmod((uint32_t)line, uy, uz);
  const int ky = (int)uy, kz = (int)uz;
  constexpr bool FWD = (MODE == XM_FWD_DECONV || MODE == XM_FWD_CONV_INV);
  __syncthreads();
  if (FWD) {
    if (t < n2)
      with_group(F.g1, [&](auto RL) {
        constexpr int N = decltype(RL)::N;
        float2 u[N];
#pragma unroll
        for (int m = 0; m < N; m++)
          u[m] = live && SPME_IN(t + n2 * m, n, CK_FFT_LINE) ? data[line + (t + n2 * m) * nlines]
                                                             : make_float2(0.f, 0.f);
        group_run<-1, true>(RL, u, tw, n, 0, 1, n2);
#pragma unroll
        for (int k1 = 0; k1 < N; k1++) ex[(k1 * n2 + t) * B + b] = u[k1];
      });
    __syncthreads();
    with_group(F.g2, [&](auto RL) {
      constexpr int N = decltype(RL)::N;
      float2 w[N];
      if (t < n1) {
#pragma unroll
        for (int j2 = 0; j2 < N; j2++) w[j2] = ex[(t * n2 + j2) * B + b];
        group_run<-1, false>(RL, w, tw, n, t, n1, 1);
      }
      __syncthreads();  // every task has read its inputs
      if (t < n1)
#pragma unroll
        for (int k2 = 0; k2 < N; k2++) ex[(t + n1 * k2) * B + b] = w[k2];  // natural order
    });
    __syncthreads();
  }
  double acc[7];
#pragma unroll
  for (int c = 0; c < 7; c++) acc[c] = 0.0;
  // the pointwise step by all threads: thread (t, b) takes the modes t, t + T,
  // ... of line b, kAhead influence entries read ahead of their use
  if (live) {
    const int T = blockDim.x >> lgB;
    const bool plane = (kz == 0) || ((g.K2 & 1) == 0 && kz == g.ldim - 1);
    const InfConst ic = load_ic(inf);
    const double s12 = iB1[ky] * iB2[kz];
    constexpr int kAhead = 4;
    for (int k0 = t; k0 < n; k0 += kAhead * T) {
      double packed[kAhead];
      float2 in[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; u++) {
        const int kx = k0 + u * T;
        packed[u] = (IM == 4 && MODE != XM_FWD_DECONV && kx < n) ? inf.A[kx * nlines + line] : 0.0;
        if (!FWD) in[u] = kx < n ? data[line + kx * nlines] : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < kAhead; u++) {
        const int kx = k0 + u * T;
        if (kx >= n) break;
        const int i = SPME_IN(kx * nlines + line, n * nlines, CK_FFT_CONV) ? kx * nlines + line : 0;
        float2 &slot = ex[kx * B + b];
        const float2 q = FWD ? slot : in[u];
        if (MODE == XM_FWD_DECONV) {
          data[i] = cscale(q, (float)(iB0[kx] * s12));
          continue;
        }
        const double ib = iB0[kx] * s12;
        double sq = (double)q.x * q.x + (double)q.y * q.y;
        if (MODE == XM_FWD_CONV_INV) sq *= ib * ib;  // |F iB|^2
        double A;
        if constexpr (IM == 4) A = compact_acc(inf, ic, g, i, kx, ky, kz, plane, sq, packed[u], acc);
        else A = influence_acc<IM>(inf, ic, g, i, kx, ky, kz, plane, sq, acc);
        if (MODE != XM_EN) {
          double f = A * ib * (MODE == XM_FWD_CONV_INV ? ib : 1.0);
          if (plane) f *= 2.0;
          slot = cscale(q, (float)f);
        }
      }
    }
  }
  if (MODE == XM_FWD_DECONV) return;
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 7; c++) {
      const double v = warp_sum(acc[c]);
      if (lane == 0) red[warp][c] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += red[w][threadIdx.x];
    partials[(long)blockIdx.x * kRedWords + threadIdx.x] = v;
  }
  if (MODE == XM_EN) return;
  with_group(F.g1, [&](auto RL) {
    constexpr int N = decltype(RL)::N;  // n1
    float2 u[N];
    if (t < n2)
#pragma unroll
      for (int m = 0; m < N; m++) {
        u[m] = ex[(t + n2 * m) * B + b];
      }
    __syncthreads();
    if (t < n2) {
      group_run<+1, true>(RL, u, tw, n, 0, 1, n2);
#pragma unroll
      for (int k1 = 0; k1 < N; k1++) ex[(k1 * n2 + t) * B + b] = u[k1];
    }
  });
  __syncthreads();
  if (t < n1 && live)
    with_group(F.g2, [&](auto RL) {
      constexpr int N = decltype(RL)::N;
      float2 w[N];
#pragma unroll
      for (int j2 = 0; j2 < N; j2++) w[j2] = ex[(t * n2 + j2) * B + b];
      group_run<+1, false>(RL, w, tw, n, t, n1, 1);
#pragma unroll
      for (int k2 = 0; k2 < N; k2++)
        if (SPME_IN(t + n1 * k2, n, CK_FFT_LINE)) data[line + (t + n1 * k2) * nlines] = w[k2];
    });
}

void fft_groups_prepare() {
  const int lim = 200 * 1024;
  const void *f[] = {(const void *)fft_gx_kernel<XM_FWD_DECONV, 1>,   (const void *)fft_gx_kernel<XM_CONV_INV, 1>,
                     (const void *)fft_gx_kernel<XM_CONV_INV, 2>,     (const void *)fft_gx_kernel<XM_CONV_INV, 4>,
                     (const void *)fft_gx_kernel<XM_FWD_CONV_INV, 1>, (const void *)fft_gx_kernel<XM_FWD_CONV_INV, 2>,
                     (const void *)fft_gx_kernel<XM_FWD_CONV_INV, 4>, (const void *)fft_gx_kernel<XM_EN, 1>,
                     (const void *)fft_gx_kernel<XM_EN, 2>,           (const void *)fft_gx_kernel<XM_EN, 4>,
                     (const void *)fft_gy_kernel<-1>,                 (const void *)fft_gy_kernel<+1>,
                     (const void *)fft_gz_r2c_kernel<8>,              (const void *)fft_gz_r2c_kernel<16>,
                     (const void *)fft_gz_r2c_kernel<32>,             (const void *)fft_gz_c2r_kernel<8>,
                     (const void *)fft_gz_c2r_kernel<16>,             (const void *)fft_gz_c2r_kernel<32>};
  for (const void *k : f) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
}

template <bool FWD>
static void launch_gz(const FftGroups &F, float *real, float2 *cplx, int planes, int rpp, const ZeroWords &zw,
                      cudaStream_t st) {
  const int m = F.n1 > F.n2 ? F.n1 : F.n2;
  const int G = m <= 8 ? 8 : (m <= 16 ? 16 : 32), lw = 32 / G;
  const int lines = planes * ((rpp + 1) / 2);
  const FastDiv lpp((uint32_t)((rpp + 1) / 2));
  const long warps = ((long)lines + lw - 1) / lw;
  int wpc = kGzWarps;
  while (wpc > 1 && warps < 148L * wpc) wpc >>= 1;
  const size_t smem = (size_t)(F.n + wpc * lw * F.n1 * (F.n2 | 1)) * sizeof(float2);
  const unsigned blocks = (unsigned)((warps + wpc - 1) / wpc);
  auto go = [&](auto GC) {
    constexpr int GG = decltype(GC)::value;
    if (FWD) fft_gz_r2c_kernel<GG><<<blocks, 32 * wpc, smem, st>>>(F, real, cplx, lines, rpp, lpp, zw);
    else fft_gz_c2r_kernel<GG><<<blocks, 32 * wpc, smem, st>>>(F, cplx, real, lines, rpp, lpp);
  };
  if (G == 8) go(std::integral_constant<int, 8>{});
  else if (G == 16) go(std::integral_constant<int, 16>{});
  else go(std::integral_constant<int, 32>{});
}
void launch_groups_z(const FftGroups &F, bool forward, float *real, float2 *cplx, int planes, int rpp,
                     const ZeroWords &zw, cudaStream_t st) {
  if (forward) launch_gz<true>(F, real, cplx, planes, rpp, zw, st);
  else launch_gz<false>(F, real, cplx, planes, rpp, zw, st);
}

// Lines per CTA (8 to 32): CTAs of at least 128 (y) or 256 (x) threads, at
// most 512, halved while the SMs would not all get two (one).
static int group_lines(const FftGroups &F, long nlines, int min_threads, int per_sm, int &threads) {
  const int m = F.n1 > F.n2 ? F.n1 : F.n2;
  int lgB = 3;
  while (lgB < 5 && (m << lgB) < min_threads) lgB++;
  while (lgB > 3 && ((nlines >> lgB) < 148L * per_sm || (m << lgB) > 512)) lgB--;
  threads = ((m << lgB) + 31) / 32 * 32;
  return lgB;
}

void launch_groups_y(const FftGroups &F, bool forward, const Geom &g, float2 *cplx, const double *partials, int nblocks,
                     double *raw, double *ev, cudaStream_t st) {
  const long nl = (long)g.K0 * g.ldim;
  int threads;
  const int lgB = group_lines(F, nl, 128, 2, threads);
  const size_t smem = (size_t)(F.n + (F.n << lgB)) * sizeof(float2);
  const unsigned blocks = (unsigned)((nl + (1 << lgB) - 1) >> lgB) + (partials ? 1 : 0);
  const FastDiv lpp((uint32_t)g.ldim);
  if (forward)
    fft_gy_kernel<-1><<<blocks, threads, smem, st>>>(F, cplx, (int)nl, lpp, (long)g.K1 * g.ldim, g.ldim, lgB, nullptr, 0,
                                                     nullptr, nullptr, nullptr);
  else
    fft_gy_kernel<+1><<<blocks, threads, smem, st>>>(F, cplx, (int)nl, lpp, (long)g.K1 * g.ldim, g.ldim, lgB, partials,
                                                     nblocks, g.cell, raw, ev);
}

template <int MODE>
static void launch_gx(const FftGroups &F, const Geom &g, const Influence &inf, const double *iB0, const double *iB1,
                      const double *iB2, float2 *cplx, double *partials, int &nblocks, cudaStream_t st) {
  const long nl = (long)g.K1 * g.ldim;
  int threads;
  const int lgB = group_lines(F, nl, 256, 1, threads);
  const size_t smem = (size_t)(F.n + (F.n << lgB)) * sizeof(float2);
  nblocks = (int)((nl + (1 << lgB) - 1) >> lgB);
  auto go = [&](auto IMC) {
    fft_gx_kernel<MODE, decltype(IMC)::value><<<nblocks, threads, smem, st>>>(F, g, inf, iB0, iB1, iB2, cplx, lgB,
                                                                              partials, FastDiv((uint32_t)g.ldim));
  };
  if (MODE == XM_FWD_DECONV || inf.mode == 1) go(std::integral_constant<int, 1>{});
  else if (inf.mode == 4) go(std::integral_constant<int, 4>{});
  else go(std::integral_constant<int, 2>{});
}
void launch_groups_x(const FftGroups &F, int mode, const Geom &g, const Influence &inf, const double *iB0,
                     const double *iB1, const double *iB2, float2 *cplx, double *partials, int &nblocks,
                     cudaStream_t st) {
  switch (mode) {
    case XM_FWD_DECONV: launch_gx<XM_FWD_DECONV>(F, g, inf, iB0, iB1, iB2, cplx, partials, nblocks, st); break;
    case XM_CONV_INV: launch_gx<XM_CONV_INV>(F, g, inf, iB0, iB1, iB2, cplx, partials, nblocks, st); break;
    case XM_FWD_CONV_INV: launch_gx<XM_FWD_CONV_INV>(F, g, inf, iB0, iB1, iB2, cplx, partials, nblocks, st); break;
    default: launch_gx<XM_EN>(F, g, inf, iB0, iB1, iB2, cplx, partials, nblocks, st); break;
  }
}

}  // namespace spme
