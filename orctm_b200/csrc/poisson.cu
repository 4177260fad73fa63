// Matrix-free Poisson solve of the nonhydrostatic pressure correction
// (petsc_solve_3D / ComputeRHS / compute_matrix, mo_petsc.f90:211-397,
// 543-782).
//
// The operator is never assembled: the wet-level counts of a column and its
// four neighbours, the reciprocal metrics and 1D vertical tables give every
// entry of compute_matrix, so the matrix costs next to no HBM traffic.
//
// The solve is iterative refinement: the outer residual r = b - A x is
// accumulated in double-double (error-free FMA products) against the exact
// FP64 matrix entries, and each correction A d = r is solved by
// preconditioned conjugate gradients (FP64, or FP32 for the refined form) on
// the row-scaled operator B = diag(1/ZP) A, whose vertical couplings become
// the symmetric ZW(K) and whose remaining asymmetry is confined to horizontal
// couplings at partial bottom cells.
//
// Red-black reduction.  Columns are coloured by i + j: the horizontal
// couplings C of B join columns of opposite colour only, and what is left, D,
// is one tridiagonal per column.  Eliminating the red columns leaves
//     S = D_b - C_br D_r^-1 C_rb        on the black ones,
// and conjugate gradients on S preconditioned with D_b take half the
// iterations that they take on B preconditioned with D (the two have the same
// spectrum up to lambda -> lambda (2 - lambda)), with vectors of half the
// length.  One iteration is three kernels:
//     red     u = D_r^-1 C_rb z + beta u        (u = D_r^-1 C_rb p)
//     black   x += alpha p ; p = z + beta p ; q = D_b p - C_br u ; p.q
//     column  r -= alpha q ; z = D_b^-1 r ; r.z, r.r
// which move 14 half-length vectors and the pivots: 62 bytes per cell
// in FP64, against 91 for an iteration of the unreduced solver before (and
// twice as many iterations).  Red unknowns are formed from the black ones
// before and after the iterations.
//
// Vectors are stored compactly per colour: column (i, j) at m = i / 2, so both
// colours use offset m + P/2 (j + JN l).  The in-row neighbours of column
// (m, j) are (m - 1 + s, j) and (m + s, j) of the other colour, s = 0 or 1 by
// the parity of the row; north and south are (m, j -+ 1).
//
// A column is shared by G lanes of a warp, each with LC consecutive levels in
// registers (a warp holds 32/G columns: 32-byte segments of a level's row).
// The tridiagonal recurrences run level by level inside a lane and as a scan
// of affine maps across the column's lanes, so the whole column is loaded at
// once and nothing is spilled.  A thread that marches down a column alone
// waits a memory latency every few levels: 27 us against 5 per launch on the
// 512 x 1 x 60 slice, and 0.62 of the copy bandwidth on 1024 x 1024 x 80.
//
// Dot products are reduced deterministically: every tile writes a partial sum
// and the last block to finish (atomic ticket) adds the partials in tile
// order and updates the solver scalars on the device, so an iteration
// needs no host round trip, and totals do not depend on the launch shape.  A
// device flag marks convergence; kernels of an already converged solve return
// at once.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "ops.h"

namespace orctm {

namespace {

#define AT(a, i, j, K) (a)[G.L.at((i), (j), (K)-1)]

inline dim3 grid2(int nx, int ny, dim3 b) { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y, 1); }

// ------------------------------------------------------- coefficients ----
struct Coef {
  double dc, w, e, n, s, u, d;  // diagonal, west, east, north, south, up, down
};

// 2D data of one column (i, j), i in [2, IE-1], j in [2, JE-1]
struct ColC {
  int ij;
  int kb, kbw, kbe, kbn, kbs;
  int kreg;                            // levels 2..kreg have the regular (all-wet) row
  bool iw, ie, in, is;                 // couplings the DMDA allows (not at the domain edge)
  double cw, ce, cn, cs, xcf, ycf;     // XU(I-1)XP, XU(I)XP, YV(J-1)YP, YV(J)YP, sums
  double zwa, zwb, zpa, zpb, zpc, iza, izb, izc;
};

__device__ __forceinline__ ColC load_col(const Geo& G, const PoissonGeo& P, int i, int j) {
  ColC c;
  const int IE = G.L.ie, JE = G.L.je;
  c.ij = G.L.at2(i, j);
  c.kb = G.gp.kb[c.ij];
  c.kbw = G.gp.kb[G.L.at2(i - 1, j)];
  c.kbe = G.gp.kb[G.L.at2(i + 1, j)];
  c.kbn = G.gp.kb[G.L.at2(i, j - 1)];
  c.kbs = G.gp.kb[G.L.at2(i, j + 1)];
  c.iw = i > 2;
  c.ie = i < IE - 1;
  c.in = j > 2;
  c.is = j < JE - 1;
  const double xuw = P.xu[G.L.at2(i - 1, j)], xue = P.xu[c.ij], xp = P.xp[c.ij];
  const double yvn = P.yv[G.L.at2(i, j - 1)], yvs = P.yv[c.ij], yp = P.yp[c.ij];
  c.cw = xuw * xp;
  c.ce = xue * xp;
  c.cn = yvn * yp;
  c.cs = yvs * yp;
  c.xcf = (xuw + xue) * xp;
  c.ycf = (yvn + yvs) * yp;
  c.zwa = P.zwa[c.ij]; c.zwb = P.zwb[c.ij];
  c.zpa = P.zpa[c.ij]; c.zpb = P.zpb[c.ij]; c.zpc = P.zpc[c.ij];
  c.iza = P.iza[c.ij]; c.izb = P.izb[c.ij]; c.izc = P.izc[c.ij];
  // below kreg every neighbour is wet and ZW/ZP are the 1D tables: K < kb - 1
  // keeps K, K+1 and the ZP selections away from the bottom specials
  const int km = min(min(c.kbw, c.kbe), min(c.kbn, c.kbs));
  c.kreg = min(km, c.kb - 2);
  return c;
}

__device__ __forceinline__ double zw_of(const ColC& c, const PoissonGeo& P, int K) {
  if (c.kb >= 1) {
    if (K == c.kb) return c.zwa;
    if (K == c.kb + 1) return c.zwb;
  }
  return P.zwn[K - 1];
}
__device__ __forceinline__ double zp_of(const ColC& c, const PoissonGeo& P, int K) {
  if (c.kb >= 1) {
    if (K == c.kb - 1) return c.zpa;
    if (K == c.kb) return c.zpb;
    if (K == c.kb + 1) return c.zpc;
  }
  return P.zpn[K - 1];
}
__device__ __forceinline__ double izp_of(const ColC& c, const PoissonGeo& P, int K) {
  if (c.kb >= 1) {
    if (K == c.kb - 1) return c.iza;
    if (K == c.kb) return c.izb;
    if (K == c.kb + 1) return c.izc;
  }
  return P.izn[K - 1];
}

// Row K of compute_matrix (mo_petsc.f90:607-767) for the column, entries the
// reference does not insert returned as 0.  With SCALED the row of
// B = diag(1/ZP) A: vertical entries ZW(K), ZW(K+1); horizontal entries and
// X_C, Y_C multiplied by 1/ZP.
template <bool SCALED>
__device__ __forceinline__ Coef row(const ColC& c, const PoissonGeo& P, int K, int KE) {
  const double zw0 = zw_of(c, P, K), zw1 = zw_of(c, P, K + 1);
  const double zp = SCALED ? 1.0 : zp_of(c, P, K);
  const double hs = SCALED ? izp_of(c, P, K) : 1.0;
  Coef r;
  double X_C = c.xcf, Y_C = c.ycf, Z_C = (zw0 + zw1) * zp;
  r.w = r.e = r.n = r.s = r.u = r.d = 0.0;
  if (K > c.kb) {  // land row: diagonal only
    r.dc = SCALED ? -((X_C + Y_C) * hs + Z_C) : -(X_C + Y_C + Z_C);
    return r;
  }
  const bool ww = K <= c.kbw, we = K <= c.kbe, wn = K <= c.kbn, ws = K <= c.kbs;
  if (!ww && we) X_C = c.ce;
  else if (ww && !we) X_C = c.cw;
  else if (!ww && !we) X_C = 0.0;
  if (!wn && ws) Y_C = c.cs;
  else if (wn && !ws) Y_C = c.cn;
  else if (!wn && !ws) Y_C = 0.0;
  const bool wd = K + 1 <= c.kb;
  if (K == 1) {
  } else if (K == KE || !wd) {
    Z_C = zw0 * zp;
  }
  r.dc = SCALED ? -((X_C + Y_C) * hs + Z_C) : -(X_C + Y_C + Z_C);
  if (c.iw && ww) r.w = c.cw * hs;
  if (c.ie && we) r.e = c.ce * hs;
  if (c.in && wn) r.n = c.cn * hs;
  if (c.is && ws) r.s = c.cs * hs;
  if (K != 1) r.u = zw0 * zp;
  if (K != KE && wd) r.d = zw1 * zp;
  return r;
}

// ------------------------------------------------------- reductions ------
// Partial sums of one tile: the block's threads are added in a fixed order.
constexpr int kThreads = 256, kWarps = kThreads / 32;

template <int NV>
__device__ __forceinline__ void tile_partial(const double (&v)[NV], SolverState* S, int tile) {
  __shared__ double sh[NV][kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double x = v[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[q][warp] = x;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double x = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) x += sh[threadIdx.x][w];
    S->partials[(size_t)threadIdx.x * S->max_blocks + tile] = x;
  }
  __syncthreads();
}

// After a block's last tile: true in thread 0 of the last block to get here,
// which then holds the totals over all tiles in v.
template <int NV>
__device__ bool grid_total(double (&v)[NV], SolverState* S, int ntiles) {
  __shared__ double sh[NV][kWarps];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < NV) __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&S->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const double* part = S->partials + (size_t)q * S->max_blocks;
    double x = 0.0;
#pragma unroll 8
    for (int b = tid; b < ntiles; b += kThreads) x += __ldcg(part + b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[q][warp] = x;
  }
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double x = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) x += sh[q][w];
      v[q] = x;
    }
    S->ticket = 0;
  }
  return tid == 0;
}

// ------------------------------------------------------- set-up ---------
__device__ __forceinline__ int red_i(int m, int j) { return 2 * m + (j & 1); }
__device__ __forceinline__ int black_i(int m, int j) { return 2 * m + 1 - (j & 1); }

// Pivots of the column tridiagonal of B (constant): dinv(K) = 1/d'(K) with
// d'(1) = d(1), d'(K) = d(K) - a(K) c(K-1) / d'(K-1), per colour in the
// compact layout: the red ones in FP64 and FP32 (the elimination is exact to
// the solve's precision), the black ones, a fixed preconditioner, in FP32 for
// both forms; and the 2D data of the columns.  Columns that are no unknowns
// keep kk = 0 (no wet level).
__global__ void k_rb_setup(Geo G, PoissonGeo P, RbGeo R, double* __restrict__ dr64,
                           float* __restrict__ dr32, float* __restrict__ db32) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int KE = G.L.ke;
  if (i > G.L.ie - 1 || j > G.L.je - 1) return;
  const ColC c = load_col(G, P, i, j);
  const bool black = (i + j) & 1;
  const RbColour& q = R.col[black];
  const int s = (i >> 1) + R.P2 * j;
  q.kk[s] = (unsigned long long)c.kb | (unsigned long long)c.kbw << 10 |
            (unsigned long long)c.kbe << 20 | (unsigned long long)c.kbn << 30 |
            (unsigned long long)c.kbs << 40;
  q.we[s] = make_double2(c.cw, c.ce);
  q.ns[s] = make_double2(c.cn, c.cs);
  q.zw[s] = make_double2(c.zwa, c.zwb);
  q.iz[s] = make_double2(c.iza, c.izb);
  double dprev = 1.0, cprev = 0.0;
  for (int K = 1; K <= c.kb; ++K) {
    const Coef r = row<true>(c, P, K, KE);
    const double d = K == 1 ? r.dc : r.dc - (r.u * dprev) * cprev;
    const double di = 1.0 / d;
    const int o = s + R.plane2 * (K - 1);
    if (black) {
      db32[o] = (float)di;
    } else {
      dr64[o] = di;
      dr32[o] = (float)di;
    }
    dprev = di;
    cprev = r.d;
  }
}

// ------------------------------------------------------- PCG kernels -----
// Where a thread stands: G lanes per column, LC levels per lane.
template <typename T, int G, int LC>
struct Lane {
  static constexpr int CW = 32 / G;          // columns per warp
  static constexpr int CT = kWarps * CW;     // columns per tile
  static constexpr int TAB = G * (LC + 1) + 1;
  int m, g, K0, tab;                         // column, lane in it, first level - 1, its table entry
  __device__ __forceinline__ Lane() {
    const int lane = threadIdx.x & 31;
    g = lane / CW;
    m = (threadIdx.x >> 5) * CW + lane % CW;
    K0 = g * LC;
    tab = g * (LC + 1);
  }
};

// ZW(K) at szw[e + e / LC], e = K - 1 = 0..KE, and 1/ZP(K) alike: the lanes
// of a column read LC + 1 entries apart (no bank conflicts).
template <typename T, int G, int LC>
__device__ __forceinline__ void load_tables(const RbGeo& R, T* szw, T* siz) {
  for (int e = threadIdx.x; e <= G * LC; e += kThreads) {
    szw[e + e / LC] = e <= R.ke ? (T)R.zwn[e] : T(0);
    if (siz) siz[e + e / LC] = e < R.ke ? (T)R.izn[e] : T(0);
  }
  __syncthreads();
}

// Couplings a(K) between levels K - 1 and K of the lane's levels and of the one
// below its last: ZW(K) inside the column (its own value at the bottom),
// 0 at the surface and below the bottom.
template <typename T, int G, int LC>
__device__ __forceinline__ void couplings(const Lane<T, G, LC>& t, const T* szw, int kb, T zwa,
                                          T (&a)[LC + 1]) {
#pragma unroll
  for (int u = 0; u <= LC; ++u) {
    const int K = t.K0 + 1 + u;
    const T zw = szw[t.tab + u + (u == LC)];
    a[u] = (K == 1 || K > kb) ? T(0) : (K == kb ? zwa : zw);
  }
}

// v <- M^-1 v for the column tridiagonal M = L D L^T with pivots 1/d and
// couplings a; returns v.M^-1 v = sum y^2 / d of this lane's levels.
template <typename T, int G, int LC>
__device__ __forceinline__ T column_solve(const Lane<T, G, LC>& t, T (&v)[LC], const T (&d)[LC],
                                          const T (&a)[LC + 1]) {
  constexpr int CW = 32 / G;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // forward: y(K) = v(K) - a(K) d(K-1) y(K-1); the lane's levels as one affine
  // map y_out = A y_in + B, scanned over the lanes above
  const T dm = __shfl_up_sync(kAll, d[LC - 1], CW);
  T A = T(1), B = T(0);
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    const T l = -(a[u] * (u ? d[u - 1] : dm));
    B = fma(l, B, v[u]);
    A = l * A;
  }
#pragma unroll
  for (int o = CW; o < 32; o <<= 1) {
    const T Ap = __shfl_up_sync(kAll, A, o), Bp = __shfl_up_sync(kAll, B, o);
    if (lane >= o) {
      B = fma(A, Bp, B);
      A *= Ap;
    }
  }
  T y = __shfl_up_sync(kAll, B, CW);
  if (t.g == 0) y = T(0);
  T rz = T(0);
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    y = fma(-(a[u] * (u ? d[u - 1] : dm)), y, v[u]);
    v[u] = y * d[u];
    rz = fma(y, v[u], rz);
  }
  // backward: z(K) = y(K) d(K) - a(K+1) d(K) z(K+1)
  A = T(1);
  B = T(0);
#pragma unroll
  for (int u = LC - 1; u >= 0; --u) {
    const T l = -(a[u + 1] * d[u]);
    B = fma(l, B, v[u]);
    A = l * A;
  }
#pragma unroll
  for (int o = CW; o < 32; o <<= 1) {
    const T Ap = __shfl_down_sync(kAll, A, o), Bp = __shfl_down_sync(kAll, B, o);
    if (lane + o < 32) {
      B = fma(A, Bp, B);
      A *= Ap;
    }
  }
  T z = __shfl_down_sync(kAll, B, CW);
  if (t.g == G - 1) z = T(0);
#pragma unroll
  for (int u = LC - 1; u >= 0; --u) {
    z = fma(-(a[u + 1] * d[u]), z, v[u]);
    v[u] = z;
  }
  return rz;
}

__device__ __forceinline__ int wet_levels(unsigned long long kk, int nb) {
  return (int)((kk >> (10 * nb)) & 1023u);
}

// Red columns.
//   kIter    u = D^-1 C v + beta u          (v = z; u is not read while beta = 0)
//   kBefore  u = D^-1 (b / ZP)              (b: full layout, scaled); sum of (b / ZP)^2
//   kAfter   x += scale (u - D^-1 C v)      (v = the black correction; x: full layout)
enum { kIter = 0, kBefore = 1, kAfter = 2 };

template <typename T, int G, int LC, int MODE>
__global__ void __launch_bounds__(kThreads) k_rb_red(RbGeo R, SolverState* S,
                                                     const T* __restrict__ v, T* __restrict__ u,
                                                     const T* __restrict__ dinv,
                                                     const double* __restrict__ b,
                                                     double* __restrict__ x, int ntiles, int nmc) {
  using Ln = Lane<T, G, LC>;
  __shared__ T szw[Ln::TAB], siz[Ln::TAB];
  if (MODE == kIter && S->converged) return;
  const T beta = MODE == kIter ? (T)S->beta : T(0);
  double scale = 1.0;
  if (MODE != kIter && sizeof(T) == 4) {
    scale = sqrt(S->res_rr);
    if (MODE == kBefore) scale = scale > 0.0 ? 1.0 / scale : 0.0;
  }
  load_tables<T, G, LC>(R, szw, siz);
  const Ln t;
  const unsigned P2 = (unsigned)R.P2, plane = (unsigned)R.plane2;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int j = 2 + tile / nmc, m = (tile % nmc) * Ln::CT + t.m;
    const unsigned s2 = (unsigned)m + P2 * (unsigned)j;
    unsigned long long kk = 0;
    if (m < R.M) kk = R.col[0].kk[s2];
    const int kb = wet_levels(kk, 0);
    T cw = 0, ce = 0, cn = 0, cs = 0, zwa = 0;
    double iza = 0, izb = 0;
    if (kb) {
      const double2 we = R.col[0].we[s2], ns = R.col[0].ns[s2], iz = R.col[0].iz[s2];
      cw = (T)we.x; ce = (T)we.y; cn = (T)ns.x; cs = (T)ns.y;
      zwa = (T)R.col[0].zw[s2].x;
      iza = iz.x; izb = iz.y;
    }
    const unsigned o0 = s2 + plane * (unsigned)t.K0;
    const unsigned ow = o0 - 1u + (unsigned)(j & 1);
    T g[LC], d[LC], a[LC + 1];
    couplings<T, G, LC>(t, szw, kb, zwa, a);
    double bb = 0.0;
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      const int K = t.K0 + 1 + q;
      const unsigned l = plane * (unsigned)q;
      g[q] = d[q] = T(0);
      if (K <= kb) {
        d[q] = dinv[o0 + l];
        if (MODE == kBefore) {
          const double hs = K == kb ? izb : (K == kb - 1 ? iza : R.izn[K - 1]);
          const unsigned f = (unsigned)red_i(m, j) + 2u * P2 * (unsigned)j + 2u * plane * (unsigned)(K - 1);
          g[q] = (T)((b[f] * scale) * hs);
          bb = fma((double)g[q], (double)g[q], bb);
        } else {
          // values of land cells and outside the unknowns are exact zeros
          const T hs = K == kb ? (T)izb : (K == kb - 1 ? (T)iza : siz[t.tab + q]);
          T h = cw * v[ow + l];
          h = fma(ce, v[ow + l + 1u], h);
          h = fma(cn, v[o0 + l - P2], h);
          h = fma(cs, v[o0 + l + P2], h);
          g[q] = hs * h;
        }
      }
    }
    column_solve<T, G, LC>(t, g, d, a);
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      const int K = t.K0 + 1 + q;
      const unsigned o = o0 + plane * (unsigned)q;
      if (K <= kb) {
        if (MODE == kIter) {
          u[o] = beta == T(0) ? g[q] : fma(beta, u[o], g[q]);
        } else if (MODE == kBefore) {
          u[o] = g[q];
        } else {
          const unsigned f = (unsigned)red_i(m, j) + 2u * P2 * (unsigned)j + 2u * plane * (unsigned)(K - 1);
          x[f] = x[f] + scale * (double)(u[o] - g[q]);
        }
      }
    }
    if (MODE == kBefore) {
      const double w[1] = {bb};
      tile_partial<1>(w, S, tile);
    }
  }
  if (MODE == kBefore) {
    double w[1];
    if (grid_total<1>(w, S, ntiles)) S->bb = w[0];
  }
}

// Black columns: x += alpha p (the previous step's), p = z + beta p,
// q = D p - C u, and alpha = rho / p.q.  The first iteration (iter = 0) reads
// neither p nor x.
template <typename T, int G, int LC>
__global__ void __launch_bounds__(kThreads) k_rb_black(RbGeo R, SolverState* S,
                                                       const T* __restrict__ z,
                                                       const T* __restrict__ u, T* __restrict__ p,
                                                       T* __restrict__ x, T* __restrict__ q,
                                                       int ntiles, int nmc) {
  using Ln = Lane<T, G, LC>;
  __shared__ T szw[Ln::TAB], siz[Ln::TAB];
  if (S->converged) return;
  const T beta = (T)S->beta, alpha = (T)S->alpha_prev;
  const bool first = S->iter == 0;
  load_tables<T, G, LC>(R, szw, siz);
  const Ln t;
  const unsigned P2 = (unsigned)R.P2, plane = (unsigned)R.plane2;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int j = 2 + tile / nmc, m = (tile % nmc) * Ln::CT + t.m;
    const unsigned s2 = (unsigned)m + P2 * (unsigned)j;
    unsigned long long kk = 0;
    if (m < R.M) kk = R.col[1].kk[s2];
    const int kb = wet_levels(kk, 0);
    const int kbw = wet_levels(kk, 1), kbe = wet_levels(kk, 2);
    const int kbn = wet_levels(kk, 3), kbs = wet_levels(kk, 4);
    T cw = 0, ce = 0, cn = 0, cs = 0, zwa = 0, zwb = 0, iza = 0, izb = 0;
    if (kb) {
      const double2 we = R.col[1].we[s2], ns = R.col[1].ns[s2], iz = R.col[1].iz[s2],
                    zw = R.col[1].zw[s2];
      cw = (T)we.x; ce = (T)we.y; cn = (T)ns.x; cs = (T)ns.y;
      zwa = (T)zw.x; zwb = (T)zw.y;
      iza = (T)iz.x; izb = (T)iz.y;
    }
    const unsigned o0 = s2 + plane * (unsigned)t.K0;
    const unsigned ow = o0 - (unsigned)(j & 1);
    T pl[LC];
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      const unsigned o = o0 + plane * (unsigned)e;
      pl[e] = T(0);
      if (t.K0 + 1 + e <= kb) {
        T pn = z[o];
        if (first) {
          x[o] = T(0);
        } else {
          const T po = p[o];
          x[o] = fma(alpha, po, x[o]);
          pn = fma(beta, po, pn);
        }
        p[o] = pn;
        pl[e] = pn;
      }
    }
    T pu = __shfl_up_sync(0xffffffffu, pl[LC - 1], Ln::CW);
    T pb = __shfl_down_sync(0xffffffffu, pl[0], Ln::CW);
    if (t.g == 0) pu = T(0);
    if (t.g == G - 1) pb = T(0);
    T pq = T(0);
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      const int K = t.K0 + 1 + e;
      if (K <= kb) {
        const unsigned o = o0 + plane * (unsigned)e, w = ow + plane * (unsigned)e;
        const T p0 = pl[e], pd = e + 1 < LC ? pl[e + 1] : pb;
        T dh = K <= kbw ? cw : T(0);
        if (K <= kbe) dh += ce;
        if (K <= kbn) dh += cn;
        if (K <= kbs) dh += cs;
        T h = cw * u[w];
        h = fma(ce, u[w + 1u], h);
        h = fma(cn, u[o - P2], h);
        h = fma(cs, u[o + P2], h);
        h = fma(dh, p0, h);
        const T hs = K == kb ? izb : (K == kb - 1 ? iza : siz[t.tab + e]);
        const T zw0 = K == kb ? zwa : szw[t.tab + e];
        const T zw1 = K + 1 == kb ? zwa : szw[t.tab + e + 1 + (e + 1 == LC)];
        T s = zw0 * (pu - p0);
        if (K < kb) s = fma(zw1, pd - p0, s);
        else if (K == 1) s = fma(-zwb, p0, s);  // Z_C of the surface row keeps ZW(2)
        s = fma(-hs, h, s);
        q[o] = s;
        pq = fma(p0, s, pq);
      }
      pu = pl[e];
    }
    const double w[1] = {(double)pq};
    tile_partial<1>(w, S, tile);
  }
  double w[1];
  if (grid_total<1>(w, S, ntiles)) {
    S->pq = w[0];
    S->alpha = S->rho / w[0];
    if (!(w[0] > 0.0) && !(w[0] < 0.0)) S->converged = 3;  // breakdown
  }
}

// Black columns: residual, z = D_b^-1 r with the FP32 pivots, r.z and r.r.
//   INIT   r = b / ZP - C u     (u = D_r^-1 (b / ZP) of the red columns)
//   else   r -= alpha q
template <typename T, int G, int LC, bool INIT>
__global__ void __launch_bounds__(kThreads) k_rb_col(RbGeo R, SolverState* S, T* __restrict__ r,
                                                     const T* __restrict__ q, T* __restrict__ z,
                                                     const float* __restrict__ dinv,
                                                     const double* __restrict__ b,
                                                     const T* __restrict__ ub, int ntiles,
                                                     int nmc) {
  using Ln = Lane<T, G, LC>;
  __shared__ T szw[Ln::TAB];
  if (!INIT && S->converged) return;
  const T alpha = INIT ? T(0) : (T)S->alpha;
  double scale = 1.0;
  if (INIT && sizeof(T) == 4) scale = S->res_rr > 0.0 ? 1.0 / sqrt(S->res_rr) : 0.0;
  load_tables<T, G, LC>(R, szw, nullptr);
  const Ln t;
  const unsigned P2 = (unsigned)R.P2, plane = (unsigned)R.plane2;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int j = 2 + tile / nmc, m = (tile % nmc) * Ln::CT + t.m;
    const unsigned s2 = (unsigned)m + P2 * (unsigned)j;
    unsigned long long kk = 0;
    if (m < R.M) kk = R.col[1].kk[s2];
    const int kb = wet_levels(kk, 0);
    const T zwa = kb ? (T)R.col[1].zw[s2].x : T(0);
    const unsigned o0 = s2 + plane * (unsigned)t.K0;
    T g[LC], d[LC], a[LC + 1], rr = T(0);
    double bb = 0.0;
    couplings<T, G, LC>(t, szw, kb, zwa, a);
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      const int K = t.K0 + 1 + e;
      const unsigned o = o0 + plane * (unsigned)e;
      g[e] = d[e] = T(0);
      if (K <= kb) {
        d[e] = (T)dinv[o];
        if (INIT) {
          const double2 we = R.col[1].we[s2], ns = R.col[1].ns[s2], iz = R.col[1].iz[s2];
          const double hs = K == kb ? iz.y : (K == kb - 1 ? iz.x : R.izn[K - 1]);
          const unsigned f = (unsigned)black_i(m, j) + 2u * P2 * (unsigned)j + 2u * plane * (unsigned)(K - 1);
          const unsigned w = o - (unsigned)(j & 1);
          const T bs = (T)((b[f] * scale) * hs);
          T h = (T)we.x * ub[w];
          h = fma((T)we.y, ub[w + 1u], h);
          h = fma((T)ns.x, ub[o - P2], h);
          h = fma((T)ns.y, ub[o + P2], h);
          bb = fma((double)bs, (double)bs, bb);
          g[e] = fma(-(T)hs, h, bs);
        } else {
          g[e] = fma(-alpha, q[o], r[o]);
        }
        r[o] = g[e];
        rr = fma(g[e], g[e], rr);
      }
    }
    const T rz = column_solve<T, G, LC>(t, g, d, a);
#pragma unroll
    for (int e = 0; e < LC; ++e)
      if (t.K0 + 1 + e <= kb) z[o0 + plane * (unsigned)e] = g[e];
    if (INIT) {
      const double w[3] = {(double)rz, (double)rr, bb};
      tile_partial<3>(w, S, tile);
    } else {
      const double w[2] = {(double)rz, (double)rr};
      tile_partial<2>(w, S, tile);
    }
  }
  double v[INIT ? 3 : 2];
  if (grid_total<INIT ? 3 : 2>(v, S, ntiles)) {
    if (INIT) {
      S->bb += v[2];  // the red columns' part is there already
      S->beta = 0.0;
      S->alpha_prev = 0.0;
    } else {
      S->beta = v[0] / S->rho;
      S->alpha_prev = S->alpha;
      S->iter += 1;
    }
    S->rho = v[0];
    S->rr = v[1];
    if (sqrt(v[1]) <= S->tol * sqrt(S->bb) || S->bb == 0.0) S->converged = 1;
    if (!(v[0] == v[0]) || !(v[1] == v[1])) S->converged = 2;  // NaN: stop
  }
}

// The black correction: the x update that the last iteration left open (none
// before the first), and its addition to the solution (full layout).
template <typename T>
__global__ void __launch_bounds__(kThreads) k_rb_after(RbGeo R, SolverState* S,
                                                       const T* __restrict__ p, T* __restrict__ d,
                                                       double* __restrict__ x) {
  const int m = blockIdx.x * 32 + (threadIdx.x & 31), K = blockIdx.z * kWarps + (threadIdx.x >> 5) + 1;
  const int j = blockIdx.y + 2;
  if (m >= R.M) return;
  const int s2 = m + R.P2 * j;
  if (K > wet_levels(R.col[1].kk[s2], 0)) return;
  const int o = s2 + R.plane2 * (K - 1);
  T v = T(0);
  if (S->iter > 0) v = fma((T)S->alpha_prev, p[o], d[o]);
  d[o] = v;
  const double scale = sizeof(T) == 4 ? sqrt(S->res_rr) : 1.0;
  const int f = black_i(m, j) + 2 * (R.P2 * j + R.plane2 * (K - 1));
  x[f] = x[f] + scale * (double)v;
}

// r = b - A x with the exact FP64 entries of compute_matrix, accumulated in
// double-double (products split exactly with an FMA), then rounded once; and
// ||r||^2, ||b||^2.  This is the outer residual of the refinement loop and
// the reported residual.
struct DD {
  double hi, lo;
};
__device__ __forceinline__ void dd_sub_prod(DD& s, double c, double x) {
  const double p = c * x;
  const double pe = __fma_rn(c, x, -p);  // c*x = p + pe exactly
  const double t = s.hi - p;             // two-sum of s.hi and -p
  const double bv = t - s.hi;
  const double e = (s.hi - (t - bv)) + (-p - bv);
  const double lo = s.lo + e - pe;
  const double hi = t + lo;
  s.lo = lo - (hi - t);
  s.hi = hi;
}

// LR levels per thread: the levels of a column are independent here, so the
// blocks split them (a thread that marches down a whole column waits for its
// loads level by level: 1.4 ms a launch on 1024 x 1024 x 80).
constexpr int kResidLevels = 8;

__global__ void __launch_bounds__(kThreads) k_resid(Geo G, PoissonGeo P, SolverState* S,
                                                    const double* __restrict__ b,
                                                    double* __restrict__ x,
                                                    double* __restrict__ r, int nbx, int nby,
                                                    int ntiles) {
  const int KE = G.L.ke, IE = G.L.ie, JE = G.L.je;
  const int tile = blockIdx.x, bx = tile % nbx, by = (tile / nbx) % nby, bz = tile / (nbx * nby);
  const int i = bx * 32 + (threadIdx.x & 31) + 2, j = by * kWarps + (threadIdx.x >> 5) + 2;
  const int K0 = bz * kResidLevels + 1, K1 = min(KE, K0 + kResidLevels - 1);
  double rr = 0.0, bb = 0.0;
  if (i <= IE - 1 && j <= JE - 1) {
    const ColC c = load_col(G, P, i, j);
    // land rows (K > kb): diagonal only with a zero right-hand side, so the
    // solution there is 0 and x is set to it; r is neither stored nor read there
    for (int K = max(c.kb + 1, K0); K <= K1; ++K)
      if (AT(x, i, j, K) != 0.0) AT(x, i, j, K) = 0.0;
    double xm = 0.0, x0 = 0.0, xp = 0.0;
    if (K0 <= c.kb) {
      if (K0 > 1) xm = AT(x, i, j, K0 - 1);
      x0 = AT(x, i, j, K0);
    }
    const int Ke = min(K1, c.kb);
    for (int K = K0; K <= Ke; ++K) {
      xp = K < c.kb ? AT(x, i, j, K + 1) : 0.0;
      const Coef rw = row<false>(c, P, K, KE);
      const double bk = AT(b, i, j, K);
      DD s{bk, 0.0};
      if (rw.u != 0.0) dd_sub_prod(s, rw.u, xm);
      if (rw.n != 0.0) dd_sub_prod(s, rw.n, AT(x, i, j - 1, K));
      if (rw.w != 0.0) dd_sub_prod(s, rw.w, AT(x, i - 1, j, K));
      dd_sub_prod(s, rw.dc, x0);
      if (rw.e != 0.0) dd_sub_prod(s, rw.e, AT(x, i + 1, j, K));
      if (rw.s != 0.0) dd_sub_prod(s, rw.s, AT(x, i, j + 1, K));
      if (rw.d != 0.0) dd_sub_prod(s, rw.d, xp);
      const double rk = s.hi + s.lo;
      AT(r, i, j, K) = rk;
      rr += rk * rk;
      bb += bk * bk;
      xm = x0;
      x0 = xp;
    }
  }
  const double w[2] = {rr, bb};
  tile_partial<2>(w, S, tile);
  double v[2];
  if (grid_total<2>(v, S, ntiles)) {
    S->res_rr = v[0];
    S->res_bb = v[1];
  }
}

__global__ void k_set_limit(SolverState* S, int limit) { S->limit = limit; }

// the last node of the device-side PCG loop's body
__global__ void k_pcg_continue(cudaGraphConditionalHandle hc, const SolverState* S, int chunk) {
  cudaGraphSetConditional(hc, (S->converged == 0 && S->iter + chunk <= S->limit) ? 1u : 0u);
}

__global__ void k_reset(SolverState* S, double tol) {
  S->converged = 0;
  S->iter = 0;
  S->ticket = 0;
  S->tol = tol;
  S->beta = 0.0;
  S->alpha_prev = 0.0;
  S->bb = 0.0;
}

// Launch shapes: at most this many blocks per SM (a block then walks several
// tiles), 0 for a block per tile.
constexpr int kShapes = 9;
const int kBlocksPerSm[kShapes] = {0, 2, 3, 4, 6, 8, 1, 5, 12};

struct Shape {
  int ntiles, nmc, grid;
};

Shape shape_of(const RbGeo& R, int columns_per_tile, int variant) {
  Shape s;
  s.nmc = (R.M + columns_per_tile - 1) / columns_per_tile;
  s.ntiles = s.nmc * (R.je - 2);
  s.grid = s.ntiles;
  const int per = kBlocksPerSm[variant >= 0 && variant < kShapes ? variant : 0];
  if (per) s.grid = std::min(s.ntiles, per * R.sms);
  return s;
}

// Calls f<T, G, LC> with the split for KE levels: four columns of doubles or
// eight of floats per warp (32-byte segments) while the lane's share fits
// registers (up to 13 doubles or 26 floats), 16 lanes per column above.
template <int N>
using Int = std::integral_constant<int, N>;

template <typename T, typename F>
void with_split(int ke, F&& f) {
  if (ke > 104) {
    if (ke <= 128) f(Int<16>{}, Int<8>{});
    else if (ke <= 208) f(Int<16>{}, Int<13>{});
    else f(Int<16>{}, Int<20>{});
  } else if constexpr (sizeof(T) == 8) {
    if (ke <= 40) f(Int<8>{}, Int<5>{});
    else if (ke <= 48) f(Int<8>{}, Int<6>{});
    else if (ke <= 64) f(Int<8>{}, Int<8>{});
    else if (ke <= 80) f(Int<8>{}, Int<10>{});
    else if (ke <= 88) f(Int<8>{}, Int<11>{});
    else f(Int<8>{}, Int<13>{});
  } else {
    if (ke <= 40) f(Int<4>{}, Int<10>{});
    else if (ke <= 48) f(Int<4>{}, Int<12>{});
    else if (ke <= 64) f(Int<4>{}, Int<16>{});
    else if (ke <= 80) f(Int<4>{}, Int<20>{});
    else if (ke <= 88) f(Int<4>{}, Int<22>{});
    else f(Int<4>{}, Int<26>{});
  }
}
static_assert(16 * 20 >= kMaxKe, "the longest column has a split");

template <typename T>
const T* red_pivots(const RbGeo& R);
template <>
const double* red_pivots<double>(const RbGeo& R) { return R.dr64; }
template <>
const float* red_pivots<float>(const RbGeo& R) { return R.dr32; }

}  // namespace

void launch_rb_setup(const Geo& G, const PoissonGeo& P, const RbGeo& R, double* dr64, float* dr32,
                     float* db32, cudaStream_t st) {
  const dim3 blk(32, 4);
  k_rb_setup<<<grid2(G.L.ie - 2, G.L.je - 2, blk), blk, 0, st>>>(G, P, R, dr64, dr32, db32);
  count_launch();
}

int pcg_col_variants() { return 6; }
int pcg_spmv_variants() { return kShapes; }

template <typename T>
void launch_rb_before(const RbGeo& R, SolverState* S, const double* b, const RbVectors<T>& v,
                      cudaStream_t st) {
  with_split<T>(R.ke, [&](auto gc, auto lc) {
    constexpr int G = decltype(gc)::value, LC = decltype(lc)::value;
    const Shape s = shape_of(R, Lane<T, G, LC>::CT, 0);
    k_rb_red<T, G, LC, kBefore><<<s.grid, kThreads, 0, st>>>(R, S, nullptr, v.ub, red_pivots<T>(R),
                                                             b, nullptr, s.ntiles, s.nmc);
    k_rb_col<T, G, LC, true><<<s.grid, kThreads, 0, st>>>(R, S, v.r, nullptr, v.z, R.db32, b, v.ub,
                                                          s.ntiles, s.nmc);
  });
  add_launches(2);
}

template <typename T>
void launch_rb_red(const RbGeo& R, SolverState* S, const RbVectors<T>& v, int variant,
                   cudaStream_t st) {
  with_split<T>(R.ke, [&](auto gc, auto lc) {
    constexpr int G = decltype(gc)::value, LC = decltype(lc)::value;
    const Shape s = shape_of(R, Lane<T, G, LC>::CT, variant);
    k_rb_red<T, G, LC, kIter><<<s.grid, kThreads, 0, st>>>(R, S, v.z, v.u, red_pivots<T>(R), nullptr,
                                                           nullptr, s.ntiles, s.nmc);
  });
  count_launch();
}

template <typename T>
void launch_rb_black(const RbGeo& R, SolverState* S, const RbVectors<T>& v, int variant,
                     cudaStream_t st) {
  with_split<T>(R.ke, [&](auto gc, auto lc) {
    constexpr int G = decltype(gc)::value, LC = decltype(lc)::value;
    const Shape s = shape_of(R, Lane<T, G, LC>::CT, variant);
    k_rb_black<T, G, LC><<<s.grid, kThreads, 0, st>>>(R, S, v.z, v.u, v.p, v.x, v.q, s.ntiles, s.nmc);
  });
  count_launch();
}

template <typename T>
void launch_rb_col(const RbGeo& R, SolverState* S, const RbVectors<T>& v, int variant,
                   cudaStream_t st) {
  with_split<T>(R.ke, [&](auto gc, auto lc) {
    constexpr int G = decltype(gc)::value, LC = decltype(lc)::value;
    const Shape s = shape_of(R, Lane<T, G, LC>::CT, variant);
    k_rb_col<T, G, LC, false><<<s.grid, kThreads, 0, st>>>(R, S, v.r, v.q, v.z, R.db32, nullptr,
                                                           nullptr, s.ntiles, s.nmc);
  });
  count_launch();
}

template <typename T>
void launch_rb_after(const RbGeo& R, SolverState* S, const RbVectors<T>& v, double* x,
                     cudaStream_t st) {
  const dim3 grid((R.M + 31) / 32, R.je - 2, (R.ke + kWarps - 1) / kWarps);
  k_rb_after<T><<<grid, kThreads, 0, st>>>(R, S, v.p, v.x, x);
  with_split<T>(R.ke, [&](auto gc, auto lc) {
    constexpr int G = decltype(gc)::value, LC = decltype(lc)::value;
    const Shape s = shape_of(R, Lane<T, G, LC>::CT, 0);
    k_rb_red<T, G, LC, kAfter><<<s.grid, kThreads, 0, st>>>(R, S, v.x, v.ub, red_pivots<T>(R),
                                                            nullptr, x, s.ntiles, s.nmc);
  });
  add_launches(2);
}

#define ORCTM_RB(T)                                                                              \
  template void launch_rb_before<T>(const RbGeo&, SolverState*, const double*, const RbVectors<T>&, \
                                    cudaStream_t);                                               \
  template void launch_rb_red<T>(const RbGeo&, SolverState*, const RbVectors<T>&, int, cudaStream_t); \
  template void launch_rb_black<T>(const RbGeo&, SolverState*, const RbVectors<T>&, int, cudaStream_t); \
  template void launch_rb_col<T>(const RbGeo&, SolverState*, const RbVectors<T>&, int, cudaStream_t); \
  template void launch_rb_after<T>(const RbGeo&, SolverState*, const RbVectors<T>&, double*, cudaStream_t);
ORCTM_RB(double)
ORCTM_RB(float)
#undef ORCTM_RB

void launch_resid(const Geo& G, const PoissonGeo& P, SolverState* S, const double* b, double* x,
                  double* r, cudaStream_t st) {
  const int nbx = (G.L.ie - 2 + 31) / 32, nby = (G.L.je - 2 + kWarps - 1) / kWarps;
  const int nt = nbx * nby * ((G.L.ke + kResidLevels - 1) / kResidLevels);
  k_resid<<<nt, kThreads, 0, st>>>(G, P, S, b, x, r, nbx, nby, nt);
  count_launch();
}

void launch_solver_reset(SolverState* S, double tol, cudaStream_t st) {
  k_reset<<<1, 1, 0, st>>>(S, tol);
  count_launch();
}

void launch_set_limit(SolverState* S, int limit, cudaStream_t st) {
  k_set_limit<<<1, 1, 0, st>>>(S, limit);
  count_launch();
}

void launch_pcg_continue(cudaGraphConditionalHandle hc, const SolverState* S, int chunk,
                         cudaStream_t st) {
  k_pcg_continue<<<1, 1, 0, st>>>(hc, S, chunk);
  count_launch();
}

size_t solver_max_blocks(const Geo& G) {
  // tiles of k_resid, and of the PCG kernels at their narrowest (16 columns)
  const size_t resid = (size_t)((G.L.ie - 2 + 31) / 32) * ((G.L.je - 2 + kWarps - 1) / kWarps) *
                       ((G.L.ke + kResidLevels - 1) / kResidLevels);
  const size_t pcg = (size_t)((G.L.ie / 2 + 1 + 15) / 16) * (G.L.je - 2);
  return std::max(resid, pcg);
}

}  // namespace orctm
