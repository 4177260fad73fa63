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
// length.  One iteration is three kernels (and on planes a fourth, the coarse
// correction of z, below):
//     red     u = D_r^-1 C_rb z + beta u        (u = D_r^-1 C_rb p)
//     black   x += alpha p ; p = z + beta p ; q = D_b p - C_br u ; p.q
//     column  r -= alpha q ; z = D_b^-1 r ; r.z, r.r
// which move 14 half-length vectors and the pivots: 62 bytes per cell
// in FP64, against 91 for an iteration of the unreduced solver before (and
// twice as many iterations).  Red unknowns are formed from the black ones
// before and after the iterations.
//
// Vectors are stored per colour, column (i, j) at m = i / 2 of row j, in tiles
// of W columns (128 bytes of a level) that hold all their levels one after
// the other: offset ((j NT + b) KE + l) W + c, b W + c = m - 1.  A tile is some 10 KB
// of consecutive memory; in the padded layout of the model's fields its levels lie
// megabytes apart on 1024 x 1024 x 80, where every block then touched some 80
// pages per vector (the operator's kernel took 1.65 ms a launch so).  The in-row
// neighbours of column (m, j) are (m - 1 + s, j) and (m + s, j) of the other
// colour, s = 0 or 1 by the parity of the row; north and south are (m, j -+ 1).
//
// A block takes a tile at a time.  A column is shared by G threads, each with LC
// consecutive levels in registers; consecutive threads hold consecutive
// columns, so every load is a full 128-byte line and a thread's loads are
// issued together.  The tridiagonal recurrences run level by level inside a
// thread and as a scan of affine maps over the column's threads through
// shared memory, so nothing is spilled or read twice.  A thread that marches
// down a column alone waits a memory latency every few levels (27 us a launch on
// the 512 x 1 x 60 slice).
//
// Dot products are reduced deterministically: every block writes a partial sum
// and the last one to finish (atomic ticket) adds the partials in block
// order and updates the solver scalars on the device, so an iteration
// needs no host round trip.  A device flag marks convergence; kernels of an
// already converged solve return at once.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "ops.h"
#include "tma.cuh"

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
constexpr int kMaxBlocks = 4096;  // the largest grid that leaves partial sums

// A block adds its threads' values in a fixed order and writes one partial;
// true in thread 0 of the last block of the grid to get here, which then holds
// the totals in v (partials added in block order).  Grids are a function of
// the sizes and the device alone, so totals are reproducible.
template <int NV, int kThreads>
__device__ bool grid_sum(double (&v)[NV], SolverState* S) {
  constexpr int kWarps = kThreads / 32;
  __shared__ double sh[NV][kWarps];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto block_sum = [&]() {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double x = v[q];
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
    }
  };
  block_sum();
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) S->partials[(size_t)q * S->max_blocks + blockIdx.x] = v[q];
    __threadfence();
    last = atomicAdd(&S->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const double* part = S->partials + (size_t)q * S->max_blocks;
    double x = 0.0;
#pragma unroll 8
    for (int b = tid; b < (int)gridDim.x; b += kThreads) x += __ldcg(part + b);
    v[q] = x;
  }
  block_sum();
  if (tid == 0) S->ticket = 0;
  return tid == 0;
}

// ------------------------------------------------------- set-up ---------
__device__ __forceinline__ int red_i(int m, int j) { return 2 * m + (j & 1); }
__device__ __forceinline__ int black_i(int m, int j) { return 2 * m + 1 - (j & 1); }


// Pivots of the column tridiagonal of B (constant): dinv(K) = 1/d'(K) with
// d'(1) = d(1), d'(K) = d(K) - a(K) c(K-1) / d'(K-1), in the layout of
// precision T: the red ones in T (the elimination is exact to
// the solve's precision), the black ones, a fixed preconditioner, in FP32 for
// both forms; the 2D data of the columns, kk with the wet levels of the column
// and of its neighbours; and the deepest wet level km of each tile.  Columns that
// are no unknowns keep kk = 0 (no wet level).
template <typename T>
__global__ void k_rb_setup(Geo G, PoissonGeo P, RbGeo R, T* __restrict__ dr,
                           float* __restrict__ db, int* __restrict__ km) {
  const int W = R.width((int)sizeof(T));
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
  const int m = (i >> 1) - 1, nt = R.nt(W);
  atomicMax(km + (black ? nt * (G.L.je + 1) : 0) + j * nt + m / W, c.kb);
  double dprev = 1.0, cprev = 0.0;
  for (int K = 1; K <= c.kb; ++K) {
    const Coef r = row<true>(c, P, K, KE);
    const double d = K == 1 ? r.dc : r.dc - (r.u * dprev) * cprev;
    const double di = 1.0 / d;
    const int o = ((j * nt + m / W) * KE + K - 1) * W + m % W;
    if (black) db[o] = (float)di;
    else dr[o] = (T)di;
    dprev = di;
    cprev = r.d;
  }
}

// ------------------------------------------------------- PCG kernels -----
// Where a thread stands: column c of the tile, levels K0 + 1 .. K0 + LC.
template <typename T, int G, int LC, int H>
struct Lane {
  using V = T;
  static constexpr int W = (128 >> H) / (int)sizeof(T);  // columns per tile
  static constexpr int NT = W * G, ROWS = G * LC, L = LC, GROUPS = G;
  int c, g, K0;
  __device__ __forceinline__ Lane() : c(threadIdx.x % W), g(threadIdx.x / W), K0(g * LC) {}
};

// ZW(K) at szw[K - 1], K = 1..KE+1, and 1/ZP(K) at siz[K - 1]
template <typename Ln, typename T>
__device__ __forceinline__ void load_tables(const RbGeo& R, T* szw, T* siz) {
  for (int e = threadIdx.x; e <= Ln::ROWS; e += Ln::NT) {
    szw[e] = e <= R.ke ? (T)R.zwn[e] : T(0);
    if (siz) siz[e] = e < R.ke ? (T)R.izn[e] : T(0);
  }
}

// the vertical profiles at level K, K - 1 the index
template <typename Ln, typename T>
__device__ __forceinline__ void load_profiles(const RbGeo& R, T (*sphi)[Ln::ROWS]) {
  for (int e = threadIdx.x; e < RbCoarse::kModes * Ln::ROWS; e += Ln::NT) {
    const int q = e / Ln::ROWS, k = e % Ln::ROWS;
    sphi[q][k] = k < R.ke ? (T)R.phi[q * R.ke + k] : T(0);
  }
}

// Couplings a(K) between levels K - 1 and K of the thread's levels and of the
// one below its last: ZW(K) inside the column (its own value at the bottom),
// 0 at the surface and below the bottom.
template <typename Ln, typename T, int LC>
__device__ __forceinline__ void couplings(const Ln& t, const T* szw, int kb, T zwa, T (&a)[LC]) {
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    const int K = t.K0 + 1 + u;
    const T zw = szw[t.K0 + u];
    a[u] = (K == 1 || K > kb) ? T(0) : (K == kb ? zwa : zw);
  }
}

// Affine maps of the threads of a column, down and up
template <typename Ln>
struct Scan {
  typename Ln::V fa[Ln::GROUPS][Ln::W], fb[Ln::GROUPS][Ln::W], ba[Ln::GROUPS][Ln::W],
      bb[Ln::GROUPS][Ln::W];
};

// A thread's part of a dot product, one term per level u.  FP32 terms are added in FP32
// four levels at a time, then in FP64.
template <typename T>
struct Dot {
  T part = T(0);
  double sum = 0.0;
  __device__ __forceinline__ void add(int u, T a, T b) {
    part = fma(a, b, part);
    if (sizeof(T) == 4 && u % 4 == 3) {
      sum += (double)part;
      part = T(0);
    }
  }
  __device__ __forceinline__ double total() const {
    return sizeof(T) == 4 ? sum + (double)part : (double)part;
  }
};

// v <- M^-1 v for the column tridiagonal M = L D L^T with pivots 1/d (dm: the
// pivot above the thread's first level) and couplings a; returns v.M^-1 v =
// sum y^2 / d of this thread's levels.  Two block barriers; first() is the first
// of them, and runs after it: every thread has its inputs in registers there.
template <typename Ln, typename T, int LC, typename F>
__device__ __forceinline__ double column_solve(const Ln& t, Scan<Ln>& sc, T (&v)[LC], const T (&d)[LC],
                                               T dm, const T (&a)[LC + 1], F&& first) {
  constexpr int G = Ln::GROUPS;
  // forward: y(K) = v(K) - a(K) d(K-1) y(K-1); the thread's levels as one affine
  // map y_out = A y_in + B, applied in turn to what comes from above
  T A = T(1), B = T(0);
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    const T l = -(a[u] * (u ? d[u - 1] : dm));
    B = fma(l, B, v[u]);
    A = l * A;
  }
  sc.fa[t.g][t.c] = A;
  sc.fb[t.g][t.c] = B;
  first();
  T y = T(0);
#pragma unroll
  for (int k = 0; k < G - 1; ++k)
    if (k < t.g) y = fma(sc.fa[k][t.c], y, sc.fb[k][t.c]);
  Dot<T> rz;
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    y = fma(-(a[u] * (u ? d[u - 1] : dm)), y, v[u]);
    v[u] = y * d[u];
    rz.add(u, y, v[u]);
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
  sc.ba[t.g][t.c] = A;
  sc.bb[t.g][t.c] = B;
  __syncthreads();
  T z = T(0);
#pragma unroll
  for (int k = G - 1; k > 0; --k)
    if (k > t.g) z = fma(sc.ba[k][t.c], z, sc.bb[k][t.c]);
#pragma unroll
  for (int u = LC - 1; u >= 0; --u) {
    z = fma(-(a[u + 1] * d[u]), z, v[u]);
    v[u] = z;
  }
  return rz.total();
}

__device__ __forceinline__ int wet_levels(unsigned long long kk, int nb) {
  return (int)((kk >> (10 * nb)) & 1023u);
}

// The tiles of one colour and what a thread sees of one: row j, the column
// m = i / 2, the offset o0 of its first level in the tiled layout, and whether
// its west neighbour of the other colour is column m (sh) or m - 1.
struct Tile {
  int j, b, m, o0;
  bool sh;
  unsigned long long kk;
};
template <typename Ln>
struct Tiles {
  const RbGeo& R;
  const RbColour& q;
  const Ln& t;
  int ntiles, nt;
  bool red;
  __device__ __forceinline__ unsigned long long kk(int tile) const {
    const int m = 1 + (tile % nt) * Ln::W + t.c;
    return tile < ntiles && m <= R.M ? __ldg(q.kk + m + R.P2 * (2 + tile / nt)) : 0ull;
  }
  __device__ __forceinline__ Tile at(int tile, unsigned long long kk) const {
    Tile a;
    a.j = 2 + tile / nt;
    a.b = tile % nt;
    a.m = 1 + a.b * Ln::W + t.c;
    a.o0 = ((a.j * nt + a.b) * R.ke + t.K0) * Ln::W + t.c;
    a.sh = (a.j & 1) == (red ? 1 : 0);
    a.kk = kk;
    return a;
  }
};

__device__ __forceinline__ void solve_gave_up(SolverState* S) {
  atomicExch(&S->converged, 4);
  atomicExch(&S->gave_up, 1);
}

// Staging.  A block's next tile is copied to shared memory while it computes
// this one: one thread issues a bulk copy per array (a tile is consecutive
// memory; down to the tile's deepest wet level), all wait on an mbarrier.  NA
// arrays of T, the pivots (D, ND = 1 or 0) and the four pairs of 2D data; the
// in-row neighbours across the tile's edge come by a copy per level.
// Loads straight to registers left the kernels waiting for most of the time
// (black kernel 106 us at 448 x 448 x 80, 10 of 14 cycles of a warp in
// long-scoreboard stalls), copies by every thread cost as many instructions as the
// computation (red kernel 67 -> 80 us).
template <typename Ln, typename D, int NA, int ND>
struct Stage {
  using T = typename Ln::V;
  static constexpr int ROWS = Ln::ROWS, W = Ln::W, N = ROWS * W;
  static constexpr size_t smem =
      16 * 4 * W + sizeof(T) * N * NA + sizeof(D) * N * ND + sizeof(T) * ROWS;
  double2* pairs;
  T *data, *edge;
  D* piv;
  uint64_t* bar;
  uint32_t phase;
  long long limit;
  bool ok;    // this thread's waits
  bool stop;  // a thread of the block has given up (the same for all)
  __device__ __forceinline__ Stage(unsigned char* dsm, uint64_t* b, const SolverState* S)
      : bar(b), phase(0), limit(S->wait), ok(true), stop(false) {
    pairs = reinterpret_cast<double2*>(dsm);
    data = reinterpret_cast<T*>(dsm + 16 * 4 * W);
    piv = reinterpret_cast<D*>(dsm + 16 * 4 * W + sizeof(T) * N * NA);
    edge = reinterpret_cast<T*>(dsm + 16 * 4 * W + sizeof(T) * N * NA + sizeof(D) * N * ND);
    if (threadIdx.x == 0) {
      mbar_init(bar, 1);
      mbar_init_fence();
    }
  }
  // Issues the copies of tile a (the block has read the slots' last contents):
  // arrays n = 0..NA-1 from v[n] at the tile's own place plus rows[n] rows.
  template <int NV>
  __device__ __forceinline__ void issue(const Tiles<Ln>& s, const Tile& a, const int* __restrict__ km,
                                        const T* const (&v)[NV], const int (&rows)[NV],
                                        const D* dinv, const T* edge_of) {
    static_assert(NV == NA || NA == 0, "");
    const int ke = s.R.ke;
    if (threadIdx.x == 0) {
      const uint32_t n = (uint32_t)__ldg(km + (s.red ? 0 : s.nt * (s.R.je + 1)) + a.j * s.nt + a.b);
      mbar_arrive_expect_tx(bar, 16 * 4 * W + n * W * (uint32_t)(sizeof(T) * NA + sizeof(D) * ND));
      const int s2 = 1 + a.b * W + s.R.P2 * a.j;
      bulk_load(pairs, s.q.zw + s2, 16 * W, bar);
      bulk_load(pairs + W, s.q.iz + s2, 16 * W, bar);
      bulk_load(pairs + 2 * W, s.q.we + s2, 16 * W, bar);
      bulk_load(pairs + 3 * W, s.q.ns + s2, 16 * W, bar);
      if (n) {
#pragma unroll
        for (int e = 0; e < NA; ++e)
          bulk_load(data + e * N, v[e] + (size_t)((a.j + rows[e]) * s.nt + a.b) * ke * W,
                    n * W * (uint32_t)sizeof(T), bar);
        if (ND)
          bulk_load(piv, dinv + (size_t)(a.j * s.nt + a.b) * ke * W, n * W * (uint32_t)sizeof(D), bar);
      }
    }
    if (NA > 0 && edge_of && s.t.c == (a.sh ? W - 1 : 0)) {
      // this column's neighbour is in the tile to the west (c = 0) or east
      const bool there = a.sh ? a.b + 1 < s.nt : a.b > 0;
      const int o = a.o0 + (a.sh ? ke * W - (W - 1) : (W - 1) - ke * W);
      const int kb = wet_levels(a.kk, 0);
#pragma unroll
      for (int q = 0; q < Ln::L; ++q) {
        const bool get = there && s.t.K0 + 1 + q <= kb;
        copy_async(edge + s.t.K0 + q, edge_of + (get ? o + W * q : 0), get);
      }
    }
  }
  __device__ __forceinline__ void wait() {
    copies_wait();
    ok = mbar_wait(bar, phase, limit);
    phase ^= 1;
  }
  // A barrier of the block after wait(): whether the tiles go on.  If a thread gave
  // up, no further copy is issued, and the block ends after this tile.
  __device__ __forceinline__ bool goes_on() {
    stop = __syncthreads_or(!ok);
    return !stop;
  }
  __device__ __forceinline__ T get(const Ln& t, int n, int q) const {
    return data[n * N + (t.K0 + q) * W + t.c];
  }
  // C v of the thread's levels without the factor 1/ZP, 0 below the bottom
  // (values of land cells and outside the unknowns are exact zeros); arrays
  // n, n+1, n+2: the tile itself and the ones north and south of it
  __device__ __forceinline__ void neighbour_sum(const Ln& t, const Tile& a, int n, double2 we,
                                                double2 ns, T (&h)[Ln::L]) const {
    const T cw = (T)we.x, ce = (T)we.y, cn = (T)ns.x, cs = (T)ns.y;
    const T co = a.sh ? cw : ce, cx = a.sh ? ce : cw;  // column m, and the other one
    const int cc = a.sh ? min(t.c + 1, W - 1) : max(t.c - 1, 0);
    const bool across = t.c == (a.sh ? W - 1 : 0);
    const int kb = wet_levels(a.kk, 0);
    const T* d = data + n * N + t.K0 * W;
#pragma unroll
    for (int q = 0; q < Ln::L; ++q) {
      h[q] = co * d[q * W + t.c];
      T x = d[q * W + cc];
      if (across) x = edge[t.K0 + q];
      h[q] = fma(cx, x, h[q]);
      h[q] = fma(cn, d[N + q * W + t.c], h[q]);
      h[q] = fma(cs, d[2 * N + q * W + t.c], h[q]);
      if (t.K0 + 1 + q > kb) h[q] = T(0);
    }
  }
  // pivots of the thread's levels and the one above the first
  __device__ __forceinline__ void pivots(const Ln& t, int kb, T& dm, T (&d)[Ln::L]) const {
    dm = t.K0 > 0 && t.K0 <= kb ? (T)piv[(t.K0 - 1) * W + t.c] : T(0);
#pragma unroll
    for (int q = 0; q < Ln::L; ++q)
      d[q] = t.K0 + 1 + q <= kb ? (T)piv[(t.K0 + q) * W + t.c] : T(0);
  }
  // A copy that did not land stops the solve; it is waited for once more, so that it
  // does not write to the next block's shared memory.
  __device__ __forceinline__ void report(SolverState* S) const {
    if (!ok) mbar_wait(bar, phase ^ 1, kWaitCycles);
    if (stop && threadIdx.x == 0) solve_gave_up(S);
  }
};

// Red columns.
//   kIter    u = D^-1 C v + beta u          (v = z; u is not used while beta = 0)
//   kBefore  u = D^-1 (b / ZP)              (b: full layout, scaled); sum of (b / ZP)^2
//   kAfter   x += scale (u - D^-1 C v)      (v = the black correction; x: full layout)
enum { kIter = 0, kBefore = 1, kAfter = 2 };

template <typename Ln, int MODE>
using RedStage = Stage<Ln, typename Ln::V, MODE == kBefore ? 0 : 3, 1>;

template <typename Ln, int MODE, typename T = typename Ln::V>
__global__ void __launch_bounds__(Ln::NT) k_rb_red(RbGeo R, SolverState* S,
                                                   const T* __restrict__ v, T* __restrict__ u,
                                                   const T* __restrict__ dinv,
                                                   const int* __restrict__ km,
                                                   const double* __restrict__ b,
                                                   double* __restrict__ x,
                                                   const float* __restrict__ cc, int ntiles, int nt) {
  constexpr int W = Ln::W, LC = Ln::L;
  extern __shared__ __align__(128) unsigned char dsm[];
  __shared__ T szw[Ln::ROWS + 1], siz[Ln::ROWS + 1], sphi[RbCoarse::kModes][Ln::ROWS];
  __shared__ Scan<Ln> scan;
  __shared__ __align__(8) uint64_t bar;
  if (MODE == kIter && S->converged) return;
  const T beta = MODE == kIter ? (T)S->beta : T(0);
  double scale = 1.0;
  if (MODE != kIter && sizeof(T) == 4) {
    scale = sqrt(S->res_rr);
    if (MODE == kBefore) scale = scale > 0.0 ? 1.0 / scale : 0.0;
  }
  const Ln t;
  const Tiles<Ln> tiles{R, R.col[0], t, ntiles, nt, true};
  RedStage<Ln, MODE> st(dsm, &bar, S);
  load_tables<Ln>(R, szw, siz);
  if (MODE == kIter && cc) load_profiles<Ln>(R, sphi);
  __syncthreads();
  auto issue = [&](const Tile& a) { st.issue(tiles, a, km, {v, v, v}, {0, -1, 1}, dinv, v); };
  int tile = blockIdx.x;
  Tile next = tiles.at(tile, tiles.kk(tile));
  issue(next);
  unsigned long long kn = tiles.kk(tile + gridDim.x);
  const int plane = 2 * R.plane2;  // full layout
  double bb = 0.0;
  for (; tile < ntiles; tile += gridDim.x) {
    const Tile a = next;
    const int kb = wet_levels(a.kk, 0);
    T g[LC], d[LC], uo[LC], cp[LC + 1], dm;
    if (MODE != kBefore) {
#pragma unroll
      for (int q = 0; q < LC; ++q) uo[q] = t.K0 + 1 + q <= kb ? u[a.o0 + W * q] : T(0);
    }
    const bool coarse = MODE == kIter && cc && t.K0 < kb;
    float cz[RbCoarse::kModes][4];  // the coarse correction west, east, north, south
    if (coarse) {
      const int s2 = a.m + R.P2 * a.j, w = s2 - 1 + (a.sh ? 1 : 0);
#pragma unroll
      for (int q = 0; q < RbCoarse::kModes; ++q) {
        const float* cq = cc + q * R.plane2;
        cz[q][0] = cq[w];
        cz[q][1] = cq[w + 1];
        cz[q][2] = cq[s2 - R.P2];
        cz[q][3] = cq[s2 + R.P2];
      }
    }
    const int f0 = red_i(a.m, a.j) + 2 * R.P2 * a.j + plane * t.K0;
    if (MODE == kBefore) {
#pragma unroll
      for (int q = 0; q < LC; ++q) g[q] = T(0);
    }
    st.wait();
    const T zwa = (T)st.pairs[t.c].x;
    const double2 iz = st.pairs[W + t.c];
    st.pivots(t, kb, dm, d);
    if (MODE == kBefore) {
#pragma unroll
      for (int q = 0; q < LC; ++q) {
        const int K = t.K0 + 1 + q;
        const double hs = K == kb ? iz.y : (K == kb - 1 ? iz.x : (double)R.izn[K <= kb ? K - 1 : 0]);
        const double bv = b[K <= kb ? f0 + plane * q : 0];
        g[q] = K <= kb ? (T)((bv * scale) * hs) : T(0);
        bb = fma((double)g[q], (double)g[q], bb);
      }
    } else {
      const double2 we = st.pairs[2 * W + t.c], ns = st.pairs[3 * W + t.c];
      st.neighbour_sum(t, a, 0, we, ns, g);
      if (coarse) {
        const T cn4[4] = {(T)we.x, (T)we.y, (T)ns.x, (T)ns.y};
        int km4 = kb;
#pragma unroll
        for (int d4 = 0; d4 < 4; ++d4) km4 = min(km4, wet_levels(a.kk, 1 + d4));
        T g0 = T(0), g1 = T(0);
#pragma unroll
        for (int d4 = 0; d4 < 4; ++d4) {
          g0 = fma(cn4[d4], (T)cz[0][d4], g0);
          g1 = fma(cn4[d4], (T)cz[1][d4], g1);
        }
#pragma unroll
        for (int q = 0; q < LC; ++q) {
          const int K = t.K0 + 1 + q;
          if (K <= km4) {
            g[q] = fma(sphi[0][t.K0 + q], g0, fma(sphi[1][t.K0 + q], g1, g[q]));
          } else if (K <= kb) {  // some neighbours end above
#pragma unroll
            for (int d4 = 0; d4 < 4; ++d4)
              if (K <= wet_levels(a.kk, 1 + d4))
                g[q] = fma(cn4[d4], fma(sphi[0][t.K0 + q], (T)cz[0][d4], sphi[1][t.K0 + q] * (T)cz[1][d4]), g[q]);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < LC; ++q) {
        const int K = t.K0 + 1 + q;
        g[q] *= K == kb ? (T)iz.y : (K == kb - 1 ? (T)iz.x : siz[t.K0 + q]);
      }
    }
    couplings(t, szw, kb, kb ? zwa : T(0), cp);
    column_solve(t, scan, g, d, dm, cp, [&] {
      if (st.goes_on() && tile + (int)gridDim.x < ntiles) {
        next = tiles.at(tile + gridDim.x, kn);
        issue(next);
        kn = tiles.kk(tile + 2 * gridDim.x);
      }
    });
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      if (t.K0 + 1 + q <= kb) {
        if (MODE == kAfter) {
          const int f = f0 + plane * q;
          x[f] = x[f] + scale * (double)(uo[q] - g[q]);
        } else {
          u[a.o0 + W * q] = MODE == kIter && beta != T(0) ? fma(beta, uo[q], g[q]) : g[q];
        }
      }
    }
    if (st.stop) break;
  }
  st.report(S);
  if (MODE == kBefore) {
    double w[1] = {bb};
    if (grid_sum<1, Ln::NT>(w, S)) S->bb = w[0];
  }
}

// Black columns: x += alpha p (the previous step's), p = z + beta p,
// q = D p - C u, and alpha = rho / p.q.  The first iteration (iter = 0) uses
// neither p nor x.
template <typename Ln>
using BlackStage = Stage<Ln, typename Ln::V, 6, 0>;

template <typename Ln, typename T = typename Ln::V>
__global__ void __launch_bounds__(Ln::NT) k_rb_black(RbGeo R, SolverState* S,
                                                     const T* __restrict__ z,
                                                     const T* __restrict__ u, T* __restrict__ p,
                                                     T* __restrict__ x, T* __restrict__ q,
                                                     const int* __restrict__ km,
                                                     const float* __restrict__ cc, int ntiles, int nt) {
  constexpr int W = Ln::W, LC = Ln::L, G = Ln::GROUPS;
  extern __shared__ __align__(128) unsigned char dsm[];
  __shared__ T szw[Ln::ROWS + 1], siz[Ln::ROWS + 1], sphi[RbCoarse::kModes][Ln::ROWS];
  __shared__ T top[2][G][W], bottom[2][G][W];  // p of the threads' first and last levels
  __shared__ __align__(8) uint64_t bar;
  if (S->converged) return;
  const T beta = (T)S->beta, alpha = (T)S->alpha_prev;
  const bool first = S->iter == 0;
  const Ln t;
  const Tiles<Ln> tiles{R, R.col[1], t, ntiles, nt, false};
  BlackStage<Ln> st(dsm, &bar, S);
  load_tables<Ln>(R, szw, siz);
  if (cc) load_profiles<Ln>(R, sphi);
  __syncthreads();
  auto issue = [&](const Tile& a) {
    st.issue(tiles, a, km, {u, u, u, z, p, x}, {0, -1, 1, 0, 0, 0}, u, u);
  };
  int tile = blockIdx.x;
  Tile next = tiles.at(tile, tiles.kk(tile));
  issue(next);
  unsigned long long kn = tiles.kk(tile + gridDim.x);
  double pq = 0.0;
  int buf = 0;
  for (; tile < ntiles; tile += gridDim.x) {
    const Tile a = next;
    const int kb = wet_levels(a.kk, 0);
    T pl[LC], xo[LC], v[LC];
    const bool coarse = cc && t.K0 < kb;
    const T c0 = coarse ? (T)cc[a.m + R.P2 * a.j] : T(0);
    const T c1 = coarse ? (T)cc[R.plane2 + a.m + R.P2 * a.j] : T(0);
    st.wait();
    const double2 zw = st.pairs[t.c], iz = st.pairs[W + t.c];
    const double2 we = st.pairs[2 * W + t.c], ns = st.pairs[3 * W + t.c];
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      const bool old = !first && t.K0 + 1 + e <= kb;
      const T po = old ? st.get(t, 4, e) : T(0);
      xo[e] = fma(alpha, po, old ? st.get(t, 5, e) : T(0));
      T zv = t.K0 + 1 + e <= kb ? st.get(t, 3, e) : T(0);
      if (coarse && t.K0 + 1 + e <= kb) zv = fma(sphi[0][t.K0 + e], c0, fma(sphi[1][t.K0 + e], c1, zv));
      pl[e] = fma(beta, po, zv);
    }
    st.neighbour_sum(t, a, 0, we, ns, v);
    top[buf][t.g][t.c] = pl[0];
    bottom[buf][t.g][t.c] = pl[LC - 1];
    if (st.goes_on() && tile + (int)gridDim.x < ntiles) {
      next = tiles.at(tile + gridDim.x, kn);
      issue(next);
      kn = tiles.kk(tile + 2 * gridDim.x);
    }
#pragma unroll
    for (int e = 0; e < LC; ++e)
      if (t.K0 + 1 + e <= kb) {
        x[a.o0 + W * e] = xo[e];
        p[a.o0 + W * e] = pl[e];
      }
    T pu = t.g == 0 ? T(0) : bottom[buf][t.g - 1][t.c];
    const T pb = t.g == G - 1 ? T(0) : top[buf][t.g + 1][t.c];
    buf ^= 1;
    const T cw = (T)we.x, ce = (T)we.y, cn = (T)ns.x, cs = (T)ns.y, zwa = (T)zw.x;
    const int kbw = wet_levels(a.kk, 1), kbe = wet_levels(a.kk, 2);
    const int kbn = wet_levels(a.kk, 3), kbs = wet_levels(a.kk, 4);
    Dot<T> pqt;
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      const int K = t.K0 + 1 + e;
      const T p0 = pl[e], pd = e + 1 < LC ? pl[e + 1] : pb;
      T dh = K <= kbw ? cw : T(0);
      dh += K <= kbe ? ce : T(0);
      dh += K <= kbn ? cn : T(0);
      dh += K <= kbs ? cs : T(0);
      const T h = fma(dh, p0, v[e]);
      const T hs = K == kb ? (T)iz.y : (K == kb - 1 ? (T)iz.x : siz[t.K0 + e]);
      const T zw0 = K == kb ? zwa : szw[t.K0 + e];
      // below the bottom nothing couples, but Z_C of the surface row keeps ZW(2)
      T zw1 = K + 1 == kb ? zwa : szw[t.K0 + e + 1];
      if (K == kb) zw1 = K == 1 ? (T)zw.y : T(0);
      T s = zw0 * (pu - p0);
      s = fma(zw1, pd - p0, s);
      s = fma(-hs, h, s);
      if (K <= kb) {
        q[a.o0 + W * e] = s;
      }
      pqt.add(e, p0, K <= kb ? s : T(0));
      pu = p0;
    }
    pq += pqt.total();
    if (st.stop) break;
  }
  st.report(S);
  double w[1] = {pq};
  if (grid_sum<1, Ln::NT>(w, S)) {
    S->pq = w[0];
    S->alpha = S->rho / w[0];
    if (S->converged == 0 && !(w[0] > 0.0) && !(w[0] < 0.0)) {
      S->converged = 3;  // breakdown: x has the last full step, and p is no direction to follow
      S->alpha_prev = 0.0;
    }
  }
}

// Black columns: residual, z = D_b^-1 r with the FP32 pivots, r.z and r.r.
//   INIT   r = b / ZP - C u     (u = D_r^-1 (b / ZP) of the red columns)
//   else   r -= alpha q
template <typename Ln, bool INIT>
using ColStage = Stage<Ln, float, INIT ? 3 : 2, 1>;

template <typename Ln, bool INIT, typename T = typename Ln::V>
__global__ void __launch_bounds__(Ln::NT) k_rb_col(RbGeo R, SolverState* S, T* __restrict__ r,
                                                   const T* __restrict__ q, T* __restrict__ z,
                                                   const float* __restrict__ dinv,
                                                   const int* __restrict__ km,
                                                   const double* __restrict__ b,
                                                   const T* __restrict__ ub, T* __restrict__ rho,
                                                   int ntiles, int nt) {
  constexpr int W = Ln::W, LC = Ln::L, NM = RbCoarse::kModes;
  extern __shared__ __align__(128) unsigned char dsm[];
  __shared__ T szw[Ln::ROWS + 1], sphi[NM][Ln::ROWS], part[NM][Ln::GROUPS][W];
  __shared__ Scan<Ln> scan;
  __shared__ __align__(8) uint64_t bar;
  if (!INIT && S->converged) return;
  const T alpha = INIT ? T(0) : (T)S->alpha;
  double scale = 1.0;
  if (INIT && sizeof(T) == 4) scale = S->res_rr > 0.0 ? 1.0 / sqrt(S->res_rr) : 0.0;
  const Ln t;
  const Tiles<Ln> tiles{R, R.col[1], t, ntiles, nt, false};
  ColStage<Ln, INIT> st(dsm, &bar, S);
  load_tables<Ln, T>(R, szw, nullptr);
  if (rho) load_profiles<Ln>(R, sphi);
  __syncthreads();
  auto issue = [&](const Tile& a) {
    if constexpr (INIT) st.issue(tiles, a, km, {ub, ub, ub}, {0, -1, 1}, dinv, ub);
    else st.issue(tiles, a, km, {q, (const T*)r}, {0, 0}, dinv, nullptr);
  };
  int tile = blockIdx.x;
  Tile next = tiles.at(tile, tiles.kk(tile));
  issue(next);
  unsigned long long kn = tiles.kk(tile + gridDim.x);
  double rz = 0.0, rr = 0.0, bb = 0.0;
  for (; tile < ntiles; tile += gridDim.x) {
    const Tile a = next;
    const int kb = wet_levels(a.kk, 0);
    T g[LC], d[LC], cp[LC + 1], dm;
    Dot<T> rrt;
    st.wait();
    const T zwa = (T)st.pairs[t.c].x;
    st.pivots(t, kb, dm, d);
    if constexpr (INIT) {
      const double2 iz = st.pairs[W + t.c];
      const int plane = 2 * R.plane2;
      const int f0 = black_i(a.m, a.j) + 2 * R.P2 * a.j + plane * t.K0;
      st.neighbour_sum(t, a, 0, st.pairs[2 * W + t.c], st.pairs[3 * W + t.c], g);
#pragma unroll
      for (int e = 0; e < LC; ++e) {
        const int K = t.K0 + 1 + e;
        const double hs = K == kb ? iz.y : (K == kb - 1 ? iz.x : (double)R.izn[K <= kb ? K - 1 : 0]);
        const T bs = K <= kb ? (T)((b[K <= kb ? f0 + plane * e : 0] * scale) * hs) : T(0);
        g[e] = K <= kb ? fma(-(T)hs, g[e], bs) : T(0);
        bb = fma((double)bs, (double)bs, bb);
      }
    } else {
#pragma unroll
      for (int e = 0; e < LC; ++e)
        g[e] = t.K0 + 1 + e <= kb ? fma(-alpha, st.get(t, 0, e), st.get(t, 1, e)) : T(0);
    }
    couplings(t, szw, kb, kb ? zwa : T(0), cp);
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      if (t.K0 + 1 + e <= kb) r[a.o0 + W * e] = g[e];
      rrt.add(e, g[e], g[e]);
    }
    if (rho) {  // the column's products with the profiles
#pragma unroll
      for (int q = 0; q < NM; ++q) {
        T f = T(0);
#pragma unroll
        for (int e = 0; e < LC; ++e) f = fma(sphi[q][t.K0 + e], g[e], f);
        part[q][t.g][t.c] = f;
      }
    }
    rz += column_solve(t, scan, g, d, dm, cp, [&] {
      const bool on = st.goes_on();
      if (rho && t.g < NM && kb) {
        T f = T(0);
#pragma unroll
        for (int k = 0; k < Ln::GROUPS; ++k) f += part[t.g][k][t.c];
        rho[t.g * R.plane2 + a.m + R.P2 * a.j] = f;
      }
      if (on && tile + (int)gridDim.x < ntiles) {
        next = tiles.at(tile + gridDim.x, kn);
        issue(next);
        kn = tiles.kk(tile + 2 * gridDim.x);
      }
    });
    rr += rrt.total();
#pragma unroll
    for (int e = 0; e < LC; ++e)
      if (t.K0 + 1 + e <= kb) z[a.o0 + W * e] = g[e];
    if (st.stop) break;
  }
  st.report(S);
  double v[INIT ? 3 : 2];
  v[0] = rz;
  v[1] = rr;
  if (INIT) v[2] = bb;
  if (grid_sum<INIT ? 3 : 2, Ln::NT>(v, S)) {
    if (INIT) {
      S->bb += v[2];  // the red columns' part is there already
      S->beta = 0.0;
      S->alpha_prev = 0.0;
    } else {
      S->beta = v[0] / S->rho;
      S->alpha_prev = S->alpha;
      S->iter += 1;
    }
    S->rz = v[0];
    if (INIT || !rho) S->rho = v[0];  // else k_rb_coarse makes rho and beta
    S->rr = v[1];
    if (S->converged == 0) {
      if (sqrt(v[1]) <= S->tol * sqrt(S->bb) || S->bb == 0.0) S->converged = 1;
      if (!(v[0] == v[0]) || !(v[1] == v[1])) S->converged = 2;  // NaN: stop
    }
  }
}

// ------------------------------------------------------- coarse space ----
// What D alone leaves to the iterations are modes that are smooth in the
// vertical: at 500 m spacing over 4000 m of water the lowest vertical mode is held by
// the horizontal couplings 50 times as strongly as by the vertical ones, and conjugate
// gradients took 74 iterations for ten decimals (256 x 256 x 60), each three
// passes over the vectors.  The preconditioner is therefore
//     M^-1 = D_b^-1 + sum_q phi_q (p_q(S_q) - d_q^-1) phi_q^T
// with the two lowest vertical profiles phi_q of the deepest column (one 1D table,
// cut at each column's bottom), the 2D operators S_q = d_q - c_q d_q^-1 c_q^T of the
// Galerkin products d = phi^T D phi, c = phi^T C phi on the red and black columns,
// and p_q(S_q) some Chebyshev steps for S_q^-1, a few planes instead of volumes.  The
// part that D_b^-1 does already, d_q^-1, is taken off; p_q is scaled
// to be no smaller, so M^-1 stays definite whatever the topography.  29 iterations
// instead of 74 on the box, 9 instead of 23 on 1024 x 1024 x 80 at 1852 m.

// The 2D operators, unscaled: diagonal (sc), couplings east and south
__global__ void k_coarse_sums(Geo G, PoissonGeo P, RbGeo R) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int KE = G.L.ke, IE = G.L.ie, JE = G.L.je;
  if (i > IE - 1 || j > JE - 1) return;
  constexpr int NM = RbCoarse::kModes;
  const ColC c = load_col(G, P, i, j);
  const ColC e = load_col(G, P, min(i + 1, IE - 1), j), s = load_col(G, P, i, min(j + 1, JE - 1));
  double dd[NM] = {}, ee[NM] = {}, ss[NM] = {};
  for (int K = 1; K <= c.kb; ++K) {
    const Coef r = row<true>(c, P, K, KE);
    // the smaller of the two entries where the operator is not symmetric
    double he = 0., hs = 0.;
    if (c.ie && K <= c.kbe) he = fmin(c.ce * izp_of(c, P, K), e.cw * izp_of(e, P, K));
    if (c.is && K <= c.kbs) hs = fmin(c.cs * izp_of(c, P, K), s.cn * izp_of(s, P, K));
#pragma unroll
    for (int q = 0; q < NM; ++q) {
      const double* f = R.phi + q * KE;
      const double f0 = f[K - 1], fu = K > 1 ? f[K - 2] : 0., fd = K < KE ? f[K] : 0.;
      dd[q] -= f0 * (r.dc * f0 + r.u * fu + r.d * fd);
      ee[q] += f0 * f0 * he;
      ss[q] += f0 * f0 * hs;
    }
  }
#pragma unroll
  for (int q = 0; q < NM; ++q) {
    const int o = q * G.L.plane + c.ij;
    R.co.sc[o] = (float)dd[q];
    R.co.ce[o] = (float)ee[q];
    R.co.cs[o] = (float)ss[q];
  }
}

// The largest sum of a column's couplings over its diagonal
__global__ void k_coarse_mu(Geo G, RbGeo R) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  if (i > G.L.ie - 1 || j > G.L.je - 1) return;
  for (int q = 0; q < RbCoarse::kModes; ++q) {
    const int o = q * G.L.plane + G.L.at2(i, j);
    const float d = R.co.sc[o];
    const float c = R.co.ce[o] + R.co.ce[o - 1] + R.co.cs[o] + R.co.cs[o - G.L.P];
    if (d > 0.f) atomicMax(reinterpret_cast<int*>(R.co.mu + q), __float_as_int(c / d));
  }
}

// Scaling to a unit diagonal: first the couplings (SC false), then sc
template <bool SC>
__global__ void k_coarse_scale(Geo G, RbGeo R) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  if (i > G.L.ie - 1 || j > G.L.je - 1) return;
  for (int q = 0; q < RbCoarse::kModes; ++q) {
    const int o = q * G.L.plane + G.L.at2(i, j);
    auto inv = [&](int a) { return R.co.sc[a] > 0.f ? rsqrtf(R.co.sc[a]) : 0.f; };
    if (SC) {
      R.co.sc[o] = inv(o);
    } else {
      R.co.ce[o] *= inv(o) * inv(o + 1);
      R.co.cs[o] *= inv(o) * inv(o + G.L.P);
    }
  }
}

// cc = (p(S) - d^-1) rho on the black columns, and its share of r.z, which
// completes rho and beta.  A block holds a region of the plane (a tile
// and a rim of 2 (steps - 1) columns that the steps spoil, as in k_sor) in shared memory,
// a colour to itself; a thread keeps its columns' couplings and Chebyshev vectors in
// registers.  FP32: the correction is a preconditioner's.
constexpr int kCoEdge = 54, kCoThreads = 512;
constexpr int kCoHalf = kCoEdge * kCoEdge / 2, kCoPad = kCoEdge / 2 + 1;
constexpr int kCoOwn = (kCoHalf + kCoThreads - 1) / kCoThreads;

template <typename T>
__global__ void __launch_bounds__(kCoThreads, 2)
    k_rb_coarse(RbGeo R, SolverState* S, const T* __restrict__ rho, float* __restrict__ cc, int ntx,
                int nty, int inner) {
  __shared__ float field[2][kCoHalf + 2 * kCoPad];
  if (S->converged) return;
  const int IE = R.ie, JE = R.je, P = 2 * R.P2, plane = 2 * R.plane2;
  const int H = (kCoEdge - inner) / 2;
  double dot = 0.0;
  for (int e = threadIdx.x; e < 2 * (kCoHalf + 2 * kCoPad); e += kCoThreads) (&field[0][0])[e] = 0.f;
  for (int tile = blockIdx.x; tile < ntx * nty * RbCoarse::kModes; tile += gridDim.x) {
    const int mode = tile / (ntx * nty), bx = tile % ntx, by = (tile / ntx) % nty;
    const int i0 = 2 + bx * inner, j0 = 2 + by * inner;
    const int i1 = min(IE - 1, i0 + inner - 1), j1 = min(JE - 1, j0 + inner - 1);
    const int ra = max(2, i0 - H), rb = min(IE - 1, i1 + H), rc = max(2, j0 - H), rd = min(JE - 1, j1 + H);
    const int nx = rb - ra + 1, ny = rd - rc + 1, hw = (nx + 1) / 2, odd = (ra + rc) & 1;
    const float *ce = R.co.ce + mode * plane, *cs = R.co.cs + mode * plane, *sc = R.co.sc + mode * plane;
    int own[2][kCoOwn], right[2][kCoOwn];
    float kw[2][kCoOwn], ke[2][kCoOwn], kn[2][kCoOwn], ks[2][kCoOwn];
    float b[kCoOwn], y[kCoOwn], dl[kCoOwn], res[kCoOwn];
    const float l = R.co.lmin[mode], th = 0.5f * (1.f + l), de = 0.5f * (1.f - l), s1 = th / de;
    float rn = 1.f / s1;
#pragma unroll
    for (int p = 0; p < 2; ++p)  // 0: red, i + j even
#pragma unroll
      for (int e = 0; e < kCoOwn; ++e) {
        const int t = threadIdx.x + e * kCoThreads, yy = t / hw, x = 2 * (t % hw) + ((yy + odd + p) & 1);
        const bool in = x < nx && yy < ny;
        const int i = ra + x, j = rc + yy, ij = in ? i + P * j : 0;
        own[p][e] = in ? kCoPad + yy * hw + x / 2 : -1;
        right[p][e] = kCoPad + yy * hw + (x + 1) / 2;
        kw[p][e] = in && x > 0 ? ce[ij - 1] : 0.f;
        ke[p][e] = in && x < nx - 1 ? ce[ij] : 0.f;
        kn[p][e] = in && yy > 0 ? cs[ij - P] : 0.f;
        ks[p][e] = in && yy < ny - 1 ? cs[ij] : 0.f;
        if (p == 1) {
          b[e] = in ? sc[ij] * (float)rho[mode * R.plane2 + (i >> 1) + R.P2 * j] : 0.f;
          res[e] = b[e];
          dl[e] = b[e] / th;
          y[e] = dl[e];
        }
      }
    __syncthreads();  // the last tile's readers are done
    auto sum = [&](int p, int e) {
      const float* f = field[1 - p];
      const int q = own[p][e], r = right[p][e];
      return kw[p][e] * f[r - 1] + ke[p][e] * f[r] + kn[p][e] * f[q - hw] + ks[p][e] * f[q + hw];
    };
    for (int k = 1; k < R.co.steps[mode]; ++k) {
#pragma unroll
      for (int e = 0; e < kCoOwn; ++e)
        if (own[1][e] >= 0) field[1][own[1][e]] = dl[e];
      __syncthreads();
#pragma unroll
      for (int e = 0; e < kCoOwn; ++e)
        if (own[0][e] >= 0) field[0][own[0][e]] = sum(0, e);
      __syncthreads();
      const float rp = rn;
      rn = 1.f / (2.f * s1 - rp);
#pragma unroll
      for (int e = 0; e < kCoOwn; ++e)
        if (own[1][e] >= 0) {
          res[e] -= dl[e] - sum(1, e);
          dl[e] = rn * rp * dl[e] + (2.f * rn / de) * res[e];
          y[e] += dl[e];
        }
    }
#pragma unroll
    for (int e = 0; e < kCoOwn; ++e) {
      const int t = threadIdx.x + e * kCoThreads, yy = t / hw, x = 2 * (t % hw) + ((yy + odd + 1) & 1);
      const int i = ra + x, j = rc + yy;
      if (own[1][e] >= 0 && i >= i0 && i <= i1 && j >= j0 && j <= j1) {
        const int s2 = mode * R.plane2 + (i >> 1) + R.P2 * j;
        const float c = -sc[i + P * j] * (R.co.gain[mode] * y[e] - b[e]);  // the operator is negative
        cc[s2] = c;
        dot += (double)rho[s2] * (double)c;
      }
    }
    __syncthreads();
  }
  double v[1] = {dot};
  if (grid_sum<1, kCoThreads>(v, S)) {
    const double rz = S->rz + v[0];
    S->beta = S->iter == 0 ? 0.0 : rz / S->rho;
    S->rho = rz;
    if (S->converged == 0 && !(rz == rz)) S->converged = 2;
  }
}

// ------------------------------------------------------- small grids -----
// The whole PCG loop in one cooperative kernel, a block per tile: the block keeps
// its red and its black tile in shared memory from the first iteration to the
// last, and only u and z go through L2, to the neighbouring tiles.  The three
// kernels of an iteration cost some 10 us each on such grids whatever the
// work (launch, first loads, last block's sum); here a phase ends with a grid-wide barrier that also carries
// its dot products.  The arithmetic and the order of the sums are those of
// the three kernels with a block per tile.  Waits are bounded by a clock budget
// (converged = 4).
struct GridSync {
  SolverState* S;
  long long limit;  // the kernel's argument: a load in the polling loop costs 4 % of a slice's step
  unsigned target;
  bool ok;
};

// All blocks' values added in block order, the same total for every thread of
// the grid (NV = 0: the barrier alone).
template <int NV, int NT>
__device__ __forceinline__ void grid_all(double (&v)[NV ? NV : 1], GridSync& g, int slot) {
  constexpr int kWarps = NT / 32;
  __shared__ double sh[NV ? NV : 1][kWarps];
  __shared__ bool up;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  SolverState* S = g.S;
  auto block_sum = [&]() {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double x = v[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) sh[q][warp] = x;
    }
    __syncthreads();
  };
  block_sum();
  g.target += gridDim.x;
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double x = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) x += sh[q][w];
      S->partials[(size_t)(slot + q) * S->max_blocks + blockIdx.x] = x;
    }
    __threadfence();
    atomicAdd(&S->gbar, 1u);
    const long long t0 = clock64();
    bool there = false;
    while (!there) {
      unsigned n;
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(n) : "l"(&S->gbar) : "memory");
      there = (int)(n - g.target) >= 0;
      if (!there && clock64() - t0 >= g.limit) break;
    }
    up = there;
  }
  __syncthreads();
  g.ok = up;
  if constexpr (NV == 0) return;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const double* part = S->partials + (size_t)(slot + q) * S->max_blocks;
    double x = 0.0;
#pragma unroll 4
    for (int b = tid; b < (int)gridDim.x; b += NT) x += __ldcg(part + b);
    v[q] = x;
  }
  block_sum();
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double x = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) x += sh[q][w];
    v[q] = x;
  }
  __syncthreads();
}

template <typename Ln>
constexpr size_t small_smem() {
  return (size_t)Ln::ROWS * Ln::W * (sizeof(typename Ln::V) * 6 + sizeof(float));
}

template <typename Ln, typename T = typename Ln::V>
__global__ void __launch_bounds__(Ln::NT, sizeof(T) == 4 ? 2 : (Ln::L <= 6 ? 4 : 3))
    k_rb_small(RbGeo R, SolverState* S, RbVectors<T> vec,
                                                     int ntiles, int nt, int maxit, long long limit) {
  constexpr int W = Ln::W, LC = Ln::L, N = Ln::ROWS * W;
  extern __shared__ __align__(128) unsigned char dsm[];
  __shared__ T szw[Ln::ROWS + 1], siz[Ln::ROWS + 1];
  __shared__ Scan<Ln> scan;
  T* zt = reinterpret_cast<T*>(dsm);  // z, u, p: the tile as its neighbouring threads see it
  T *ut = zt + N, *ps = ut + N, *xs = ps + N, *rs = xs + N, *ds = rs + N;
  float* db = reinterpret_cast<float*>(ds + N);
  if (S->converged) return;
  const Ln t;
  const Tiles<Ln> reds{R, R.col[0], t, ntiles, nt, true}, blacks{R, R.col[1], t, ntiles, nt, false};
  const Tile a = reds.at(blockIdx.x, reds.kk(blockIdx.x));
  const Tile k = blacks.at(blockIdx.x, blacks.kk(blockIdx.x));
  load_tables<Ln>(R, szw, siz);
  const int row = nt * R.ke * W;
  const int me = t.K0 * W + t.c;
  const int kba = wet_levels(a.kk, 0), kbk = wet_levels(k.kk, 0);
  auto s2 = [&](const Tile& q) { return q.kk ? q.m + R.P2 * q.j : 0; };
  const double2 we0 = R.col[0].we[s2(a)], ns0 = R.col[0].ns[s2(a)], iz0 = R.col[0].iz[s2(a)];
  const double2 we1 = R.col[1].we[s2(k)], ns1 = R.col[1].ns[s2(k)], iz1 = R.col[1].iz[s2(k)];
  const T zwa0 = kba ? (T)R.col[0].zw[s2(a)].x : T(0);
  const double2 zw1 = R.col[1].zw[s2(k)];
  const T zwa1 = kbk ? (T)zw1.x : T(0);
#pragma unroll
  for (int q = 0; q < LC; ++q) {
    const int K = t.K0 + 1 + q, o = me + W * q;
    zt[o] = K <= kbk ? vec.z[k.o0 + W * q] : T(0);
    rs[o] = K <= kbk ? vec.r[k.o0 + W * q] : T(0);
    db[o] = K <= kbk ? vec.db[k.o0 + W * q] : 0.f;
    ds[o] = K <= kba ? vec.dr[a.o0 + W * q] : T(0);
    ut[o] = ps[o] = xs[o] = T(0);
  }
  __syncthreads();
  // C v of the thread's levels without 1/ZP: the tile itself from shared memory,
  // its neighbours' tiles from L2 (written by other blocks before the last barrier)
  auto neighbours = [&](const Tile& q, int kb, const T* tile, const T* all, double2 we, double2 ns,
                        T (&h)[LC]) {
    const T cw = (T)we.x, ce = (T)we.y, cn = (T)ns.x, cs = (T)ns.y;
    const T co = q.sh ? cw : ce, cx = q.sh ? ce : cw;
    const bool across = t.c == (q.sh ? W - 1 : 0);
    const int cc = (q.sh ? min(t.c + 1, W - 1) : max(t.c - 1, 0)) - t.c;
    const int ko = across && (q.sh ? q.b + 1 < nt : q.b > 0) ? kb : 0;
    const int oo = q.o0 + (q.sh ? R.ke * W - (W - 1) : (W - 1) - R.ke * W);
    const int kn = min(kb, wet_levels(q.kk, 3)), ks = min(kb, wet_levels(q.kk, 4));
    T vn[LC], vs[LC], vo[LC];
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      const int K = t.K0 + 1 + e;
      vn[e] = K <= kn ? __ldcg(all + q.o0 - row + W * e) : T(0);
      vs[e] = K <= ks ? __ldcg(all + q.o0 + row + W * e) : T(0);
      vo[e] = K <= ko ? __ldcg(all + oo + W * e) : T(0);
    }
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      h[e] = co * tile[me + W * e];
      const T x = across ? vo[e] : tile[me + W * e + cc];
      h[e] = fma(cx, x, h[e]);
      h[e] = fma(cn, vn[e], h[e]);
      h[e] = fma(cs, vs[e], h[e]);
      if (t.K0 + 1 + e > kb) h[e] = T(0);
    }
  };
  GridSync g{S, limit, 0u, true};
  double rho = S->rho, rr = S->rr, alpha = 0.0, beta = 0.0;
  const double tol = S->tol, bb = S->bb;
  int iter = 0, conv = 0;
  while (!conv && iter < maxit) {
    // ---- red: u = D^-1 C z + beta u
    T h[LC], d[LC], cp[LC + 1];
    neighbours(a, kba, zt, vec.z, we0, ns0, h);
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      const int K = t.K0 + 1 + q;
      h[q] *= K == kba ? (T)iz0.y : (K == kba - 1 ? (T)iz0.x : siz[t.K0 + q]);
      d[q] = ds[me + W * q];
    }
    T dm = t.K0 > 0 ? ds[me - W] : T(0);
    couplings(t, szw, kba, zwa0, cp);
    column_solve(t, scan, h, d, dm, cp, [] { __syncthreads(); });
#pragma unroll
    for (int q = 0; q < LC; ++q)
      if (t.K0 + 1 + q <= kba) {
        const T u = beta != 0.0 ? fma((T)beta, ut[me + W * q], h[q]) : h[q];
        ut[me + W * q] = u;
        vec.u[a.o0 + W * q] = u;
      }
    // ---- black: x += alpha p, p = z + beta p (both of this block alone)
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      const int o = me + W * q;
      const T po = ps[o];
      xs[o] = fma((T)alpha, po, xs[o]);
      ps[o] = fma((T)beta, po, zt[o]);
    }
    double none[1];
    grid_all<0, Ln::NT>(none, g, 0);
    if (!g.ok) break;
    // q = D p - C u
    neighbours(k, kbk, ut, vec.u, we1, ns1, h);
    T qv[LC];
    Dot<T> pqt;
    {
      const T cw = (T)we1.x, ce = (T)we1.y, cn = (T)ns1.x, cs = (T)ns1.y;
      const int kbw = wet_levels(k.kk, 1), kbe = wet_levels(k.kk, 2);
      const int kbn = wet_levels(k.kk, 3), kbs = wet_levels(k.kk, 4);
      T pu = t.K0 > 0 ? ps[me - W] : T(0);
      const T pb = t.g < Ln::GROUPS - 1 ? ps[me + W * LC] : T(0);
#pragma unroll
      for (int e = 0; e < LC; ++e) {
        const int K = t.K0 + 1 + e;
        const T p0 = ps[me + W * e], pd = e + 1 < LC ? ps[me + W * (e + 1)] : pb;
        T dh = K <= kbw ? cw : T(0);
        dh += K <= kbe ? ce : T(0);
        dh += K <= kbn ? cn : T(0);
        dh += K <= kbs ? cs : T(0);
        const T hh = fma(dh, p0, h[e]);
        const T hs = K == kbk ? (T)iz1.y : (K == kbk - 1 ? (T)iz1.x : siz[t.K0 + e]);
        const T zw0 = K == kbk ? zwa1 : szw[t.K0 + e];
        T zwn = K + 1 == kbk ? zwa1 : szw[t.K0 + e + 1];
        if (K == kbk) zwn = K == 1 ? (T)zw1.y : T(0);
        T s = zw0 * (pu - p0);
        s = fma(zwn, pd - p0, s);
        s = fma(-hs, hh, s);
        qv[e] = K <= kbk ? s : T(0);
        pqt.add(e, p0, qv[e]);
        pu = p0;
      }
    }
    double w1[1] = {pqt.total()};
    grid_all<1, Ln::NT>(w1, g, 0);
    if (!g.ok) break;
    alpha = rho / w1[0];
    if (!(w1[0] > 0.0) && !(w1[0] < 0.0)) {
      conv = 3;
      alpha = 0.0;  // breakdown: x keeps the last full step
      break;
    }
    // ---- column: r -= alpha q, z = D^-1 r
    Dot<T> rrt;
#pragma unroll
    for (int e = 0; e < LC; ++e) {
      h[e] = fma(-(T)alpha, qv[e], rs[me + W * e]);
      rs[me + W * e] = h[e];
      rrt.add(e, h[e], h[e]);
      d[e] = (T)db[me + W * e];
    }
    dm = t.K0 > 0 ? (T)db[me - W] : T(0);
    couplings(t, szw, kbk, zwa1, cp);
    const double rz = column_solve(t, scan, h, d, dm, cp, [] { __syncthreads(); });
#pragma unroll
    for (int e = 0; e < LC; ++e)
      if (t.K0 + 1 + e <= kbk) {
        zt[me + W * e] = h[e];
        vec.z[k.o0 + W * e] = h[e];
      }
    double w2[2] = {rz, rrt.total()};
    grid_all<2, Ln::NT>(w2, g, 1);
    if (!g.ok) break;
    beta = w2[0] / rho;
    rho = w2[0];
    rr = w2[1];
    ++iter;
    if (sqrt(rr) <= tol * sqrt(bb)) conv = 1;
    if (!(rho == rho) || !(rr == rr)) conv = 2;  // NaN: stop
  }
  if (!g.ok) conv = 4;
  // x without its last update, which k_rb_after makes with p and alpha_prev
#pragma unroll
  for (int q = 0; q < LC; ++q)
    if (t.K0 + 1 + q <= kbk) {
      vec.x[k.o0 + W * q] = xs[me + W * q];
      vec.p[k.o0 + W * q] = ps[me + W * q];
    }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S->iter = iter;
    S->rho = rho;
    S->rr = rr;
    S->beta = beta;
    S->alpha_prev = alpha;
    if (conv != 4) S->converged = conv;
  }
  if (conv == 4 && threadIdx.x == 0) solve_gave_up(S);
}

// The black correction: the x update that the last iteration left open (none
// before the first, nor with alpha_prev = 0 after a breakdown, where p need not be
// finite), and its addition to the solution (full layout).
template <typename T>
__global__ void __launch_bounds__(128) k_rb_after(RbGeo R, SolverState* S, const T* __restrict__ p,
                                                  T* __restrict__ d, double* __restrict__ x) {
  const int W = R.width((int)sizeof(T));
  const int nb = R.nt(W), b = blockIdx.x % nb;
  const int m = 1 + b * W + threadIdx.x % W;
  const int K = blockIdx.z * (128 / W) + threadIdx.x / W + 1, j = blockIdx.x / nb + 2;
  if (m > R.M || K > wet_levels(R.col[1].kk[m + R.P2 * j], 0)) return;
  const int o = ((j * nb + b) * R.ke + K - 1) * W + threadIdx.x % W;
  const T alpha = (T)S->alpha_prev;
  T v = S->iter > 0 ? d[o] : T(0);
  if (S->iter > 0 && alpha != T(0)) v = fma(alpha, p[o], v);
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

// kResidLevels levels per thread: the levels of a column are independent here, so the
// blocks split them.  A thread that marches down a whole column waits for its loads
// level by level, 0.12 ms a launch on 256 x 256 x 60 and 0.06 on 512 x 1 x 60, now 0.09
// and 0.03; on 1024 x 1024 x 80, where columns are many, 1.41 ms against 1.55.  Bound by
// instructions: 280 a cell, 120 of them FP64, at 40 % of the issue slots.
constexpr int kResidLevels = 8, kResidThreads = 128;

__global__ void __launch_bounds__(kResidThreads) k_resid(Geo G, PoissonGeo P, SolverState* S,
                                                    const double* __restrict__ b,
                                                    double* __restrict__ x,
                                                    double* __restrict__ r, int nbx, int nby,
                                                    int ntiles) {
  const int KE = G.L.ke, IE = G.L.ie, JE = G.L.je;
  double rr = 0.0, bb = 0.0;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int bx = tile % nbx, by = (tile / nbx) % nby, bz = tile / (nbx * nby);
    const int i = bx * 32 + (threadIdx.x & 31) + 2, j = by * (kResidThreads / 32) + (threadIdx.x >> 5) + 2;
    const int K0 = bz * kResidLevels + 1, K1 = min(KE, K0 + kResidLevels - 1);
    if (i > IE - 1 || j > JE - 1) continue;
    const ColC c = load_col(G, P, i, j);
    // land rows (K > kb): diagonal only with a zero right-hand side, so the
    // solution there is 0 and x is set to it; r is neither stored nor read there
    for (int K = max(c.kb + 1, K0); K <= K1; ++K)
      if (AT(x, i, j, K) != 0.0) AT(x, i, j, K) = 0.0;
    double xm = 0.0, x0 = 0.0;
    if (K0 <= c.kb) {
      if (K0 > 1) xm = AT(x, i, j, K0 - 1);
      x0 = AT(x, i, j, K0);
    }
    // the loads of four levels are issued together; an entry that the reference
    // does not insert is 0 and its neighbour's value is not used
#pragma unroll 1
    for (int Kb = K0; Kb <= min(K1, c.kb); Kb += 4) {
      double vb[4], vw[4], ve[4], vn[4], vs[4], vd[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int K = min(Kb + e, c.kb);
        vb[e] = AT(b, i, j, K);
        vw[e] = AT(x, i - 1, j, K);
        ve[e] = AT(x, i + 1, j, K);
        vn[e] = AT(x, i, j - 1, K);
        vs[e] = AT(x, i, j + 1, K);
        vd[e] = AT(x, i, j, min(K + 1, c.kb));
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int K = Kb + e;
        if (K > min(K1, c.kb)) break;
        const Coef rw = row<false>(c, P, K, KE);
        DD s{vb[e], 0.0};
        if (rw.u != 0.0) dd_sub_prod(s, rw.u, xm);
        if (rw.n != 0.0) dd_sub_prod(s, rw.n, vn[e]);
        if (rw.w != 0.0) dd_sub_prod(s, rw.w, vw[e]);
        dd_sub_prod(s, rw.dc, x0);
        if (rw.e != 0.0) dd_sub_prod(s, rw.e, ve[e]);
        if (rw.s != 0.0) dd_sub_prod(s, rw.s, vs[e]);
        if (rw.d != 0.0) dd_sub_prod(s, rw.d, vd[e]);
        const double rk = s.hi + s.lo;
        AT(r, i, j, K) = rk;
        rr += rk * rk;
        bb += vb[e] * vb[e];
        xm = x0;
        x0 = vd[e];
      }
    }
  }
  double v[2] = {rr, bb};
  if (grid_sum<2, kResidThreads>(v, S)) {
    S->res_rr = v[0];
    S->res_bb = v[1];
  }
}

__global__ void k_set_limit(SolverState* S, int limit) { S->limit = limit; }

// the last node of the device-side PCG loop's body
__global__ void k_pcg_continue(cudaGraphConditionalHandle hc, const SolverState* S, int chunk) {
  cudaGraphSetConditional(hc, (S->converged == 0 && S->iter + chunk <= S->limit) ? 1u : 0u);
}

__global__ void k_reset(SolverState* S, double tol, bool first) {
  if (first) S->gave_up = 0;
  S->converged = 0;
  S->iter = 0;
  S->ticket = 0;
  S->gbar = 0;
  S->tol = tol;
  S->beta = 0.0;
  S->alpha_prev = 0.0;
  S->bb = 0.0;
}

__global__ void k_set_wait(SolverState* S, long long cycles) { S->wait = cycles; }

struct Shape {
  int ntiles, nt, grid;
};

// A persistent grid: as many blocks as run at once, each walking tiles.  The
// blocks per SM are asked for once per kernel and device, after the opt-in to
// the staging's shared memory (a fixed size per kernel).
constexpr int kMaxDevices = 64;

template <auto Kernel, typename L>
Shape shape_of(const RbGeo& R, size_t smem) {
  static std::atomic<int> per_sm[kMaxDevices];
  const int dev = R.device & (kMaxDevices - 1);
  int n = per_sm[dev].load(std::memory_order_acquire);
  if (!n) {
    cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, Kernel, L::NT, smem) != cudaSuccess || n < 1) n = 1;
    per_sm[dev].store(n, std::memory_order_release);
  }
  Shape s;
  s.nt = R.nt(L::W);
  s.ntiles = s.nt * (R.je - 2);
  s.grid = std::min({s.ntiles, n * R.sms, kMaxBlocks});
  return s;
}

// Calls f with the Lane type for columns of KE levels: 8 threads of 5 to 13
// levels, in longer columns more threads of 10, beyond 160 levels in tiles of half
// the width (a tile of six arrays has to fit shared memory).  A thread's
// registers hold some 4 values per level; with fewer levels per
// thread the work that a thread does once (its column's 2D data, the
// scan) outweighs its levels.
template <typename T, typename F>
void with_split(int ke, F&& f) {
  if (ke <= 40) f((Lane<T, 8, 5, 0>*)nullptr);
  else if (ke <= 48) f((Lane<T, 8, 6, 0>*)nullptr);
  else if (ke <= 64) f((Lane<T, 8, 8, 0>*)nullptr);
  else if (ke <= 80) f((Lane<T, 8, 10, 0>*)nullptr);
  else if (ke <= 88) f((Lane<T, 8, 11, 0>*)nullptr);
  else if (ke <= 104) f((Lane<T, 8, 13, 0>*)nullptr);
  else if (ke <= RbGeo::kWide) f((Lane<T, 16, 10, 0>*)nullptr);
  else f((Lane<T, 32, 10, 1>*)nullptr);
}
static_assert(32 * 10 >= kMaxKe && 16 * 10 >= RbGeo::kWide, "the longest column has a split");

}  // namespace

size_t rb_elements(const RbGeo& R, int elem_bytes) {
  const int W = R.width(elem_bytes);
  return (size_t)R.nt(W) * W * R.ke * (R.je + 1);
}
size_t rb_tiles(const RbGeo& R, int elem_bytes) {
  return (size_t)2 * R.nt(R.width(elem_bytes)) * (R.je + 1);
}

template <typename T>
void launch_rb_setup(const Geo& G, const PoissonGeo& P, const RbGeo& R, const RbVectors<T>& v,
                     cudaStream_t st) {
  const dim3 blk(32, 4);
  k_rb_setup<T><<<grid2(G.L.ie - 2, G.L.je - 2, blk), blk, 0, st>>>(G, P, R, v.dr, v.db, v.km);
  count_launch();
}

#define ORCTM_LANE(l) std::remove_pointer_t<decltype(l)>

template <typename T>
void launch_rb_before(const RbGeo& R, SolverState* S, const double* b, const RbVectors<T>& v,
                      cudaStream_t st) {
  with_split<T>(R.ke, [&](auto* l) {
    using L = ORCTM_LANE(l);
    constexpr size_t m1 = RedStage<L, kBefore>::smem, m2 = ColStage<L, true>::smem;
    const Shape s = shape_of<k_rb_red<L, kBefore>, L>(R, m1);
    k_rb_red<L, kBefore><<<s.grid, L::NT, m1, st>>>(R, S, (const T*)nullptr, v.ub, v.dr, v.km, b, nullptr,
                                                    (const float*)nullptr, s.ntiles, s.nt);
    const Shape c = shape_of<k_rb_col<L, true>, L>(R, m2);
    k_rb_col<L, true><<<c.grid, L::NT, m2, st>>>(R, S, v.r, (const T*)nullptr, v.z, v.db, v.km, b, v.ub,
                                                 v.coarse ? v.rho : (T*)nullptr, c.ntiles, c.nt);
  });
  add_launches(2);
}

template <typename T>
void launch_rb_red(const RbGeo& R, SolverState* S, const RbVectors<T>& v, cudaStream_t st) {
  with_split<T>(R.ke, [&](auto* l) {
    using L = ORCTM_LANE(l);
    constexpr size_t m = RedStage<L, kIter>::smem;
    const Shape s = shape_of<k_rb_red<L, kIter>, L>(R, m);
    k_rb_red<L, kIter><<<s.grid, L::NT, m, st>>>(R, S, v.z, v.u, v.dr, v.km, nullptr, nullptr,
                                                 v.coarse ? v.cc : (const float*)nullptr, s.ntiles, s.nt);
  });
  count_launch();
}

template <typename T>
void launch_rb_black(const RbGeo& R, SolverState* S, const RbVectors<T>& v, cudaStream_t st) {
  with_split<T>(R.ke, [&](auto* l) {
    using L = ORCTM_LANE(l);
    constexpr size_t m = BlackStage<L>::smem;
    const Shape s = shape_of<k_rb_black<L>, L>(R, m);
    k_rb_black<L><<<s.grid, L::NT, m, st>>>(R, S, v.z, v.u, v.p, v.x, v.q, v.km,
                                           v.coarse ? v.cc : (const float*)nullptr, s.ntiles, s.nt);
  });
  count_launch();
}

template <typename T>
void launch_rb_col(const RbGeo& R, SolverState* S, const RbVectors<T>& v, cudaStream_t st) {
  with_split<T>(R.ke, [&](auto* l) {
    using L = ORCTM_LANE(l);
    constexpr size_t m = ColStage<L, false>::smem;
    const Shape s = shape_of<k_rb_col<L, false>, L>(R, m);
    k_rb_col<L, false><<<s.grid, L::NT, m, st>>>(R, S, v.r, v.q, v.z, v.db, v.km, nullptr, (const T*)nullptr,
                                                 v.coarse ? v.rho : (T*)nullptr, s.ntiles, s.nt);
  });
  count_launch();
}

// The coarse correction of z; follows every k_rb_col of the iterations, and the first
template <typename T>
void launch_rb_coarse(const RbGeo& R, SolverState* S, const RbVectors<T>& v, cudaStream_t st) {
  if (!v.coarse) return;
  const int inner = kCoEdge - 4 * (std::max(R.co.steps[0], R.co.steps[1]) - 1);
  const int ntx = (R.ie - 2 + inner - 1) / inner, nty = (R.je - 2 + inner - 1) / inner;
  const long long n = (long long)ntx * nty * RbCoarse::kModes;
  k_rb_coarse<T><<<(int)std::min<long long>(n, kMaxBlocks), kCoThreads, 0, st>>>(R, S, v.rho, v.cc, ntx,
                                                                               nty, inner);
  count_launch();
}

// The 2D operators; co.mu (zeroed by the caller) tells how to use them (coarse_plan)
void launch_coarse_setup(const Geo& G, const PoissonGeo& P, const RbGeo& R, cudaStream_t st) {
  const dim3 blk(32, 4), gr = grid2(G.L.ie - 2, G.L.je - 2, blk);
  k_coarse_sums<<<gr, blk, 0, st>>>(G, P, R);
  k_coarse_mu<<<gr, blk, 0, st>>>(G, R);
  k_coarse_scale<false><<<gr, blk, 0, st>>>(G, R);
  k_coarse_scale<true><<<gr, blk, 0, st>>>(G, R);
  add_launches(4);
}

// The eigenvalues of a scaled S lie between 1 - mu^2 and 1.  Enough Chebyshev
// steps for an error of 0.15 on them, none below 0.05 (the few modes there are
// left to the iterations; more steps cost more than they save).  Where D alone
// leaves no eigenvalue below 0.5 it takes some ten iterations and the coarse space
// is not used.
void coarse_plan(RbCoarse& co, const float* mu) {
  co.on = 1.f - mu[0] * mu[0] < 0.5f;
  for (int q = 0; q < RbCoarse::kModes; ++q) {
    const double l = std::min(0.95, std::max(0.05, 1.0 - (double)mu[q] * mu[q]));
    const double a = std::acosh((1.0 + l) / (1.0 - l));
    co.steps[q] = std::max(1, (int)std::ceil(std::acosh(1.0 / 0.15) / a));
    co.lmin[q] = (float)l;
    co.gain[q] = (float)(1.0 / (1.0 - 1.0 / std::cosh(co.steps[q] * a)));
  }
}

template <typename T>
void launch_rb_after(const RbGeo& R, SolverState* S, const RbVectors<T>& v, double* x,
                     cudaStream_t st) {
  const int W = R.width((int)sizeof(T));
  const dim3 grid(R.nt(W) * (R.je - 2), 1, (R.ke + 128 / W - 1) / (128 / W));
  k_rb_after<T><<<grid, 128, 0, st>>>(R, S, v.p, v.x, x);
  with_split<T>(R.ke, [&](auto* l) {
    using L = ORCTM_LANE(l);
    constexpr size_t m = RedStage<L, kAfter>::smem;
    const Shape s = shape_of<k_rb_red<L, kAfter>, L>(R, m);
    k_rb_red<L, kAfter><<<s.grid, L::NT, m, st>>>(R, S, v.x, v.ub, v.dr, v.km, nullptr, x,
                                                  (const float*)nullptr, s.ntiles, s.nt);
  });
  add_launches(2);
}

// Whether the grid is small enough for k_rb_small: a tile per resident block, and
// columns of up to 104 levels (one shape of block).  It does without the coarse
// space: with it the separate kernels take as long at the largest such grids (97 x 131
// x 41: 1.9 ms a step both ways) and longer on a slice (640 x 1 x 50: 9.4 ms against 4.9).
template <typename T>
bool rb_small(const RbGeo& R) {
  bool fits = false;
  with_split<T>(R.ke, [&](auto* l) {
    using L = ORCTM_LANE(l);
    if constexpr (L::GROUPS == 8) {
      const Shape s = shape_of<k_rb_small<L>, L>(R, small_smem<L>());
      fits = s.grid >= s.ntiles;
    }
  });
  return fits;
}

template <typename T>
bool launch_rb_small(const RbGeo& R, SolverState* S, const RbVectors<T>& v, int maxit,
                     long long limit, cudaStream_t st) {
  bool done = false;
  with_split<T>(R.ke, [&](auto* l) {
    using L = ORCTM_LANE(l);
    if constexpr (L::GROUPS == 8) {
      constexpr size_t m = small_smem<L>();
      const Shape s = shape_of<k_rb_small<L>, L>(R, m);
      if (s.grid < s.ntiles) return;
      RbGeo r = R;
      RbVectors<T> vec = v;
      int ntiles = s.ntiles, nt = s.nt;
      void* args[] = {&r, &S, &vec, &ntiles, &nt, &maxit, &limit};
      done = cudaLaunchCooperativeKernel((const void*)&k_rb_small<L>, dim3(s.grid), dim3(L::NT), args,
                                         m, st) == cudaSuccess;
      if (done) count_launch();
      else (void)cudaGetLastError();  // the three kernels take its place
    }
  });
  return done;
}

#define ORCTM_RB(T)                                                                              \
  template bool rb_small<T>(const RbGeo&);                                                      \
  template bool launch_rb_small<T>(const RbGeo&, SolverState*, const RbVectors<T>&, int, long long, \
                                  cudaStream_t);                                                \
  template void launch_rb_setup<T>(const Geo&, const PoissonGeo&, const RbGeo&, const RbVectors<T>&, \
                                   cudaStream_t);                                                \
  template void launch_rb_before<T>(const RbGeo&, SolverState*, const double*, const RbVectors<T>&, \
                                    cudaStream_t);                                               \
  template void launch_rb_red<T>(const RbGeo&, SolverState*, const RbVectors<T>&, cudaStream_t); \
  template void launch_rb_black<T>(const RbGeo&, SolverState*, const RbVectors<T>&, cudaStream_t); \
  template void launch_rb_col<T>(const RbGeo&, SolverState*, const RbVectors<T>&, cudaStream_t); \
  template void launch_rb_coarse<T>(const RbGeo&, SolverState*, const RbVectors<T>&, cudaStream_t); \
  template void launch_rb_after<T>(const RbGeo&, SolverState*, const RbVectors<T>&, double*, cudaStream_t);
ORCTM_RB(double)
ORCTM_RB(float)
#undef ORCTM_RB

void launch_resid(const Geo& G, const PoissonGeo& P, SolverState* S, const double* b, double* x,
                  double* r, cudaStream_t st) {
  const int nbx = (G.L.ie - 2 + 31) / 32, nby = (G.L.je - 2 + kResidThreads / 32 - 1) / (kResidThreads / 32);
  const int nt = nbx * nby * ((G.L.ke + kResidLevels - 1) / kResidLevels);
  const int grid = std::min(nt, kMaxBlocks);
  k_resid<<<grid, kResidThreads, 0, st>>>(G, P, S, b, x, r, nbx, nby, nt);
  count_launch();
}

void launch_solver_reset(SolverState* S, double tol, bool first, cudaStream_t st) {
  k_reset<<<1, 1, 0, st>>>(S, tol, first);
  count_launch();
}

void launch_set_wait(SolverState* S, long long cycles, cudaStream_t st) {
  k_set_wait<<<1, 1, 0, st>>>(S, cycles);
  count_launch();
}

long long solver_wait_cycles() { return kWaitCycles; }

void launch_set_limit(SolverState* S, int limit, cudaStream_t st) {
  k_set_limit<<<1, 1, 0, st>>>(S, limit);
  count_launch();
}

void launch_pcg_continue(cudaGraphConditionalHandle hc, const SolverState* S, int chunk,
                         cudaStream_t st) {
  k_pcg_continue<<<1, 1, 0, st>>>(hc, S, chunk);
  count_launch();
}

int solver_max_blocks() { return kMaxBlocks; }

}  // namespace orctm
