// Tracer diffusion (OCTDIFF_BASE + OCTDIFF_TS: octdiff_base.f90:182-221,
// octdiff_ts.f90:51-59, 294-407) and momentum diffusion with quadratic
// bottom drag (OCVISC, FREESLIP branch: ocvisc.f90:37-478, 615-688).
//
// Implicit vertical diffusion is one tridiagonal solve per water column, by one
// thread for the tracers and u, v, shared by the threads of a block for w
// (tridiag.cuh).  The tracers' horizontal biharmonic operator is one
// fused pass (the first Laplacian formed per level in shared memory, never
// stored); the momentum one is two passes (a Laplacian into a scratch field,
// then the flux-form update).  Arithmetic follows the reference's operation order in IEEE binary64,
// with two changes that stay within a few ulp: the stencils multiply by
// reciprocal metrics and per-face coefficients computed once at set-up
// instead of dividing by the metrics, and the remaining divisions (by
// thicknesses and Thomas pivots) use div_nr (within 1 ulp of IEEE division).
#include <type_traits>

#include <algorithm>

#include "common.cuh"
#include "ops.h"
#include "tridiag.cuh"

namespace orctm {

namespace {

#define AT(a, i, j, K) (a)[G.L.at((i), (j), (K)-1)]

inline dim3 grid2(int nx, int ny, dim3 b) { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y, 1); }

// ------------------------------------------------------------- OCTDIFF ----
// Implicit vertical diffusion of ntr tracers (TRIDSY built once per column).
// Columns outside i in [2,IE1], j in [2,JE1] are copied unchanged.
struct TrPtrs {
  const double* in[8];
  double* out[8];
};

// The eliminated diagonals of a column solve are kept per thread (local
// memory, cached in L1/L2).  Keeping them in shared memory instead was
// measured 2.1-2.5x slower on c3: 640 B per column limits a B200 SM to about
// 350 resident columns, too few to hide the solves' memory latency.
constexpr int kVertBlock = 64;

__global__ void __launch_bounds__(kVertBlock) k_tdiff_vert(Geo G, TrPtrs tp, int ntr,
                                                           const double* __restrict__ dvo,
                                                           const double* __restrict__ zo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke;
  if (i > IE || j > JE) return;
  const bool interior = i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  if (!interior) {
    for (int n = 0; n < ntr; ++n)
      for (int K = 1; K <= KE; ++K) AT(tp.out[n], i, j, K) = AT(tp.in[n], i, j, K);
    return;
  }
  const int ij = G.L.at2(i, j);
  const double zij = zo[ij];
  // TRIDSY(K,1..3) of octdiff_base.f90:188-194; only the eliminated diagonal
  // is kept per level, TRIDSY(K,3) is recomputed by the same expression
  auto den = [&](int K) {
    const double zzsurf = K == 1 ? 1. : 0.;
    return thick(G.gp, G.dzw, ij, K) + zzsurf * (zij) + G.almzer;
  };
  auto tri3 = [&](int K, double dn) { return div_nr(-G.dt * AT(dvo, i, j, K + 1) * G.di[K], dn); };
  double t2p[kMaxKe];
  double ylast[8];
  double t2prev = 1.0, t3prev = 0.0;
  for (int K = 1; K <= KE; ++K) {
    const double dn = den(K);
    const double t1 = div_nr(-G.dt * AT(dvo, i, j, K) * wet(G.gp, ij, K) * G.di[K - 1], dn);
    const double t3 = tri3(K, dn);
    double t2 = 1. - t1 - t3;
    double m = 0.0;
    if (K >= 2) {
      m = div_nr(t1, t2prev);                       // TRIDSY(K-1,1) after elimination
      t2 = t2 - div_nr(t3prev * t1, t2prev);        // TRIDSY(K,2) after elimination
    }
    t2p[K - 1] = t2;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      if (n >= ntr) break;
      const double tk = AT(tp.in[n], i, j, K);
      const double y = K == 1 ? tk : tk - m * ylast[n];  // T1O(K)
      AT(tp.out[n], i, j, K) = y;
      ylast[n] = y;
    }
    t2prev = t2;
    t3prev = t3;
  }
  double nxt[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    if (n >= ntr) break;
    nxt[n] = div_nr(AT(tp.out[n], i, j, KE), t2p[KE - 1]);
    AT(tp.out[n], i, j, KE) = nxt[n];
  }
  for (int l = KE - 1; l >= 1; --l) {
    const double t3 = tri3(l, den(l));
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      if (n >= ntr) break;
      nxt[n] = div_nr(AT(tp.out[n], i, j, l) - t3 * nxt[n], t2p[l - 1]);
      AT(tp.out[n], i, j, l) = nxt[n];
    }
  }
}

// The same solve with the tracer count known at compile time and the loads
// of U levels issued together before they are used: the input and output
// arrays may alias as far as the compiler knows, so the one-level form above
// waits a full memory latency per level in each sweep.  Every value is
// formed by the same expressions in the same order, so the results equal
// k_tdiff_vert's bit for bit.
template <int NTR, int U>
__global__ void __launch_bounds__(kVertBlock) k_tdiff_vert_b(Geo G, TrPtrs tp,
                                                             const double* __restrict__ dvo,
                                                             const double* __restrict__ zo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke;
  if (i > IE || j > JE) return;
  const int pl = G.L.plane;
  const int base = G.L.at(i, j, 0);
  const bool interior = i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  if (!interior) {
    for (int K0 = 1; K0 <= KE; K0 += U) {
      double v[NTR][U];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int n = 0; n < NTR; ++n)
          v[n][u] = K0 + u <= KE ? tp.in[n][base + (K0 + u - 1) * pl] : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int n = 0; n < NTR; ++n)
          if (K0 + u <= KE) tp.out[n][base + (K0 + u - 1) * pl] = v[n][u];
    }
    return;
  }
  const int ij = G.L.at2(i, j);
  const double zij = zo[ij];
  auto den = [&](int K) {
    const double zzsurf = K == 1 ? 1. : 0.;
    return thick(G.gp, G.dzw, ij, K) + zzsurf * (zij) + G.almzer;
  };
  double t2p[kMaxKe];
  double ylast[NTR];
  double t2prev = 1.0, t3prev = 0.0;
  // forward elimination, U levels per batch: DVO(K..K+U) and the tracers of
  // K..K+U-1 are loaded first
  for (int K0 = 1; K0 <= KE; K0 += U) {
    double lt[NTR][U], ld[U + 1];
#pragma unroll
    for (int u = 0; u <= U; ++u) ld[u] = K0 + u <= KE + 1 ? dvo[base + (K0 + u - 1) * pl] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int n = 0; n < NTR; ++n)
        lt[n][u] = K0 + u <= KE ? tp.in[n][base + (K0 + u - 1) * pl] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int K = K0 + u;
      if (K > KE) break;
      const double dn = den(K);
      const double t1 = div_nr(-G.dt * ld[u] * wet(G.gp, ij, K) * G.di[K - 1], dn);
      const double t3 = div_nr(-G.dt * ld[u + 1] * G.di[K], dn);
      double t2 = 1. - t1 - t3;
      double m = 0.0;
      if (K >= 2) {
        m = div_nr(t1, t2prev);
        t2 = t2 - div_nr(t3prev * t1, t2prev);
      }
      t2p[K - 1] = t2;
#pragma unroll
      for (int n = 0; n < NTR; ++n) {
        const double tk = lt[n][u];
        const double y = K == 1 ? tk : tk - m * ylast[n];
        tp.out[n][base + (K - 1) * pl] = y;
        ylast[n] = y;
      }
      t2prev = t2;
      t3prev = t3;
    }
  }
  // back substitution, U levels per batch: the forward values and DVO of
  // l-U+1..l loaded first
  double nxt[NTR];
#pragma unroll
  for (int n = 0; n < NTR; ++n) {
    nxt[n] = div_nr(ylast[n], t2p[KE - 1]);
    tp.out[n][base + (KE - 1) * pl] = nxt[n];
  }
  for (int l0 = KE - 1; l0 >= 1; l0 -= U) {
    double ly[NTR][U], ld[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = l0 - u;
      ld[u] = l >= 1 ? dvo[base + l * pl] : 0.0;  // DVO(l+1)
#pragma unroll
      for (int n = 0; n < NTR; ++n) ly[n][u] = l >= 1 ? tp.out[n][base + (l - 1) * pl] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = l0 - u;
      if (l < 1) break;
      const double t3 = div_nr(-G.dt * ld[u] * G.di[l], den(l));
#pragma unroll
      for (int n = 0; n < NTR; ++n) {
        nxt[n] = div_nr(ly[n][u] - t3 * nxt[n], t2p[l - 1]);
        tp.out[n][base + (l - 1) * pl] = nxt[n];
      }
    }
  }
}

// Laplacian and biharmonic update fused (octdiff_ts.f90:342-399), all
// tracers in one launch.  A block of 32 x 8 cells marches down the levels;
// per level it stages the 36 x 12 tile of the vertically diffused tracer in
// shared memory, forms the masked Laplacian T1O on the 34 x 10 positions its
// cells need, and applies the biharmonic update, so the Laplacian never goes
// to HBM.  The geometry a thread needs (wet-level counts, reciprocal metrics,
// face terms) is loaded once for all levels and tracers, and the loads of the
// next level are issued before the current one is computed.  The Laplacian
// (0 outside the interior) and the biharmonic factor W / ((DDPO + ALMZER +
// ZZSURF ZO) DLXP DLYP) DZW use 1/(DLXP DLYP), reciprocal metrics and the
// face terms AULX DLYU / DLXU and AULY DLXV / DLYV precomputed, multiplied in
// the reference's order.  The blocks cover i in [1, IE], j in [1, JE]: cells
// outside the interior are copied.  (Measured on c3: one launch per level,
// reloading the geometry each time, was 2.1x slower than this form.)
constexpr int kHbX = 32, kHbY = 8;
constexpr int kHbTx = kHbX + 4, kHbTy = kHbY + 4;   // tracer tile
constexpr int kHbLx = kHbX + 2, kHbLy = kHbY + 2;   // Laplacian tile
constexpr int kHbT = kHbTx * kHbTy, kHbL = kHbLx * kHbLy, kHbN = kHbX * kHbY;
constexpr int kHbTf = (kHbT + kHbN - 1) / kHbN, kHbLf = (kHbL + kHbN - 1) / kHbN;

template <bool SPLIT>
__global__ void __launch_bounds__(kHbN) k_tdiff_hbih(Geo G, TrPtrs tp, int ntr, int levels,
                                                     const double* __restrict__ zo) {
  __shared__ double ts[kHbT];
  __shared__ double ls[kHbL];
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + kHbX * ty;
  const int i0 = blockIdx.x * kHbX + 1, j0 = blockIdx.y * kHbY + 1;
  const int plane = G.L.plane;
  // tracer-tile entries this thread loads (element (i0-2+hx, j0-2+hy));
  // entries outside the field's plane [0, IE] x [0, JE] are not loaded and
  // hold 0 (no Laplacian or update that is formed reads them)
  int toff[kHbTf];
  bool tval[kHbTf], tin[kHbTf];
#pragma unroll
  for (int f = 0; f < kHbTf; ++f) {
    const int e = tid + f * kHbN;
    const int hy = e / kHbTx, hx = e - hy * kHbTx;
    const int ii = i0 - 2 + hx, jj = j0 - 2 + hy;
    tval[f] = e < kHbT;
    tin[f] = tval[f] && ii >= 0 && ii <= IE && jj >= 0 && jj <= JE;
    toff[f] = tin[f] ? G.L.at2(ii, jj) : 0;
  }
  // Laplacian positions this thread forms, with their level-independent data
  struct LapPos {
    int e, c, kb, w, ea, n, s;
    bool in;
    double rxw, rxe, rxp, ryn, rys, ryp;
  };
  LapPos lp[kHbLf];
#pragma unroll
  for (int f = 0; f < kHbLf; ++f) {
    LapPos& L = lp[f];
    L.e = tid + f * kHbN;
    const int hy = L.e / kHbLx, hx = L.e - hy * kHbLx;
    const int i = i0 - 1 + hx, j = j0 - 1 + hy;
    L.in = L.e < kHbL && i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
    L.c = (hy + 1) * kHbTx + (hx + 1);
    if (L.in) {
      const int ij = G.L.at2(i, j);
      L.kb = G.gp.kb[ij];
      L.w = G.gp.kb[G.L.at2(i - 1, j)];
      L.ea = G.gp.kb[G.L.at2(i + 1, j)];
      L.n = G.gp.kb[G.L.at2(i, j - 1)];
      L.s = G.gp.kb[G.L.at2(i, j + 1)];
      L.rxw = G.rdlxu[G.L.at2(i - 1, j)];
      L.rxe = G.rdlxu[ij];
      L.rxp = G.rdlxp[ij];
      L.ryn = G.rdlyv[G.L.at2(i, j - 1)];
      L.rys = G.rdlyv[ij];
      L.ryp = G.rdlyp[ij];
    }
  }
  // this thread's cell
  const int i = i0 + tx, j = j0 + ty;
  const bool cell = i <= IE && j <= JE;
  const bool inner = cell && i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  int kbc = 0, kbw = 0, kbe = 0, kbn = 0, kbs = 0;
  double tfw = 0, tfe = 0, tfn = 0, tfs = 0, rar = 0, bot = 0, zc = 0;
  if (inner) {
    const int ijc = G.L.at2(i, j);
    kbc = G.gp.kb[ijc];
    kbw = G.gp.kb[G.L.at2(i - 1, j)];
    kbe = G.gp.kb[G.L.at2(i + 1, j)];
    kbn = G.gp.kb[G.L.at2(i, j - 1)];
    kbs = G.gp.kb[G.L.at2(i, j + 1)];
    tfw = G.tfx[G.L.at2(i - 1, j)];
    tfe = G.tfx[ijc];
    tfn = G.tfy[G.L.at2(i, j - 1)];
    tfs = G.tfy[ijc];
    rar = G.rareap[ijc];
    bot = G.gp.bot[ijc];
    zc = zo[ijc];
  }
  const int me_t = (ty + 2) * kHbTx + (tx + 2), me_l = (ty + 1) * kHbLx + (tx + 1);
  const int own = cell ? G.L.at(i, j, 0) : 0;
  auto wet_at = [](int kb, int K) { return K <= kb ? 1.0 : 0.0; };
  // all tracers and levels, or (SPLIT) a tracer and a part of the levels
  const int n0 = SPLIT ? blockIdx.z % ntr : 0, n1 = SPLIT ? n0 + 1 : ntr;
  const int K0 = SPLIT ? 1 + (blockIdx.z / ntr) * levels : 1;
  const int K1 = SPLIT ? min(KE, K0 + levels - 1) : KE;
  for (int n = n0; n < n1; ++n) {
    const double* __restrict__ T = tp.in[n];
    double* __restrict__ O = tp.out[n];
    double nx[kHbTf];
  #pragma unroll
    for (int f = 0; f < kHbTf; ++f) nx[f] = tin[f] ? T[toff[f] + plane * (K0 - 1)] : 0.0;
    for (int K = K0; K <= K1; ++K) {
      __syncthreads();  // the previous level's tiles are no longer read
  #pragma unroll
      for (int f = 0; f < kHbTf; ++f)
        if (tval[f]) ts[tid + f * kHbN] = nx[f];
      if (K < K1) {
  #pragma unroll
        for (int f = 0; f < kHbTf; ++f)
          if (tin[f]) nx[f] = T[toff[f] + plane * K];
      }
      __syncthreads();
  #pragma unroll
      for (int f = 0; f < kHbLf; ++f) {
        const LapPos& L = lp[f];
        if (L.e >= kHbL) continue;
        double r = 0.0;
        if (L.in) {
          const double c = ts[L.c];
          r = wet_at(L.kb, K) *
              ((wet_at(L.w, K) * (ts[L.c - 1] - c) * L.rxw +
                wet_at(L.ea, K) * (ts[L.c + 1] - c) * L.rxe) *
                   L.rxp +
               (wet_at(L.n, K) * (ts[L.c - kHbTx] - c) * L.ryn +
                wet_at(L.s, K) * (ts[L.c + kHbTx] - c) * L.rys) *
                   L.ryp);
        }
        ls[L.e] = r;
      }
      __syncthreads();
      if (cell) {
        const double t = ts[me_t];
        double r = t;
        if (inner) {
          const double zzsurf = K == 1 ? 1. : 0.;
          const double c = ls[me_l];
          const double th = K < kbc ? G.dzw[K - 1] : (K == kbc ? bot : 0.0);
          const double fac = div_nr(wet_at(kbc, K) * rar, th + G.almzer + zzsurf * (zc));
          r = t - fac * G.dzw[K - 1] *
                      (wet_at(kbw, K) * tfw * (ls[me_l - 1] - c) +
                       wet_at(kbe, K) * tfe * (ls[me_l + 1] - c) +
                       wet_at(kbn, K) * tfn * (ls[me_l - kHbLx] - c) +
                       wet_at(kbs, K) * tfs * (ls[me_l + kHbLx] - c));
        }
        O[own + plane * (K - 1)] = r;
      }
    }
  }
}

// -------------------------------------------------------------- OCVISC ----
// Infinities and NaN on land.  A mask is a factor 0 in the reference's expressions, and
// 0 times such a value is NaN, in its own cell and in its neighbours.  The horizontal
// passes do not load land cells unless the vertical solves, which write every level,
// have met a value that is not finite: they note it at `bad` (element (0, 0) of SPEEDU,
// no u-point, which k_visc_speed clears).
// bottom speeds SPEEDU/SPEEDV (ocvisc.f90:53-104): evaluated at the single
// level where the mask drops from 1 to 0 (or at KE when the column is full)
__global__ void k_visc_speed(Geo G, const double* __restrict__ uoo, const double* __restrict__ voe,
                             double* __restrict__ spu, double* __restrict__ spv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int IE = G.L.ie, JE = G.L.je;
  if (i > IE || j > JE) return;
  const int ij = G.L.at2(i, j);
  double su = 0., sv = 0.;
  if (i >= 1 && i <= IE - 1 && j >= 2 && j <= JE - 1) {
    const int K = G.gu.kb[ij];
    if (K >= 1) {
      const double a = 0.25 * (AT(voe, i, j, K) + AT(voe, i + 1, j, K) + AT(voe, i, j - 1, K) +
                               AT(voe, i + 1, j - 1, K));
      const double u = AT(uoo, i, j, K);
      su = fmx(sqrt(u * u + a * a), 1.E-3);
    }
  }
  if (i >= 2 && i <= IE - 1 && j >= 1 && j <= JE - 1) {
    const int K = G.gv.kb[ij];
    if (K >= 1) {
      const double a = 0.25 * (AT(uoo, i, j, K) + AT(uoo, i - 1, j, K) + AT(uoo, i, j + 1, K) +
                               AT(uoo, i - 1, j + 1, K));
      const double v = AT(voe, i, j, K);
      sv = fmx(sqrt(v * v + a * a), 1.E-3);
    }
  }
  spu[ij] = su;
  spv[ij] = sv;
}

// implicit vertical diffusion of u (DIR = 0, ocvisc.f90:168-218) or v
// (DIR = 1, ocvisc.f90:114-165) with quadratic bottom drag in the last row.
// The loads of U levels are issued together before they are used (X and AVO of
// both columns in the forward sweep, the forward values and AVO in the
// backward one).  The tracers and u, v keep the reference's elimination level
// by level: the scans of tridiag.cuh differ from it in the last digits, which the
// convective switches of the whole step amplify (to 4e-8 of u after twenty
// steps of the laboratory tank, where this form stays bit for bit).
// Both directions are one launch, the grid's z index: 256 x 256 columns fill a fifth
// of the chip's warps.
template <int DIR, int U>
__device__ __forceinline__ void visc_uv(const Geo& G, const double* __restrict__ X,
                                        const double* __restrict__ keep,
                                        const double* __restrict__ avo,
                                        const double* __restrict__ speed, double* __restrict__ O,
                                        double* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke;
  if (i > IE || j > JE) return;
  bool ok = true;
  const bool interior = DIR == 0 ? (i >= 1 && i <= IE - 1 && j >= 2 && j <= JE - 1)
                                 : (i >= 2 && i <= IE - 1 && j >= 1 && j <= JE - 1);
  const bool valid = DIR == 0 ? (j >= 1) : (i >= 1);
  if (!valid) return;
  const int pl = G.L.plane;
  const int base = G.L.at(i, j, 0);
  if (!interior) {
    for (int K = 1; K <= KE; ++K) {
      const double v = keep[base + (K - 1) * pl];
      ok &= finite(v);
      O[base + (K - 1) * pl] = v;
    }
    if (!ok) *bad = 1.;
    return;
  }
  const ColGeo& cg = DIR == 0 ? G.gu : G.gv;
  const int ij = G.L.at2(i, j);
  const int ij2 = DIR == 0 ? G.L.at2(i + 1, j) : G.L.at2(i, j + 1);
  const double BOFRIC = 3.E-3, RAYFRIC = 3.E-3;
  const double sp = speed[ij];
  // TRIDSY(K,1) and TRIDSY(K,3) from AVO of levels K (a0, b0) and K+1 (a1, b1)
  // of the two columns
  auto tri = [&](int K, double a0, double b0, double a1, double b1, double& t1, double& t3) {
    const double am = wet(cg, ij, K), dd = thick(cg, G.dzw, ij, K);
    const double avup = 0.5 * (a0 + b0) * am;
    if (K < KE) {
      const double am1 = wet(cg, ij, K + 1);
      const double avlo = 0.5 * (a1 + b1) * am1 + (BOFRIC + RAYFRIC * dd * sp) * (am - am1);
      t1 = div_nr(-G.dt * avup * am * G.di[K - 1], G.almzer + dd);
      t3 = div_nr(-G.dt * avlo * am * G.di[K], G.almzer + dd);
    } else {
      const double avlo = (BOFRIC + RAYFRIC * dd * sp) * am;
      t1 = div_nr(-G.dt * avup * am * G.di[K - 1], G.almzer + dd);
      t3 = div_nr(-G.dt * avlo * am * G.di[K], G.almzer + dd);
    }
  };
  double t2p[kMaxKe];
  double t2prev = 1.0, t3prev = 0.0, yprev = 0.0;
  for (int K0 = 1; K0 <= KE; K0 += U) {
    double la[U + 1], lb[U + 1], lx[U];
#pragma unroll
    for (int u = 0; u <= U; ++u) {
      const bool ok = K0 + u <= KE;
      la[u] = ok ? avo[ij + (K0 + u - 1) * pl] : 0.0;
      lb[u] = ok ? avo[ij2 + (K0 + u - 1) * pl] : 0.0;
      if (u < U) lx[u] = ok ? X[base + (K0 + u - 1) * pl] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int K = K0 + u;
      if (K > KE) break;
      double t1, t3;
      tri(K, la[u], lb[u], la[u + 1], lb[u + 1], t1, t3);
      double t2 = 1. - t1 - t3;
      t3 = K < KE ? t3 * wet(cg, ij, K + 1) : 0.;
      const double xk = lx[u];
      double y = xk;
      if (K >= 2) {
        const double m = div_nr(t1, t2prev);
        t2 = t2 - div_nr(t3prev * t1, t2prev);
        y = xk - m * yprev;
      }
      t2p[K - 1] = t2;
      O[base + (K - 1) * pl] = y;
      yprev = y;
      t2prev = t2;
      t3prev = t3;
    }
  }
  double nxt = div_nr(wet(cg, ij, KE) * yprev, t2p[KE - 1]);
  ok &= finite(nxt);
  O[base + (KE - 1) * pl] = nxt;
  for (int l0 = KE - 1; l0 >= 1; l0 -= U) {
    double la[U], lb[U], la1[U], lb1[U], ly[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = l0 - u;
      const bool ok = l >= 1;
      la[u] = ok ? avo[ij + (l - 1) * pl] : 0.0;
      lb[u] = ok ? avo[ij2 + (l - 1) * pl] : 0.0;
      la1[u] = ok ? avo[ij + l * pl] : 0.0;
      lb1[u] = ok ? avo[ij2 + l * pl] : 0.0;
      ly[u] = ok ? O[base + (l - 1) * pl] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = l0 - u;
      if (l < 1) break;
      double t1, t3;
      tri(l, la[u], lb[u], la1[u], lb1[u], t1, t3);
      t3 = t3 * wet(cg, ij, l + 1);
      nxt = div_nr((ly[u] - t3 * nxt) * wet(cg, ij, l), t2p[l - 1]);
      ok &= finite(nxt);
      O[base + (l - 1) * pl] = nxt;
    }
  }
  if (!ok) *bad = 1.;
}
template <int U>
__global__ void __launch_bounds__(kVertBlock) k_visc_uv_b(Geo G, const double* __restrict__ xu,
                                                          const double* __restrict__ xv,
                                                          const double* __restrict__ keepu,
                                                          const double* __restrict__ keepv,
                                                          const double* __restrict__ avo,
                                                          const double* __restrict__ spu,
                                                          const double* __restrict__ spv,
                                                          double* __restrict__ ou,
                                                          double* __restrict__ ov, double* bad) {
  if (blockIdx.z == 0) visc_uv<0, U>(G, xu, keepu, avo, spu, ou, bad);
  else visc_uv<1, U>(G, xv, keepv, avo, spv, ov, bad);
}

// implicit vertical diffusion of w, levels 2..KE (ocvisc.f90:225-270); the
// levels 1 and KEP are carried.  Row K of the solve is level K + 1.
// (Up to 48 levels two blocks fit an SM: 64 registers a thread.)
template <typename Ln>
__global__ void __launch_bounds__(Ln::NT, Ln::LC <= 3 ? 2 : 1) k_visc_w(Geo G, const double* __restrict__ Wi,
                                                   const double* __restrict__ avo,
                                                   double* __restrict__ O, double* bad) {
  constexpr int LC = Ln::LC;
  __shared__ TriScan<Ln, 1> scan;
  const Ln t;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke, pl = G.L.plane;
  const int nb = (IE + Ln::W) / Ln::W;
  const int i = blockIdx.x % nb * Ln::W + t.c, j = blockIdx.x / nb + 1;
  const bool valid = i >= 1 && i <= IE;
  const bool interior = i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  const int base = G.L.at(i, j, t.K0 + 1), ij = G.L.at2(i, j);  // level K0 + 2
  double x[1][LC], a[LC], b[LC], c[LC], av[LC + 2];
#pragma unroll
  for (int u = 0; u < LC + 2; ++u) {  // AVO of levels K0 + 1 ...
    const int K = t.K0 + 1 + u;
    av[u] = interior && K <= KE ? avo[base + (u - 1) * pl] : 0.;
  }
#pragma unroll
  for (int u = 0; u < LC; ++u) x[0][u] = valid && t.K0 + 2 + u <= KE ? Wi[base + u * pl] : 0.;
  if (valid && t.g == 0) {
    const int top = G.L.at(i, j, 0);
    O[top] = Wi[top];
    O[top + KE * pl] = Wi[top + KE * pl];
  }
  const int kb = interior ? G.gp.kb[ij] : 0;
  const double bot = interior ? G.gp.bot[ij] : 0.;
  auto thickness = [&](int K) { return K < kb ? G.dzw[K - 1] : (K == kb ? bot : 0.0); };
  auto den = [&](int K) { return 2.0 * G.almzer + thickness(K - 1) + thickness(K); };
  // TRIDSY(K,3) from AVO of levels K and K + 1
  auto lower = [&](int K, double a0, double a1, double dn, double rd) {
    const double avlo = K < KE && K <= kb ? 0.5 * (a1 + a0) : 0.0;
    return quotient(-2.0 * G.dt * avlo * G.di[K - 1], dn, rd);
  };
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    const int K = t.K0 + 2 + u;
    // land: the masks' factor 0 of the coefficients
    a[u] = 0. * (av[u] + av[u + 1]);
    c[u] = 0. * (av[u + 1] + av[u + 2]);
    b[u] = 1. - a[u] - c[u];
    if (K <= KE && K <= kb) {
      const double dn = den(K), rd = div_nr(1., dn);
      a[u] = quotient(-2.0 * G.dt * (0.5 * (av[u] + av[u + 1])) * G.di[K - 2], dn, rd);
      c[u] = lower(K, av[u + 1], av[u + 2], dn, rd);
      b[u] = 1. - a[u] - c[u];
      if (K == 2) a[u] = 0.;
    }
  }
  const int Kp = t.K0 + 1;  // the level above the thread's first
  const double cprev = Kp >= 2 && Kp < KE && Kp <= kb ? lower(Kp, av[0], av[1], den(Kp), div_nr(1., den(Kp))) : 0.;
  bool ok = true;
  if (valid && t.g == 0) ok = finite(Wi[G.L.at(i, j, 0)]);
  if (valid && !interior) {
#pragma unroll
    for (int u = 0; u < LC; ++u)
      if (t.K0 + 2 + u <= KE) {
        ok &= finite(x[0][u]);
        O[base + u * pl] = x[0][u];
      }
  }
  // levels below the bottom end as 0 (NaN where the mask's factor 0 gives it)
#pragma unroll
  for (int u = 0; u < LC; ++u)
    if (t.K0 + 2 + u > kb) x[0][u] = 0. * x[0][u];
  tri_solve<Ln, 1>(t, scan, a, b, c, cprev, x);
  if (interior) {
#pragma unroll
    for (int u = 0; u < LC; ++u)
      if (t.K0 + 2 + u <= KE) {
        ok &= finite(x[0][u]);
        O[base + u * pl] = x[0][u];
      }
  }
  if (!ok) *bad = 1.;
}

// The horizontal passes of OCVISC: a thread takes kViscLevels levels of a point,
// so the geometry of the point and its four neighbours (some 15 values for each
// staggering) is loaded once for them; the loads of four levels are issued together.
// (A thread per point and level reloaded it every level: 5.4 ms for the two
// passes on 1024 x 1024 x 80.)  Where a neighbour is outside the staggering's range,
// its term, which the reference omits, is 0.
constexpr int kViscLevels = 8;
enum { S_U = 0, S_V = 1, S_W = 2 };

// wet levels of a point's neighbours (0: no term) and the loads of its stencil
struct Cross {
  int c, e, w, n, s;
};
template <int ST>
__device__ __forceinline__ Cross cross_kb(const Geo& G, int i, int j) {
  const ColGeo& cg = ST == S_U ? G.gu : ST == S_V ? G.gv : G.gp;
  const int ij = G.L.at2(i, j);
  constexpr int i0 = ST == S_U ? 0 : 1, j0 = ST == S_V ? 0 : 1;
  Cross k;
  k.c = cg.kb[ij];
  k.e = i < G.L.ie ? cg.kb[ij + 1] : 0;
  k.w = i > i0 ? cg.kb[ij - 1] : 0;
  k.n = j > j0 ? cg.kb[ij - G.L.P] : 0;
  k.s = j < G.L.je ? cg.kb[ij + G.L.P] : 0;
  return k;
}

// first Laplacians UK1O (u), VK1E (v), WN1O (w), ocvisc.f90:350-438, 617-669
template <int ST, bool ALL>
__device__ __forceinline__ void visc_lap(const Geo& G, const double* __restrict__ f,
                                         double* __restrict__ out, int i, int j, int K0) {
  const int IE = G.L.ie, JE = G.L.je, P = G.L.P, pl = G.L.plane;
  constexpr int i0 = ST == S_U ? 0 : 1, j0 = ST == S_V ? 0 : 1;
  if (i < i0 || j < j0) return;
  const bool iin = i > i0 && i < IE, jin = j > j0 && j < JE;
  const int ij = G.L.at2(i, j);
  Cross k = cross_kb<ST>(G, i, j);
  double ce = 0., cw = 0., cn = 0., cs = 0., rx = 0., ry = 0.;
  if (iin || jin) {
    if (ST == S_U) {
      ce = i < IE ? G.rdlxp[ij + 1] : 0.;
      cw = G.rdlxp[ij];
      rx = G.rdlxu[ij];
      cn = G.rdlypsi[ij - P];
      cs = G.rdlypsi[ij];
      ry = G.rdlyu[ij];
    } else if (ST == S_V) {
      ce = G.rdlxpsi[ij];
      cw = G.rdlxpsi[ij - 1];
      rx = G.rdlxv[ij];
      cn = G.rdlyp[ij];
      cs = j < JE ? G.rdlyp[ij + P] : 0.;
      ry = G.rdlyv[ij];
    } else {
      ce = G.rdlxu[ij];
      cw = G.rdlxu[ij - 1];
      rx = G.rdlxp[ij];
      cn = G.rdlyv[ij - P];
      cs = G.rdlyv[ij];
      ry = G.rdlyp[ij];
    }
  } else {
    k.c = 0;  // a corner
  }
  const bool all = ALL && (iin || jin);
  const int o0 = G.L.at(i, j, K0 - 1), n = min(kViscLevels, G.L.ke + 1 - K0);
  for (int q0 = 0; q0 < n; q0 += 4) {
    double c[4], e[4], w[4], no[4], so[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int K = K0 + q0 + q, o = o0 + (q0 + q) * pl;
      const bool land = all && q0 + q < n, wet = K <= k.c;  // (k.c <= KE)
      c[q] = wet || land ? f[o] : 0.;
      e[q] = (wet && K <= k.e) || (land && i < IE) ? f[o + 1] : c[q];
      w[q] = (wet && K <= k.w) || (land && i > i0) ? f[o - 1] : c[q];
      no[q] = (wet && K <= k.n) || (land && j > j0) ? f[o - P] : c[q];
      so[q] = (wet && K <= k.s) || (land && j < JE) ? f[o + P] : c[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (q0 + q >= n) break;
      const int K = K0 + q0 + q;
      double r;
      if (!all) {  // a neighbour without water gives c - c = 0, as its mask does
        const double x = ((e[q] - c[q]) * ce - (c[q] - w[q]) * cw) * rx;
        const double y = ((no[q] - c[q]) * cn - (c[q] - so[q]) * cs) * ry;
        r = K <= k.c ? x + y : 0.;
      } else {
        const double x = ((K <= k.e ? ce : 0.) * (e[q] - c[q]) - (K <= k.w ? cw : 0.) * (c[q] - w[q])) * rx;
        const double y = ((K <= k.n ? cn : 0.) * (no[q] - c[q]) - (K <= k.s ? cs : 0.) * (c[q] - so[q])) * ry;
        r = (K <= k.c ? 1. : 0.) * (x + y);
      }
      out[o0 + (q0 + q) * pl] = r;
    }
  }
}

__global__ void __launch_bounds__(128, 7) k_visc_lap(Geo G, const double* __restrict__ uk,
                                                  const double* __restrict__ vk,
                                                  const double* __restrict__ wn,
                                                  double* __restrict__ u1,
                                                  double* __restrict__ v1,
                                                  double* __restrict__ w1, const double* bad,
                                                  int chunks) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y;
  if (i > G.L.ie || j > G.L.je) return;
  const int K0 = (blockIdx.z % chunks) * kViscLevels + 1;
  auto run = [&](auto all) {
    constexpr bool A = decltype(all)::value;
    switch (blockIdx.z / chunks) {
      case 0: visc_lap<S_U, A>(G, uk, u1, i, j, K0); break;
      case 1: visc_lap<S_V, A>(G, vk, v1, i, j, K0); break;
      default: visc_lap<S_W, A>(G, wn, w1, i, j, K0); break;
    }
  };
  if (*bad == 0.) run(std::false_type{});
  else run(std::true_type{});
}

// second passes, ocvisc.f90:445-477 (u, v) and 673-688 (w).  The face terms
// AUL.. * width / length are precomputed per face (G.ugx .. G.wgy) and the cell
// areas' reciprocals per cell, so a cell needs no division except by its
// thickness (w).  keep: the values of points outside the update range.
template <int ST, bool ALL>
__device__ __forceinline__ void visc_bih(const Geo& G, const double* __restrict__ keep,
                                         const double* __restrict__ f,
                                         const double* __restrict__ l, double* __restrict__ out,
                                         int i, int j, int K0) {
  const int IE = G.L.ie, JE = G.L.je, P = G.L.P, pl = G.L.plane;
  constexpr int i0 = ST == S_U ? 0 : 1, j0 = ST == S_V ? 0 : 1;
  if (i < i0 || j < j0) return;
  const int kbot = G.L.ke + (ST == S_W);  // KEP of w is carried
  const int o0 = G.L.at(i, j, K0 - 1), n = min(kViscLevels, kbot + 1 - K0);
  if (!(i > i0 && i < IE && j > j0 && j < JE)) {
    for (int q = 0; q < n; ++q) out[o0 + q * pl] = keep[o0 + q * pl];
    return;
  }
  const int ij = G.L.at2(i, j);
  const Cross k = cross_kb<ST>(G, i, j);
  double ge, gw, gn, gs, area, rarea;
  if (ST == S_U) {
    ge = G.ugx[ij + 1];
    gw = G.ugx[ij];
    gn = G.ugy[ij - P];
    gs = G.ugy[ij];
    area = G.dlxu[ij] * G.dlyu[ij];
    rarea = G.rareau[ij];
  } else if (ST == S_V) {
    ge = G.vgx[ij];
    gw = G.vgx[ij - 1];
    gn = G.vgy[ij];
    gs = G.vgy[ij + P];
    area = G.dlxv[ij] * G.dlyv[ij];
    rarea = G.rareav[ij];
  } else {
    ge = G.wgx[ij];
    gw = G.wgx[ij - 1];
    gn = G.wgy[ij - P];
    gs = G.wgy[ij];
    area = G.dlxp[ij] * G.dlyp[ij];
    rarea = G.rareap[ij];
  }
  // w: thicknesses of the cell and its faces, at least MINVALUE
  int kue = 0, kuw = 0, kvn = 0, kvs = 0;
  double bc = 0., bue = 0., buw = 0., bvn = 0., bvs = 0.;
  if (ST == S_W) {
    kue = G.gu.kb[ij];
    kuw = G.gu.kb[ij - 1];
    kvn = G.gv.kb[ij - P];
    kvs = G.gv.kb[ij];
    bc = G.gp.bot[ij];
    bue = G.gu.bot[ij];
    buw = G.gu.bot[ij - 1];
    bvn = G.gv.bot[ij - P];
    bvs = G.gv.bot[ij];
  }
  for (int q0 = 0; q0 < n; q0 += 4) {
    double v[4], c[4], e[4], w[4], no[4], so[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int K = K0 + q0 + q, o = o0 + (q0 + q) * pl;
      const bool land = ALL && K <= G.L.ke, wet = K <= k.c;
      v[q] = K <= kbot ? f[o] : 0.;
      c[q] = wet || land ? l[o] : 0.;
      e[q] = (wet && K <= k.e) || land ? l[o + 1] : c[q];
      w[q] = (wet && K <= k.w) || land ? l[o - 1] : c[q];
      no[q] = (wet && K <= k.n) || land ? l[o - P] : c[q];
      so[q] = (wet && K <= k.s) || land ? l[o + P] : c[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int K = K0 + q0 + q;
      if (q0 + q >= n) break;
      double r = 0.;
      if (K <= k.c || (ALL && K <= G.L.ke)) {
        const double wet = K <= k.c ? 1. : 0.;
        double fe = ge, fw = gw, fn = gn, fs = gs;
        if (ALL) {
          fe = K <= k.e ? fe : 0.;
          fw = K <= k.w ? fw : 0.;
          fn = K <= k.n ? fn : 0.;
          fs = K <= k.s ? fs : 0.;
        }
        if (ST == S_W) {
          const double mv = G.minvalue, dz = __ldg(G.dzw + K - 1);
          auto th = [&](int kb, double bot) { return fmx(K < kb ? dz : (K == kb ? bot : 0.0), mv); };
          const double dzp = th(k.c, bc);
          r = div_nr(wet * rarea, dzp) *
              (area * dzp * v[q] -
               (fe * th(kue, bue) * (e[q] - c[q]) - fw * th(kuw, buw) * (c[q] - w[q]) +
                fn * th(kvn, bvn) * (no[q] - c[q]) - fs * th(kvs, bvs) * (c[q] - so[q])));
        } else {
          r = wet * rarea * (area * v[q] - (fe * (e[q] - c[q]) - fw * (c[q] - w[q]) +
                                            fn * (no[q] - c[q]) - fs * (c[q] - so[q])));
        }
      }
      if (ST == S_W && K > G.L.ke) r = v[q];
      out[o0 + (q0 + q) * pl] = r;
    }
  }
}

__global__ void __launch_bounds__(128) k_visc_bih(
    Geo G, const double* __restrict__ uoo, const double* __restrict__ voe,
    const double* __restrict__ uk, const double* __restrict__ vk, const double* __restrict__ wn,
    const double* __restrict__ u1, const double* __restrict__ v1, const double* __restrict__ w1,
    double* __restrict__ uo, double* __restrict__ vo, double* __restrict__ wo, const double* bad,
    int chunks) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y;
  if (i > G.L.ie || j > G.L.je) return;
  const int K0 = (blockIdx.z % chunks) * kViscLevels + 1;
  auto run = [&](auto all) {
    constexpr bool A = decltype(all)::value;
    switch (blockIdx.z / chunks) {
      case 0: visc_bih<S_U, A>(G, uoo, uk, u1, uo, i, j, K0); break;
      case 1: visc_bih<S_V, A>(G, voe, vk, v1, vo, i, j, K0); break;
      default: visc_bih<S_W, A>(G, wn, wn, w1, wo, i, j, K0); break;
    }
  };
  if (*bad == 0.) run(std::false_type{});
  else run(std::true_type{});
}

}  // namespace

void launch_octdiff_vert(const Geo& G, int ntr, const double* const* in, double* const* out,
                         const double* dvo, const double* zo, cudaStream_t st) {
  TrPtrs tp{};
  for (int n = 0; n < ntr; ++n) {
    tp.in[n] = in[n];
    tp.out[n] = out[n];
  }
  const dim3 b(32, kVertBlock / 32);
  const dim3 gr = grid2(G.L.ie, G.L.je, b);
  switch (ntr) {
    case 1: k_tdiff_vert_b<1, 4><<<gr, b, 0, st>>>(G, tp, dvo, zo); break;
    case 2: k_tdiff_vert_b<2, 4><<<gr, b, 0, st>>>(G, tp, dvo, zo); break;
    case 3: k_tdiff_vert_b<3, 4><<<gr, b, 0, st>>>(G, tp, dvo, zo); break;
    case 4: k_tdiff_vert_b<4, 4><<<gr, b, 0, st>>>(G, tp, dvo, zo); break;
    default: k_tdiff_vert<<<gr, b, 0, st>>>(G, tp, ntr, dvo, zo); break;
  }
  count_launch();
}

void launch_octdiff_hbih(const Geo& G, int ntr, const double* const* in, double* const* out,
                         const double* zo, cudaStream_t st) {
  TrPtrs tp{};
  for (int n = 0; n < ntr; ++n) {
    tp.in[n] = in[n];
    tp.out[n] = out[n];
  }
  const dim3 b(kHbX, kHbY);
  dim3 gr = grid2(G.L.ie, G.L.je, b);
  // On planes of less than three blocks per SM a block takes one tracer and a part of
  // the levels, at least eight: four rounds of blocks, where one block for all left
  // the chip waiting (OCTDIFF of 512 x 1 x 60 0.131 ms, now 0.071, 97 x 131 x 41 0.150 and
  // 0.100, 256 x 256 x 60 0.38 and 0.33); on larger ones it marches through all, its
  // geometry loaded once (413 x 311 x 83 0.79 ms against 0.81 in parts).
  const int blocks = gr.x * gr.y;
  if (blocks < 3 * 148) {
    const int parts = std::min((4 * 2 * 148 + blocks * ntr - 1) / (blocks * ntr), (G.L.ke + 7) / 8);
    const int levels = (G.L.ke + parts - 1) / parts;
    gr.z = ntr * ((G.L.ke + levels - 1) / levels);
    k_tdiff_hbih<true><<<gr, b, 0, st>>>(G, tp, ntr, levels, zo);
  } else {
    k_tdiff_hbih<false><<<gr, b, 0, st>>>(G, tp, ntr, G.L.ke, zo);
  }
  count_launch();
}

void launch_ocvisc(const Geo& G, const double* uoo, const double* voe, const double* wno,
                   const double* uko, const double* vke, const double* avo, double* spu,
                   double* spv, double* ukv, double* vkv, double* wnv, double* u1, double* v1,
                   double* w1, double* uo, double* vo, double* wo, cudaStream_t st) {
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke;
  const dim3 b2(32, 4), bc(32, kVertBlock / 32), b3(32, 4);
  double* bad = spu + G.L.at2(0, 0);  // cleared by k_visc_speed
  k_visc_speed<<<grid2(IE + 1, JE + 1, b2), b2, 0, st>>>(G, uoo, voe, spu, spv);
  count_launch();
  dim3 gv = grid2(IE + 1, JE + 1, bc);
  gv.z = 2;
  k_visc_uv_b<4><<<gv, bc, 0, st>>>(G, uoo, voe, uko, vke, avo, spu, spv, ukv, vkv, bad);
  count_launch();
  with_tri_split(KE, [&](auto* l) {
    using Ln = std::remove_pointer_t<decltype(l)>;
    const int nb = (IE + Ln::W) / Ln::W;  // rows in x: y ends at 65535
    k_visc_w<Ln><<<nb * JE, Ln::NT, 0, st>>>(G, wno, avo, wnv, bad);
  });
  count_launch();
  const int chunks = (KE + 1 + kViscLevels - 1) / kViscLevels;
  dim3 gl = grid2(IE + 1, JE + 1, b3);
  gl.z = 3 * chunks;
  k_visc_lap<<<gl, b3, 0, st>>>(G, ukv, vkv, wnv, u1, v1, w1, bad, chunks);
  count_launch();
  k_visc_bih<<<gl, b3, 0, st>>>(G, uoo, voe, ukv, vkv, wnv, u1, v1, w1, uo, vo, wo, bad, chunks);
  count_launch();
}

}  // namespace orctm
