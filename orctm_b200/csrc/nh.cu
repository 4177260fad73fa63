// Nonhydrostatic pressure correction OCVTOT_NH (ocvtot_nh.f90:1-259) around
// the Poisson solve (poisson.cu): the right-hand side DIVG*WETO
// (ocvtot_nh.f90:11-62, ComputeRHS mo_petsc.f90:298-376) and, after the
// solve, the open-boundary PNH fill, the u/v pressure-gradient correction and
// the continuity re-diagnosis of WNO (ocvtot_nh.f90:150-236).
#include <algorithm>

#include "common.cuh"
#include "ops.h"

namespace orctm {

namespace {

#define AT(a, i, j, K) (a)[G.L.at((i), (j), (K)-1)]

inline dim3 grid2(int nx, int ny, dim3 b) { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y, 1); }
inline dim3 grid3(int nx, int ny, int nz, dim3 b) {
  return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y, nz);
}

// ------------------------------------------------------------ RHS --------
// b = DIVG * WETO for the interior cells (ocvtot_nh.f90:11-62,
// mo_petsc.f90:298-376); other entries of b are left untouched (zero).
// A thread takes kNhLevels levels of a column, the loads of four issued
// together, with the column's metrics and their reciprocals formed once (div_by:
// the quotients of a division).  Seven fields pass through memory; one level per
// thread, nine divisions each, took 2.36 ms on 1024 x 1024 x 80.
constexpr int kNhLevels = 8;

__global__ void __launch_bounds__(128) k_nh_rhs(Geo G, const double* __restrict__ uoo,
                         const double* __restrict__ uoo1,
                         const double* __restrict__ voe, const double* __restrict__ voe1,
                         const double* __restrict__ wno, const double* __restrict__ wno1,
                         const double* __restrict__ zo, double* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke, P = G.L.P, pl = G.L.plane;
  if (i > IE - 1 || j > JE - 1) return;
  const double DT = G.dt, rdt = rcp_for(DT);
  const int ij = G.L.at2(i, j);
  const double dlxp = G.dlxp[ij], dlyp = G.dlyp[ij], rx = rcp_for(dlxp), ry = rcp_for(dlyp);
  const int kb = G.gp.kb[ij];
  const double bot = G.gp.bot[ij];
  const int K0 = 1 + blockIdx.z * kNhLevels, K1 = min(KE, K0 + kNhLevels - 1);
  int o = ij + (K0 - 1) * pl;
  double gw0 = div_by(wno[o] - wno1[o], DT, rdt);
#pragma unroll 1
  for (int Kb = K0; Kb <= K1; Kb += 4) {
    double du[4], dum[4], dv[4], dvm[4], dw[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int q = ij + (min(Kb + e, K1) - 1) * pl;
      du[e] = uoo[q] - uoo1[q];
      dum[e] = uoo[q - 1] - uoo1[q - 1];
      dv[e] = voe[q] - voe1[q];
      dvm[e] = voe[q - P] - voe1[q - P];
      dw[e] = wno[q + pl] - wno1[q + pl];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int K = Kb + e;
      if (K > K1) break;
      const double divgu = div_by(div_by(du[e], DT, rdt) - div_by(dum[e], DT, rdt), dlxp, rx);
      const double divgv = div_by(div_by(dvm[e], DT, rdt) - div_by(dv[e], DT, rdt), dlyp, ry);
      const double gw1 = div_by(dw[e], DT, rdt);
      const double th = fmx(K < kb ? G.dzw[K - 1] : (K == kb ? bot : 0.0), 1.E-3);
      const double divgw = (gw0 - gw1) / (K >= 2 ? th : th + zo[ij]);
      const double divg = divgu + divgv + divgw;
      b[ij + (K - 1) * pl] = divg * (K <= kb ? 1.0 : 0.0);
      gw0 = gw1;
    }
  }
}

// ------------------------------------------------------- post solve -----
// PNH: interior from the solution, open-boundary halo copied from the first
// interior row/column (ocvtot_nh.f90:154-186), the rest kept; and the u/v
// correction by its gradient (ocvtot_nh.f90:189-203).  One kernel: the three
// values of PNH that a point needs come from the solution directly.
__global__ void __launch_bounds__(128) k_nh_puv(Geo G, const double* __restrict__ x,
                         const double* __restrict__ pold, double* __restrict__ pnh,
                         const double* __restrict__ uoo, const double* __restrict__ voe,
                         double* __restrict__ uo, double* __restrict__ vo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke, P = G.L.P, pl = G.L.plane;
  if (i > IE || j > JE) return;
  const int ij = G.L.at2(i, j);
  // where PNH of column (ii, jj) comes from: the solution or its old value, at an
  // offset (the west/east fill, J = 2..JE1, then the north/south one)
  struct Source {
    const double* f;
    int o;
  };
  auto source = [&](int ii, int jj) {
    if (jj == 1 && G.ob_n) jj = 2;
    if (jj == JE && G.ob_s) jj = JE - 1;
    if (jj >= 2 && jj <= JE - 1) {
      if (ii >= 2 && ii <= IE - 1) return Source{x, ii + P * jj};
      if (ii == 1 && G.ob_w) return Source{x, 2 + P * jj};
      if (ii == IE && G.ob_e) return Source{x, IE - 1 + P * jj};
    }
    return Source{pold, ii + P * jj};
  };
  const bool inu = i >= 1 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  const bool inv = i >= 2 && i <= IE - 1 && j >= 1 && j <= JE - 1;
  const bool hasp = i >= 1 && j >= 1;
  const Source p0 = source(max(i, 1), max(j, 1));
  const Source pe = inu ? source(i + 1, j) : p0, ps = inv ? source(i, j + 1) : p0;
  const int kbu = inu ? G.gu.kb[ij] : 0, kbv = inv ? G.gv.kb[ij] : 0;
  const double fu = inu ? G.dtdxuo[ij] : 0.0, fv = inv ? G.dpye[ij] : 0.0;
  const int K0 = blockIdx.z * kNhLevels, K1 = min(KE, K0 + kNhLevels);
#pragma unroll 1
  for (int Kb = K0; Kb < K1; Kb += 4) {
    double a[4], e4[4], s4[4], u[4], v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int q = min(Kb + e, K1 - 1) * pl;
      a[e] = p0.f[p0.o + q];
      e4[e] = pe.f[pe.o + q];
      s4[e] = ps.f[ps.o + q];
      u[e] = j >= 1 ? uoo[ij + q] : 0.0;
      v[e] = i >= 1 ? voe[ij + q] : 0.0;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int K = Kb + e + 1, q = (K - 1) * pl;
      if (K > K1) break;
      if (hasp) pnh[ij + q] = a[e];
      if (inu) u[e] = u[e] + (K <= kbu ? 1.0 : 0.0) * fu * (a[e] - e4[e]);
      if (inv) v[e] = v[e] + (K <= kbv ? 1.0 : 0.0) * fv * (s4[e] - a[e]);
      if (j >= 1) uo[ij + q] = u[e];
      if (i >= 1) vo[ij + q] = v[e];
    }
  }
}

// WNO re-diagnosed from continuity, bottom up (ocvtot_nh.f90:215-236); the loads of
// eight levels issued together
__global__ void __launch_bounds__(128) k_nh_w(Geo G, const double* __restrict__ uoo,
                       const double* __restrict__ voe, double* __restrict__ wno) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke, P = G.L.P, pl = G.L.plane;
  if (i > IE || j > JE) return;
  const int ij = G.L.at2(i, j), ijw = G.L.at2(i - 1, j), ijn = G.L.at2(i, j - 1);
  const int kb = G.gp.kb[ij], kbw = G.gu.kb[ijw], kbe = G.gu.kb[ij], kbn = G.gv.kb[ijn], kbs = G.gv.kb[ij];
  const double bw = G.gu.bot[ijw], be = G.gu.bot[ij], bn = G.gv.bot[ijn], bs = G.gv.bot[ij];
  const double yw = G.dlyu[ijw], ye = G.dlyu[ij], xs = G.dlxv[ij], xn = G.dlxv[ijn];
  const double fx = G.dtdxpo[ij], fy = G.dtdyo[ij], dlyp = G.dlyp[ij], dlxp = G.dlxp[ij];
  const double ry = rcp_for(dlyp), rx = rcp_for(dlxp);
  auto th = [&](int K, int k, double bot) { return K < k ? G.dzw[K - 1] : (K == k ? bot : 0.0); };
  double w = 0.0;
  wno[ij + KE * pl] = 0.0;
  constexpr int U = 8;
#pragma unroll 1
  for (int Kb = KE; Kb >= 1; Kb -= U) {
    double uw[U], ue[U], vs[U], vn[U];
#pragma unroll
    for (int e = 0; e < U; ++e) {
      const int o = ij + (max(Kb - e, 1) - 1) * pl;
      uw[e] = uoo[o - 1];
      ue[e] = uoo[o];
      vs[e] = voe[o];
      vn[e] = voe[o - P];
    }
#pragma unroll
    for (int e = 0; e < U; ++e) {
      const int K = Kb - e;
      if (K < 1) break;
      const double we = K <= kb ? 1.0 : 0.0;
      w = w + G.dti * we * div_by(fx * (uw[e] * th(K, kbw, bw) * yw - ue[e] * th(K, kbe, be) * ye), dlyp, ry) +
          G.dti * we * div_by(+fy * (vs[e] * th(K, kbs, bs) * xs - vn[e] * th(K, kbn, bn) * xn), dlxp, rx);
      wno[ij + (K - 1) * pl] = w;
    }
  }
}

}  // namespace

void launch_nh_rhs(const Geo& G, const double* uoo, const double* uoo1, const double* voe,
                   const double* voe1, const double* wno, const double* wno1, const double* zo,
                   double* b, cudaStream_t st) {
  const dim3 bk(32, 4);
  const int nz = (G.L.ke + kNhLevels - 1) / kNhLevels;
  k_nh_rhs<<<grid3(G.L.ie - 2, G.L.je - 2, nz, bk), bk, 0, st>>>(G, uoo, uoo1, voe, voe1, wno,
                                                                     wno1, zo, b);
  count_launch();
}


void launch_nh_post(const Geo& G, const double* x, const double* pold, double* pnh,
                    const double* uoo, const double* voe, double* uo, double* vo, double* wno,
                    cudaStream_t st) {
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke;
  const dim3 b3(32, 4), b2(32, 4);
  k_nh_puv<<<grid3(IE + 1, JE + 1, (KE + kNhLevels - 1) / kNhLevels, b3), b3, 0, st>>>(G, x, pold, pnh, uoo,
                                                                                      voe, uo, vo);
  count_launch();
  k_nh_w<<<grid2(IE, JE, b2), b2, 0, st>>>(G, uo, vo, wno);
  count_launch();
}

namespace {
// Rows of a field from consecutive memory to the padded layout; one thread per
// element of kUnpackRows rows.
constexpr int kUnpackRows = 8;
__global__ void __launch_bounds__(128) k_unpack(const double* __restrict__ src,
                                                double* __restrict__ dst, int ni, int nj, int rows,
                                                int P, int plane) {
  const int i = blockIdx.y * 128 + threadIdx.x;
  if (i >= ni) return;
#pragma unroll
  for (int q = 0; q < kUnpackRows; ++q) {
    const int row = blockIdx.x * kUnpackRows + q;  // of all levels
    if (row >= rows) return;
    dst[i + P * (row % nj) + plane * (row / nj)] = src[(size_t)row * ni + i];
  }
}
}  // namespace

void launch_unpack(const double* src, double* dst, int ni, int nj, int rows, int P, int plane,
                   cudaStream_t st) {
  const dim3 grid((rows + kUnpackRows - 1) / kUnpackRows, (ni + 127) / 128);
  k_unpack<<<grid, 128, 0, st>>>(src, dst, ni, nj, rows, P, plane);
  count_launch();
}

}  // namespace orctm
