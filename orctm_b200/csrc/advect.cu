// Mass-conserving limited advection (Maier-Reimer scheme) of tracers and of
// the u, v, w momenta: OCADPO (ocadpo.f90:94-348), OCUAD (ocuad.f90:1-271),
// OCVAD (ocvad.f90:1-271) and OCWAD (ocwad.f90:1-238).
//
// Each routine is three direction-split sweeps z -> x -> y.  Per sweep a cell
// volume V and the field T are updated from face transports
//     RN = V + WTP(-) - WTP(0) - WTM(0) + WTM(+)
//     T' = (T*V + TRP(-) - TRP(0) - TRM(0) + TRM(+)) / RN
//
// Two kernels per routine:
//   k_adv_zx   the z and the x sweep.  A warp holds 32 neighbouring columns of a row
//              (28 of them its own) and marches down the levels: the z sweep of a
//              level comes from a register window of its column, its result stays in registers
//              and the x sweep takes the neighbours' values and transports
//              from the other lanes by shuffles.
//   k_adv_y    the y sweep.  A warp holds 32 columns of one level and marches along
//              the rows with a register window; the warps of a block are
//              consecutive levels, which share the rows' 2D data through L1.
// Neither has a barrier or a shared-memory tile, a face's transports are formed once per
// marching thread, and the intermediate field and volume go through memory once
// instead of twice.  (Before, three kernels with a thread per cell or face reloaded the
// 2D geometry at every level and exchanged transports through shared
// memory: 195 bytes per cell and some 1100 instructions for three tracers,
// 12.4 ms on 1024 x 1024 x 80; 4.2-4.6 ms for each momentum component.)
// Every sweep writes a fresh buffer, so neighbouring columns always read the previous
// sweep's values.  Arithmetic is IEEE binary64 in the reference's operation order
// (built with --fmad=false), except that the three divisions of a face and a
// cell use div_nr (within 1 ulp of IEEE division), so results match the CPU
// restatement to a few ulp.
#include "common.cuh"
#include "ops.h"

namespace orctm {

namespace {

#define AT(a, i, j, K) (a)[G.L.at((i), (j), (K)-1)]

enum { V_ADPO = 0, V_UAD = 1, V_VAD = 2, V_WAD = 3 };

// Index ranges of a routine: its points start at (i0, j0); the x and y sweeps
// update i in [iL, IE - 1], j in [jL, JE - 1], levels from kL to KE.
template <int VAR> struct Rng;
template <> struct Rng<V_ADPO> { static constexpr int i0 = 1, j0 = 1, iL = 2, jL = 2, kL = 1; };
template <> struct Rng<V_UAD>  { static constexpr int i0 = 0, j0 = 1, iL = 1, jL = 2, kL = 1; };
template <> struct Rng<V_VAD>  { static constexpr int i0 = 1, j0 = 0, iL = 2, jL = 1, kL = 1; };
template <> struct Rng<V_WAD>  { static constexpr int i0 = 1, j0 = 1, iL = 2, jL = 2, kL = 2; };

template <int VAR>
__device__ __forceinline__ const ColGeo& cell_columns(const Geo& G) {
  return VAR == V_UAD ? G.gu : VAR == V_VAD ? G.gv : G.gp;
}

// Advected fields of one launch.  The driver calls OCADPO once per tracer with
// unchanged velocities (orctm.f90:1459-1460 and the passive tracers after
// them): the transports WTP/WTM, the volumes RN and the geometry factors
// depend on the velocities and the geometry only, so one launch advects up to
// kMaxFused tracers with them, each with the arithmetic of a separate call.
constexpr int kMaxFused = 4;

struct TrIO {
  const double* in[kMaxFused];
  double* out[kMaxFused];
};

// transports of a cell: to the previous cell (p) and to the next one (m)
template <int N>
struct Fl {
  double wtp, wtm;
  double trp[N], trm[N];
};

template <int N>
__device__ __forceinline__ Fl<N> zero_fl() {
  Fl<N> f;
  f.wtp = f.wtm = 0.;
#pragma unroll
  for (int n = 0; n < N; ++n) f.trp[n] = f.trm[n] = 0.;
  return f;
}

// Infinities and NaN.  In the reference's expressions a transport without outflow is
// 0 times an average, which is NaN if that is not finite, and MIN(cap, NaN) is cap.
// The short cuts of `limited` do not show that, so a march notes whether one of its
// values was not finite (Seen), and is then done again in full, without short cuts.
// The values are noted where they are used: noted at its load, a value in flight is
// waited for.  OCUAD + OCVAD + OCWAD + OCADPO of three tracers on 301 x 403 x 67: 1.86 ms,
// as without the note; 2.27 with short cuts that are safe one by one.
struct Seen {
  unsigned top = 0;  // the largest high word without its sign
  __device__ __forceinline__ double operator()(double x) {
    top = max(top, (unsigned)__double2hiint(x) & 0x7fffffffu);
    return x;
  }
  // a value that is 0 or above, or NaN
  __device__ __forceinline__ void nonneg(double x) { top = max(top, (unsigned)__double2hiint(x)); }
  __device__ __forceinline__ bool nonfinite() const { return top >= 0x7ff00000u; }
};

// The limited upwind pair: TRP takes the average with ta, TRM with tb; SCHA is
// multiplied by the masks' product w (0 or 1), SCH capped by cap, and 0 with
// flat.  (ocadpo.f90:107-125, 203-232; ocuad.f90:41-52 without masks)  Where a
// factor makes the result 0 (no outflow: land; SCHA = 0: a uniform field, a
// local extremum) the steps it makes idle are passed by, which a whole warp often
// can; in full they are not (an outflow of infinity divides to 0 there, NaN stays).
__device__ __forceinline__ void limited(bool full, double up, double um, double t, double ta,
                                        double tb, double vol, double cap, bool w, bool flat,
                                        double& trp, double& trm) {
  trp = trm = 0.;
  const double out = up + um;
  if (out == 0. && !full) return;
  double sch = 0.;
  if ((w || full) && !flat) {
    const double abl = fabs(ta - tb);
    const double zwabl = fabs(ta + tb - 2. * t);
    const double num = abl - zwabl;
    if (!(num <= 0.) || full) {
      double scha = fmx(0., div_in_range(num, abl + 1.E-20));
      if (!w) scha = 0. * scha;
      const double x = scha * vol;
      sch = fmn(cap, div_in_range(x, out + 1.E-20));
      if (full && out > 1e300) sch = fmn(cap, 0. * x);
    }
  }
  const double schi = 1. - sch;
  trp = up * (schi * t + sch * 0.5 * (t + ta));
  trm = um * (schi * t + sch * 0.5 * (t + tb));
}

// update from the transports before (WTP, TRP), own and after (WTM, TRM)
__device__ __forceinline__ void apply(double t, double v, double mwtp, double mtrp, double cwtp,
                                      double cwtm, double ctrp, double ctrm, double pwtm,
                                      double ptrm, double& tn, double& vn) {
  const double rn = v + mwtp - cwtp - cwtm + pwtm;
  tn = div_nr(t * v + mtrp - ctrp - ctrm + ptrm, rn);
  vn = rn;
}

constexpr unsigned kAll = 0xffffffffu;
__device__ __forceinline__ double from_west(double x) { return __shfl_up_sync(kAll, x, 1); }
__device__ __forceinline__ double from_east(double x) { return __shfl_down_sync(kAll, x, 1); }

// -------------------------------------------------------- z and x sweeps ---
constexpr int kZxCells = 28, kZxRows = 4;

// ocadpo.f90:94-232, ocuad.f90:20-148, ocvad.f90:20-148, ocwad.f90:14-...;
// the block's levels are klen from 1 + klen blockIdx.z (full: without short cuts).
// Returns whether a value of the march was not finite, for the whole warp
template <int VAR, int N>
__device__ __forceinline__ bool march_zx(const Geo& G, const TrIO& io, const double* __restrict__ wo,
                                         const double* __restrict__ zo,
                                         const double* __restrict__ uko, double* __restrict__ Vo,
                                         int klen, bool full) {
  using R = Rng<VAR>;
  Seen seen;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke, pl = G.L.plane;
  const int lane = threadIdx.x;
  const int i = R::i0 + blockIdx.x * kZxCells + lane - 2;
  const int j = R::j0 + blockIdx.y * kZxRows + threadIdx.y;
  if (j > JE) return false;  // the whole warp
  const int kbot = VAR == V_WAD ? KE + 1 : KE;  // levels of the field
  const int Ka = 1 + blockIdx.z * klen, Kb = min(kbot, Ka + klen - 1);
  if (Ka > kbot) return false;
  const bool cell = i >= R::i0 && i <= IE;             // a point of the field
  const bool own = cell && lane >= 2 && lane < 2 + kZxCells;
  const int ij = G.L.at2(i, j), b0 = G.L.at(i, j, 0);
  const ColGeo& cg = cell_columns<VAR>(G);
  const int kb = cell ? cg.kb[ij] : 0;
  const double bot = cell ? cg.bot[ij] : 0.;
  auto thick_c = [&](int K) { return K < kb ? __ldg(G.dzw + K - 1) : (K == kb ? bot : 0.0); };

  // ---- z: metrics, volumes, interface velocity ww(K) between levels K - 1 and K
  const bool zin = cell && i >= R::iL && i <= IE - 1 && j >= R::jL && j <= JE - 1;
  const double dlxc = !cell ? 0. : VAR == V_UAD ? G.dlxu[ij] : VAR == V_VAD ? G.dlxv[ij] : G.dlxp[ij];
  const double dlyc = !cell ? 0. : VAR == V_UAD ? G.dlyu[ij] : VAR == V_VAD ? G.dlyv[ij] : G.dlyp[ij];
  const double area = dlxc * dlyc;
  const double cdt = zin ? 0.5 * G.dt * G.dlyp[ij] * G.dlxp[ij] : 0.;
  const double zij = cell && (VAR == V_ADPO || VAR == V_WAD) ? seen(zo[ij]) : 0.;
  const double wsurf = VAR == V_ADPO && cell ? seen(wo[b0]) : 0.;
  auto v0 = [&](int K) {
    if (K > kb) return 0.;
    if (VAR == V_WAD) {
      if (K == 1) return area * (thick_c(1) + zij) / 2.0;
      if (K == 2) return area * (thick_c(1) + thick_c(2) + zij) / 2.0;
      return area * (thick_c(K - 1) + thick_c(K)) / 2.0;
    }
    double s = area * thick_c(K);
    if (VAR == V_ADPO && K == 1) s = s + area * (zij - wsurf * G.dt);
    return s;
  };
  auto raw_w = [&](int K) -> double {  // wo at level K, 0 outside its levels
    return zin && K >= 1 && K <= KE + 1 ? wo[b0 + (K - 1) * pl] : 0.;
  };
  auto raw_w2 = [&](int K) -> double {
    return zin && K >= 1 && K <= KE + 1 ? wo[b0 + (VAR == V_UAD ? 1 : G.L.P) + (K - 1) * pl] : 0.;
  };
  // ww(K) as the level above (w at K - 1) and this one (K) give it
  auto face_w = [&](int K, double wabove) {
    const double w = raw_w(K);
    if (VAR == V_ADPO) return w;
    if (VAR == V_WAD) return 0.5 * (w + wabove);
    return 0.5 * (w + raw_w2(K));
  };
  auto load_t = [&](int n, int K) -> double {
    return cell && K >= 1 && K <= kbot ? io.in[n][b0 + (K - 1) * pl] : 0.;
  };

  // ---- x: face coefficients of the column
  const bool xrow = j >= R::jL && j <= JE - 1;          // rows that the x sweep updates
  const bool uin = i >= 0 && i <= IE && xrow;           // u-points that may be read
  const int kbu = uin ? G.gu.kb[ij] : 0;
  const double botu = uin ? G.gu.bot[ij] : 0.;
  auto thick_u = [&](int K) { return K < kbu ? __ldg(G.dzw + K - 1) : (K == kbu ? botu : 0.0); };
  const int kbu2 = VAR == V_VAD && uin ? G.gu.kb[ij + G.L.P] : 0;
  const double botu2 = VAR == V_VAD && uin ? G.gu.bot[ij + G.L.P] : 0.;
  auto thick_u2 = [&](int K) { return K < kbu2 ? __ldg(G.dzw + K - 1) : (K == kbu2 ? botu2 : 0.0); };
  const double hdt = 0.5 * G.dt;
  double cup = 0., cum = 0.;  // factors of the eastward and the westward transport
  bool flux_here, edge = false;
  if (VAR == V_ADPO) {
    flux_here = xrow && i >= 2 && i <= IE - 1;
    cup = uin ? G.dlyu[ij] : 0.;
  } else if (VAR == V_UAD) {
    flux_here = xrow && i >= 0 && i <= IE;
    edge = i == 0 || i == IE;
    if (flux_here) {
      cup = hdt * G.dlyp[i < IE ? ij + 1 : ij];
      cum = edge ? G.dlyu[ij] : G.dlyp[ij];
    }
  } else if (VAR == V_VAD) {
    flux_here = xrow && i >= 1 && i <= IE;
    edge = i == 1 || i == IE;
    if (flux_here) {
      cup = hdt * (0.5 * (G.dlyu[ij] + G.dlyu[ij + G.L.P]));
      cum = 0.5 * (G.dlyu[ij - 1] + G.dlyu[ij - 1 + G.L.P]);
    }
  } else {
    flux_here = xrow && i >= 2 && i <= IE - 1;
    if (flux_here) {
      cup = hdt * G.dlyu[ij];
      cum = hdt * G.dlyu[ij - 1];
    }
  }
  const int kbw = __shfl_up_sync(kAll, kb, 1), kbe = __shfl_down_sync(kAll, kb, 1);
  const int kb3 = min(kb, min(kbw, kbe));
  const bool xup = own && i >= R::iL && i <= IE - 1 && xrow;
  auto u_at = [&](int K) -> double {  // uko of the u-point; for VAD row j + 1 below
    return uin && K >= 1 && K <= KE ? uko[b0 + (K - 1) * pl] : 0.;
  };

  // ---- start of the march: the window at K = Ka
  constexpr int kLast = VAR == V_WAD;  // 1: no clamping, the level KE + 1 exists
  double tu[N], t0[N], tl[N];          // T(K-1), T(K), T(K+1), clamped at the ends
  double wk;                           // wo at the level of the last interface (WAD)
  double ww1;                          // ww(K+1)
  Fl<N> fc, fm;
  fm = fc = zero_fl<N>();
  auto zflux = [&](int K, double w0, double w1, const double (&a)[N], const double (&c)[N],
                   const double (&b)[N], double vol) {
    Fl<N> f;
    f.wtp = cdt * (w0 + fabs(w0));
    f.wtm = cdt * (fabs(w1) - w1);
    seen.nonneg(f.wtp + f.wtm);
    const int klo = K + 1 < KE ? K + 1 : KE;
    const double cap = VAR == V_ADPO ? (klo <= kb ? 1. : 0.)
                       : VAR == V_WAD ? (K + 1 <= KE && K + 1 <= kb ? 1. : 0.) : 1.;
    const bool flat = VAR == V_ADPO && (K == 1 || K == KE);
#pragma unroll
    for (int n = 0; n < N; ++n)
      limited(full, f.wtp, f.wtm, c[n], a[n], b[n], vol, cap, true, flat, f.trp[n], f.trm[n]);
    return f;
  };
  // transports of the level above the first and below the last one of WAD
  // (ocwad.f90:72-83): the interface's flux of the mean of its two values
  auto wad_top = [&](double w1, double ta, double tb) {
    Fl<N> f = zero_fl<N>();
    f.wtm = cdt * (fabs(w1) - w1);
    f.trm[0] = f.wtm * (0.5 * (ta + tb));
    return f;
  };
  auto wad_bottom = [&](double w0, double ta, double tb) {
    Fl<N> f = zero_fl<N>();
    f.wtp = cdt * (w0 + fabs(w0));
    f.trp[0] = f.wtp * (0.5 * (ta + tb));
    return f;
  };
  const int Kz = R::kL;  // first level of the z sweep
  double vk = v0(Ka);
  {
    const double wa = VAR == V_WAD ? raw_w(Ka - 1) : 0.;
    const double w0 = face_w(Ka, wa);
    const double wKa = VAR == V_WAD ? raw_w(Ka) : 0.;
    ww1 = face_w(Ka + 1, wKa);
    wk = VAR == V_WAD ? raw_w(Ka + 1) : 0.;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      t0[n] = load_t(n, Ka);
      tu[n] = !kLast && Ka == 1 ? t0[n] : load_t(n, Ka - 1);
      tl[n] = !kLast && Ka == KE ? t0[n] : load_t(n, Ka + 1);
      seen(tu[n]);
      seen(t0[n]);
      seen(tl[n]);
    }
    if (Ka > Kz) {
      const int Km = Ka - 1;
      double tuu[N];
#pragma unroll
      for (int n = 0; n < N; ++n) tuu[n] = seen(!kLast && Km == 1 ? tu[n] : load_t(n, Km - 1));
      const double wu = VAR == V_WAD ? raw_w(Km - 1) : 0.;
      fm = zflux(Km, face_w(Km, wu), w0, tuu, tu, t0, v0(Km));
    } else if (VAR == V_WAD && Ka == 1) {
      fc = wad_top(ww1, t0[0], tl[0]);  // becomes fm of level 2
    }
    if (Ka >= Kz && Ka <= KE) fc = zflux(Ka, w0, ww1, tu, t0, tl, vk);
  }
  double udp = 0.;  // WAD: u times thickness at the level above
  if (VAR == V_WAD && Ka > 1) udp = u_at(Ka - 1) * thick_u(Ka - 1);
  // loads of the next level, one step ahead
  double tn2[N], un = u_at(Ka), un2 = VAR == V_VAD && uin && Ka <= KE ? uko[b0 + G.L.P + (Ka - 1) * pl] : 0.;
#pragma unroll
  for (int n = 0; n < N; ++n) tn2[n] = load_t(n, Ka + 2);

#pragma unroll 1
  for (int K = Ka; K <= Kb; ++K) {
    const double ucur = un, ucur2 = un2;
    un = u_at(K + 1);
    if (VAR == V_VAD) un2 = uin && K + 1 <= KE ? uko[b0 + G.L.P + K * pl] : 0.;
    // flux of level K + 1
    Fl<N> fp = zero_fl<N>();
    double vn = 0., ww2 = 0., tll[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      tll[n] = seen(!kLast && K + 1 >= KE ? tl[n] : tn2[n]);
      tn2[n] = load_t(n, K + 3);
    }
    if (K < KE) {
      vn = v0(K + 1);
      ww2 = face_w(K + 2, wk);
      if (VAR == V_WAD) wk = raw_w(K + 2);
      fp = zflux(K + 1, ww1, ww2, t0, tl, tll, vn);
    } else if (VAR == V_WAD && K == KE) {
      fp = wad_bottom(ww1, t0[0], tl[0]);
    }
    // z update: RN = V + WTP(K+1) - WTP(K) - WTM(K) + WTM(K-1)
    double t1[N], v1 = vk;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      t1[n] = t0[n];
      if (zin && K >= Kz && K <= KE && K <= kb) {
        double vt;
        apply(t0[n], vk, fp.wtp, fp.trp[n], fc.wtp, fc.wtm, fc.trp[n], fc.trm[n], fm.wtm, fm.trm[n],
              t1[n], vt);
        v1 = vt;
      }
    }
    // x transports
    double up = 0., um = 0.;
    if (VAR == V_ADPO) {
      const double c = hdt * thick_u(K);
      up = c * cup * (ucur + fabs(ucur));
      um = from_west(c * (fabs(ucur) - ucur) * cup);
    } else {
      const double ud = ucur * thick_u(K);
      double uos;
      if (VAR == V_UAD) {
        const double ude = from_east(ud);
        uos = i == IE ? ud : 0.5 * (ud + ude);
      } else if (VAR == V_VAD) {
        uos = 0.5 * (ud + ucur2 * thick_u2(K));
      } else {
        uos = 0.5 * (ud + udp);
        udp = ud;
      }
      double uwe = from_west(uos);
      if (VAR == V_UAD && i == 0) uwe = ud;
      up = cup * (uos + fabs(uos));
      um = VAR == V_WAD ? cum * (fabs(uwe) - uwe) : hdt * (fabs(uwe) - uwe) * cum;
    }
    const bool live = flux_here && K >= R::kL && K <= KE;
    if (!live) up = um = 0.;
    seen.nonneg(up + um);
    const double wtp_w = from_west(up), wtm_e = from_east(um);
    const bool w3 = VAR == V_ADPO || VAR == V_WAD ? K <= kb3 : true;
    const bool upd = xup && K >= R::kL && K <= KE && K <= kb;
    double v2 = v1;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      seen(t1[n]);
      const double te = from_east(t1[n]), tw = from_west(t1[n]);
      double trp = 0., trm = 0.;
      if (live) {
        if (edge) {
          trp = up * t1[n];
          trm = um * t1[n];
        } else {
          limited(full, up, um, t1[n], te, tw, v1, 1., w3, false, trp, trm);
        }
      }
      // RN = V + WTP(I-1) - WTP(I) - WTM(I) + WTM(I+1)
      const double trp_w = from_west(trp), trm_e = from_east(trm);
      double t2 = t1[n];
      if (upd) apply(t1[n], v1, wtp_w, trp_w, up, um, trp, trm, wtm_e, trm_e, t2, v2);
      if (own) io.out[n][b0 + (K - 1) * pl] = t2;
    }
    if (own && K <= KE) Vo[b0 + (K - 1) * pl] = v2;
    // down one level
    fm = fc;
    fc = fp;
    vk = vn;
    ww1 = ww2;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      t0[n] = tl[n];
      tl[n] = tll[n];
    }
  }
  return __any_sync(kAll, seen.nonfinite());
}

// Blocks per SM: one momentum field fits 80 registers a thread, which hides more
// latency than 96 (OCVAD's 250 us on 301 x 403 x 67 are 230 so)
template <int VAR, int N>
__global__ void __launch_bounds__(32 * kZxRows, N == 1 ? (VAR == V_ADPO ? 5 : 6) : 7 - N)
    k_adv_zx(Geo G, TrIO io, const double* __restrict__ wo, const double* __restrict__ zo,
             const double* __restrict__ uko, double* __restrict__ Vo, int klen) {
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass)
    if (!march_zx<VAR, N>(G, io, wo, zo, uko, Vo, klen, pass)) return;
}

// ---------------------------------------------------------------- y sweep ---
constexpr int kYLevels = 8;

// ocadpo.f90:264-348, ocuad.f90:184-271, ocvad.f90:184-271, ocwad.f90:160-238;
// jlen rows per block.  The J = 0 edge of OCVAD reads DLXU(I,0) in the
// reference, outside DLXU's bounds; DLXV(I,0) is used.
// Returns as march_zx, for the thread's own column.
template <int VAR, int N>
__device__ __forceinline__ bool march_y(const Geo& G, const TrIO& io, const double* __restrict__ V,
                                        const double* __restrict__ vke, int jlen, bool full) {
  using R = Rng<VAR>;
  Seen seen;
  const int IE = G.L.ie, JE = G.L.je, KE = G.L.ke, P = G.L.P;
  const int i = blockIdx.x * 32 + threadIdx.x;
  const int K = blockIdx.z * kYLevels + threadIdx.y + 1;
  const int kbot = VAR == V_WAD ? KE + 1 : KE;
  if (K > kbot || i < R::i0 || i > IE) return false;
  const int ja = R::j0 + blockIdx.y * jlen, jb = min(JE, ja + jlen - 1);
  if (ja > JE) return false;
  const int lev = (K - 1) * G.L.plane + i;  // offset of row 0
  const bool klev = K >= R::kL && K <= KE;
  const bool col = klev && i >= R::iL && i <= IE - 1;  // columns that the sweep updates
  if (!col) {
    for (int j = ja; j <= jb; ++j)
#pragma unroll
      for (int n = 0; n < N; ++n) io.out[n][lev + P * j] = io.in[n][lev + P * j];
    return false;
  }
  const double hdt = 0.5 * G.dt;
  const double dz = G.dzw[K - 1], dzu = VAR == V_WAD ? G.dzw[K - 2] : 0.;
  const ColGeo& cg = cell_columns<VAR>(G);
  auto vd = [&](int ii, int q, int KK, double d) {  // vke times thickness
    const int s = ii + P * q, kbv = G.gv.kb[s];
    return vke[s + (KK - 1) * G.L.plane] * (KK < kbv ? d : (KK == kbv ? G.gv.bot[s] : 0.0));
  };
  // face between rows q and q + 1: its velocity fv and the factor cf
  struct Face { double v, c; };
  auto face = [&](int q) {
    Face f{0., 0.};
    if (q < 0 || q > JE) return f;
    const int s = i + P * q;
    if (VAR == V_ADPO) {
      const int kbv = G.gv.kb[s];
      const double th = K < kbv ? dz : (K == kbv ? G.gv.bot[s] : 0.0);
      f.v = vke[lev + P * q];
      f.c = hdt * th * G.dlxv[s];
    } else if (VAR == V_UAD) {
      f.v = 0.5 * (vd(i, q, K, dz) + vd(i + 1, q, K, dz));
      f.c = hdt * (0.5 * (G.dlxv[s] + G.dlxv[s + 1]));
    } else if (VAR == V_VAD) {
      // f.c is the factor of the p-row q (the one before the face)
      f.v = q == JE ? vd(i, JE, K, dz) : 0.5 * (vd(i, q, K, dz) + vd(i, q + 1, K, dz));
      f.c = q >= 1 ? hdt * G.dlxp[s] : hdt * G.dlxv[s];
    } else {
      f.v = 0.5 * (vd(i, q, K, dz) + vd(i, q, K - 1, dzu));
      f.c = hdt * G.dlxv[s];
    }
    return f;
  };
  constexpr int qLo = VAR == V_VAD ? 0 : VAR == V_UAD ? 1 : 2;
  const int qHi = VAR == V_VAD || VAR == V_UAD ? JE : JE - 1;
  constexpr bool masked = VAR == V_ADPO || VAR == V_WAD;
  auto kb_at = [&](int q) { return q >= R::j0 && q <= JE ? cg.kb[i + P * q] : 0; };
  auto t_at = [&](int n, int q) -> double { return q >= R::j0 && q <= JE ? io.in[n][lev + P * q] : 0.; };
  auto v_at = [&](int q) -> double { return q >= R::j0 && q <= JE ? V[lev + P * q] : 0.; };
  // transports of row q from the faces before (fb: q - 1) and after (fa: q)
  auto flux = [&](int q, const Face& fb, const Face& fa, const double (&tb)[N], const double (&t)[N],
                  const double (&ta)[N], double vol, bool w3) {
    Fl<N> f = zero_fl<N>();
    if (q < qLo || q > qHi) return f;
    double vno = fb.v, cu = fb.c, cd = fa.c;
    if (VAR == V_VAD) {
      if (q == 0) vno = vd(i, 0, K, dz);
      cu = fa.c;
      cd = q == JE ? hdt * G.dlxu[i + P * JE] : hdt * G.dlxp[i + P * (q + 1)];
    }
    f.wtp = cu * (vno + fabs(vno));
    f.wtm = cd * (fabs(fa.v) - fa.v);
    seen.nonneg(f.wtp + f.wtm);
    const bool edge = VAR == V_UAD ? (q == 1 || q == JE) : VAR == V_VAD ? (q == 0 || q == JE) : false;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (edge) {
        f.trp[n] = f.wtp * t[n];
        f.trm[n] = f.wtm * t[n];
      } else {
        limited(full, f.wtp, f.wtm, t[n], tb[n], ta[n], vol, 1., masked ? w3 : true, false,
                f.trp[n], f.trm[n]);
      }
    }
    return f;
  };
  // window at the first row: T of rows ja - 1, ja, ja + 1, transports of ja - 1, ja
  double tp[N], t0[N], tn[N];
  Fl<N> fp, fc;
  Face fa;  // face after row ja
  int kp, k0, kn;
  double v0;
  {
    double tpp[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      tpp[n] = t_at(n, ja - 2);
      tp[n] = t_at(n, ja - 1);
      t0[n] = t_at(n, ja);
      tn[n] = t_at(n, ja + 1);
      seen(tpp[n]);
      seen(tp[n]);
      seen(t0[n]);
      seen(tn[n]);
    }
    const int kpp = kb_at(ja - 2);
    kp = kb_at(ja - 1);
    k0 = kb_at(ja);
    kn = kb_at(ja + 1);
    v0 = seen(v_at(ja));
    const Face f2 = face(ja - 2), f1 = face(ja - 1);
    fa = face(ja);
    fp = flux(ja - 1, f2, f1, tpp, tp, t0, seen(v_at(ja - 1)), K <= min(kpp, min(kp, k0)));
    fc = flux(ja, f1, fa, tp, t0, tn, v0, K <= min(kp, min(k0, kn)));
  }
  // values of the row after next, one step ahead
  double tnn[N], v1 = v_at(ja + 1);
  int knn = kb_at(ja + 2);
#pragma unroll
  for (int n = 0; n < N; ++n) tnn[n] = t_at(n, ja + 2);
#pragma unroll 1
  for (int j = ja; j <= jb; ++j) {
    const double vnx = v_at(j + 2);
    const int k3 = kb_at(j + 3);
    double t3[N];
#pragma unroll
    for (int n = 0; n < N; ++n) t3[n] = t_at(n, j + 3);
    const Face fb = fa;
    fa = face(j + 1);
    seen(v1);
#pragma unroll
    for (int n = 0; n < N; ++n) seen(tnn[n]);
    const Fl<N> fn = flux(j + 1, fb, fa, t0, tn, tnn, v1, K <= min(k0, min(kn, knn)));
    // RN = V + WTP(J+1) - WTP(J) - WTM(J) + WTM(J-1)
    const bool upd = j >= R::jL && j <= JE - 1 && K <= k0;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      double x = t0[n], vt;
      if (upd) apply(t0[n], v0, fn.wtp, fn.trp[n], fc.wtp, fc.wtm, fc.trp[n], fc.trm[n], fp.wtm, fp.trm[n], x, vt);
      io.out[n][lev + P * j] = x;
      t0[n] = tn[n];
      tn[n] = tnn[n];
      tnn[n] = t3[n];
    }
    fp = fc;
    fc = fn;
    v0 = v1;
    v1 = vnx;
    k0 = kn;
    kn = knn;
    knn = k3;
  }
  return seen.nonfinite();
}

template <int VAR, int N>
__global__ void __launch_bounds__(32 * kYLevels, N == 1 ? 4 : 2)
    k_adv_y(Geo G, TrIO io, const double* __restrict__ V, const double* __restrict__ vke, int jlen) {
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass)
    if (!march_y<VAR, N>(G, io, V, vke, jlen, pass)) return;
}

// Levels per block of k_adv_zx and rows per block of k_adv_y: a march
// repeats two transports at its start, so it is as long as the grid allows
// while every SM still gets some blocks; the results do not depend on it.
inline int march_length(int n, long long blocks_of_one, int least) {
  constexpr long long kWanted = 148 * 16;  // warps of 128 to 256 threads in flight several times over
  int parts = (int)((kWanted + blocks_of_one - 1) / blocks_of_one);
  if (parts < 1) parts = 1;
  int len = (n + parts - 1) / parts;
  return len < least ? least : len;
}

// io: N fields through the z and x sweeps into mid, through the y sweep into out
template <int VAR, int N>
void advect(const Geo& G, const TrIO& zx, const TrIO& y, const double* uko, const double* vke,
            const double* wo, const double* zo, double* vol, cudaStream_t st) {
  using R = Rng<VAR>;
  const int nx = G.L.ie + 1 - R::i0, ny = G.L.je + 1 - R::j0, nz = G.L.ke + (VAR == V_WAD);
  {
    const int gx = (nx + kZxCells - 1) / kZxCells, gy = (ny + kZxRows - 1) / kZxRows;
    const int len = march_length(nz, (long long)gx * gy, 8);
    k_adv_zx<VAR, N><<<dim3(gx, gy, (nz + len - 1) / len), dim3(32, kZxRows), 0, st>>>(
        G, zx, wo, zo, uko, vol, len);
    count_launch();
  }
  {
    const int gx = (G.L.ie + 32) / 32, gz = (nz + kYLevels - 1) / kYLevels;
    const int len = march_length(ny, (long long)gx * gz, 8);
    k_adv_y<VAR, N><<<dim3(gx, (ny + len - 1) / len, gz), dim3(32, kYLevels), 0, st>>>(G, y, vol, vke, len);
    count_launch();
  }
}

template <int VAR>
void advect_one(const Geo& G, const double* T, double* mid, double* out, const double* uko,
                const double* vke, const double* wo, const double* zo, double* vol, cudaStream_t st) {
  TrIO a{}, b{};
  a.in[0] = T;
  a.out[0] = mid;
  b.in[0] = mid;
  b.out[0] = out;
  advect<VAR, 1>(G, a, b, uko, vke, wo, zo, vol, st);
}

}  // namespace

// T -> out through the z and x sweeps (into mid) and the y sweep; vol: scratch volumes
void launch_ocadpo(const Geo& G, const double* T, const double* uko, const double* vke,
                   const double* wo, const double* zo, double* out, double* mid, double* vol,
                   cudaStream_t st) {
  advect_one<V_ADPO>(G, T, mid, out, uko, vke, wo, zo, vol, st);
}

// ntr tracers T[n] -> out[n], kMaxFused at a time; mid[n]: after the x sweep
void launch_ocadpo_all(const Geo& G, int ntr, const double* const* T, double* const* out,
                       double* const* mid, const double* uko, const double* vke,
                       const double* wo, const double* zo, double* vol, cudaStream_t st) {
  for (int n0 = 0; n0 < ntr; n0 += kMaxFused) {
    const int nt = ntr - n0 < kMaxFused ? ntr - n0 : kMaxFused;
    TrIO a{}, b{};
    for (int n = 0; n < nt; ++n) {
      a.in[n] = T[n0 + n];
      a.out[n] = mid[n0 + n];
      b.in[n] = mid[n0 + n];
      b.out[n] = out[n0 + n];
    }
    switch (nt) {
      case 1: advect<V_ADPO, 1>(G, a, b, uko, vke, wo, zo, vol, st); break;
      case 2: advect<V_ADPO, 2>(G, a, b, uko, vke, wo, zo, vol, st); break;
      case 3: advect<V_ADPO, 3>(G, a, b, uko, vke, wo, zo, vol, st); break;
      default: advect<V_ADPO, 4>(G, a, b, uko, vke, wo, zo, vol, st); break;
    }
  }
}

void launch_ocuad(const Geo& G, const double* T, const double* uko, const double* vke,
                  const double* wo, double* out, double* mid, double* vol, cudaStream_t st) {
  advect_one<V_UAD>(G, T, mid, out, uko, vke, wo, nullptr, vol, st);
}

void launch_ocvad(const Geo& G, const double* T, const double* uko, const double* vke,
                  const double* wo, double* out, double* mid, double* vol, cudaStream_t st) {
  advect_one<V_VAD>(G, T, mid, out, uko, vke, wo, nullptr, vol, st);
}

void launch_ocwad(const Geo& G, const double* T, const double* uko, const double* vke,
                  const double* wo, const double* zo, double* out, double* mid, double* vol,
                  cudaStream_t st) {
  advect_one<V_WAD>(G, T, mid, out, uko, vke, wo, zo, vol, st);
}

}  // namespace orctm
