// Implicit vertical diffusion: tridiagonal solves of many water columns at
// once, each column shared by G threads of a block.
//
// A block holds W neighbouring columns of one row, one thread per column and
// chunk of LC consecutive levels (consecutive threads are consecutive columns:
// coalesced).  Everything a thread needs of its levels is loaded once, together,
// and stays in registers.  The Thomas recurrences cross the chunks as scans through
// shared memory:
//   - the eliminated diagonal t(K) = b(K) - c(K-1) a(K) / t(K-1): a chunk is
//     one linear fractional map of the value above it;
//   - the forward and backward substitutions: affine maps.
// One thread per column, the form before, forms the values level by
// level: it waits a memory latency every few levels and divides
// six times a level.  This form takes the pivots' reciprocals once and refines the
// quotients with them: products with the reciprocals alone left the results two per
// cent further from an 80-bit evaluation than the plain elimination, which refined they
// equal (k_na_vert 42 us instead of 38 on 150 x 137 x 90, k_visc_w 188 either way on 301 x 403 x 67).
#pragma once
#include "common.cuh"

namespace orctm {

template <int W_, int G_, int LC_>
struct TriLane {
  static constexpr int W = W_, G = G_, LC = LC_, NT = W_ * G_;
  int c, g, K0;
  __device__ __forceinline__ TriLane() : c(threadIdx.x % W), g(threadIdx.x / W), K0(g * LC) {}
};

// The scans' shared memory: the backward maps take the place of the diagonal's
template <typename Ln, int N>
struct TriScan {
  static constexpr int M = N + 1 > 4 ? N + 1 : 4;
  double m[M][Ln::G][Ln::W], f[N + 1][Ln::G][Ln::W];
};

// Solves a(K) x(K-1) + b(K) x(K) + c(K) x(K+1) = x(K) in place for N right-hand
// sides.  a is 0 in the first row; cprev is c of the row above the thread's first.
// Rows past the last are to be a = c = x = 0, b = 1.  Every thread of the block calls it.
template <typename Ln, int N>
__device__ __forceinline__ void tri_solve(const Ln& t, TriScan<Ln, N>& s, double (&a)[Ln::LC],
                                          double (&b)[Ln::LC], double (&c)[Ln::LC], double cprev,
                                          double (&x)[N][Ln::LC]) {
  constexpr int LC = Ln::LC, G = Ln::G;
  {
    // t_out = (p t_in + q) / (r t_in + w); a row without coupling starts afresh
    double p = 1., q = 0., r = 0., w = 1.;
#pragma unroll
    for (int u = 0; u < LC; ++u) {
      const double ca = (u ? c[u - 1] : cprev) * a[u];
      const double np = fma(b[u], p, -(ca * r)), nq = fma(b[u], q, -(ca * w));
      const bool cut = ca == 0.;
      r = cut ? 0. : p;
      w = cut ? 1. : q;
      p = cut ? 0. : np;
      q = cut ? b[u] : nq;
    }
    s.m[0][t.g][t.c] = p;
    s.m[1][t.g][t.c] = q;
    s.m[2][t.g][t.c] = r;
    s.m[3][t.g][t.c] = w;
  }
  __syncthreads();
  double tp = 1.;
  for (int k = 0; k < t.g; ++k)
    tp = div_nr(fma(s.m[0][k][t.c], tp, s.m[1][k][t.c]), fma(s.m[2][k][t.c], tp, s.m[3][k][t.c]));
  // minus the multipliers m(K) = a(K) / t(K-1) into a, t(K) into b, 1 / t(K) into r where
  // that costs no block per SM (else it is formed twice)
  constexpr bool kKeep = LC >= 4 && LC <= 10;
  double rp = div_nr(1., tp), cp = cprev, r[kKeep ? LC : 1];
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    const double m = quotient(a[u], tp, rp);
    tp = fma(-cp, m, b[u]);
    rp = div_nr(1., tp);
    if (kKeep) r[u] = rp;
    cp = c[u];
    a[u] = -m;
    b[u] = tp;
  }
  double A = 1., B[N];
#pragma unroll
  for (int n = 0; n < N; ++n) B[n] = 0.;
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    A *= a[u];
#pragma unroll
    for (int n = 0; n < N; ++n) B[n] = fma(a[u], B[n], x[n][u]);
  }
  s.f[N][t.g][t.c] = A;
#pragma unroll
  for (int n = 0; n < N; ++n) s.f[n][t.g][t.c] = B[n];
  __syncthreads();
#pragma unroll
  for (int n = 0; n < N; ++n) B[n] = 0.;
  for (int k = 0; k < t.g; ++k) {
    const double Ak = s.f[N][k][t.c];
#pragma unroll
    for (int n = 0; n < N; ++n) B[n] = fma(Ak, B[n], s.f[n][k][t.c]);
  }
  // the forward values into x, 1 / t(K) into a
#pragma unroll
  for (int u = 0; u < LC; ++u) {
#pragma unroll
    for (int n = 0; n < N; ++n) {
      B[n] = fma(a[u], B[n], x[n][u]);
      x[n][u] = B[n];
    }
    a[u] = kKeep ? r[u] : div_nr(1., b[u]);
  }
  A = 1.;
#pragma unroll
  for (int n = 0; n < N; ++n) B[n] = 0.;
#pragma unroll
  for (int u = LC - 1; u >= 0; --u) {
    const double l = -(c[u] * a[u]);
    A *= l;
#pragma unroll
    for (int n = 0; n < N; ++n) B[n] = fma(l, B[n], x[n][u] * a[u]);
  }
  s.m[N][t.g][t.c] = A;
#pragma unroll
  for (int n = 0; n < N; ++n) s.m[n][t.g][t.c] = B[n];
  __syncthreads();
#pragma unroll
  for (int n = 0; n < N; ++n) B[n] = 0.;
  for (int k = G - 1; k > t.g; --k) {
    const double Ak = s.m[N][k][t.c];
#pragma unroll
    for (int n = 0; n < N; ++n) B[n] = fma(Ak, B[n], s.m[n][k][t.c]);
  }
#pragma unroll
  for (int u = LC - 1; u >= 0; --u)
#pragma unroll
    for (int n = 0; n < N; ++n) {
      B[n] = quotient(fma(-c[u], B[n], x[n][u]), b[u], a[u]);
      x[n][u] = B[n];
    }
}

// Calls f with the TriLane type for rows of `ke` levels: 16 chunks of 3 to 7
// levels, in longer columns half as many columns per block and up to 20 levels
// (the registers of a thread hold 3 + N values per level).
template <typename F>
void with_tri_split(int ke, F&& f) {
  if (ke <= 48) f((TriLane<32, 16, 3>*)nullptr);
  else if (ke <= 64) f((TriLane<32, 16, 4>*)nullptr);
  else if (ke <= 80) f((TriLane<32, 16, 5>*)nullptr);
  else if (ke <= 96) f((TriLane<32, 16, 6>*)nullptr);
  else if (ke <= 112) f((TriLane<32, 16, 7>*)nullptr);
  else if (ke <= 160) f((TriLane<16, 16, 10>*)nullptr);
  else f((TriLane<16, 16, 20>*)nullptr);
}
static_assert(16 * 20 >= kMaxKe, "the longest column has a split");

}  // namespace orctm
