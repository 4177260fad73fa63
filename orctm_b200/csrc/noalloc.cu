// orctm_octdiff_noalloc: tracer diffusion of one tracer (OCTDIFF_BASE +
// OCTDIFF_TS) for callers that cannot allocate device memory.
//
// Who needs it.  Some callers are not allowed to call cudaMalloc: code that
// runs while a CUDA graph is being captured (an allocation would break the
// capture), host programs whose device memory is owned by another runtime or
// pool (an OpenACC/OpenMP-offload Fortran model, a framework allocator) and
// must not take memory behind its back, and time-critical loops that must
// not block on the driver's allocator.  orctm_create needs device memory for
// its handle; this entry point needs none: the caller passes device pointers
// to every input and output in the reference's own Fortran layouts, and the
// two scratch fields the routine needs live in one fixed array compiled into
// the library.
//
// The scratch array.  g_noalloc_scratch below is a file-scope __device__
// array of kNoAllocMaxCells * 2 doubles (32 MiB).  Every GPU that loads the
// library holds it until the process exits.  All calls on a device share it
// and it keeps the last call's contents; every element a call reads was
// written earlier in that same call, so nothing has to be cleared between
// calls.  Calls whose kernels overlap on the GPU (different streams, or
// host threads, without ordering) race on it: order them on one stream.
//
// The device address of the array is looked up with cudaGetSymbolAddress on
// the first call made on each device, with that device current; make that
// first call before any stream capture begins.  Sizes beyond the maximum are
// rejected with ORCTM_E_TOO_LARGE before anything is launched.
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/orctm_gpu.h"
#include "common.cuh"
#include "ops.h"
#include "tridiag.cuh"

namespace orctm {

namespace {

constexpr long long kNoAllocMaxCells = 1LL << 21;  // IE*JE*KE limit, 2,097,152 cells
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) double g_noalloc_scratch[2 * kNoAllocMaxCells];

std::mutex g_na_mutex;
double* g_na_ptr[kNoAllocMaxDevices] = {};

struct NaArgs {
  int IE, JE, KE;
  double dt, almzer, aulapts;
  const double *dvo, *ddpo, *weto, *di, *dzw, *dlxp, *dlyp, *dlxu, *dlyu, *dlxv, *dlyv, *zo;
};

// Fortran-layout accessors (p-points 1..IE x 1..JE, u-points 0..IE, v-points 0..JE)
__device__ __forceinline__ long long p3(const NaArgs& a, int i, int j, int k) {
  return ((long long)(k - 1) * a.JE + (j - 1)) * a.IE + (i - 1);
}
__device__ __forceinline__ long long p2(const NaArgs& a, int i, int j) {
  return (long long)(j - 1) * a.IE + (i - 1);
}
__device__ __forceinline__ long long u2(const NaArgs& a, int i, int j) {
  return (long long)(j - 1) * (a.IE + 1) + i;
}
__device__ __forceinline__ long long v2(const NaArgs& a, int i, int j) {
  return (long long)j * a.IE + (i - 1);
}

// implicit vertical diffusion (octdiff_base.f90:182-204, octdiff_ts.f90:294-324);
// columns outside the interior are copied
template <typename Ln>
__global__ void __launch_bounds__(Ln::NT) k_na_vert(NaArgs a, const double* __restrict__ T,
                                                    double* __restrict__ O) {
  constexpr int LC = Ln::LC;
  __shared__ TriScan<Ln, 1> scan;
  const Ln t;
  const int IE = a.IE, JE = a.JE, KE = a.KE, pl = IE * JE;
  const int nb = (IE + Ln::W - 1) / Ln::W;
  const int i = blockIdx.x % nb * Ln::W + t.c + 1, j = blockIdx.x / nb + 1;
  const bool valid = i <= IE;
  const bool interior = i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  const int base = (int)p3(a, i, j, t.K0 + 1);
  double x[1][LC], ta[LC], tb[LC], tc[LC], d[LC + 1], th[LC], wt[LC];
#pragma unroll
  for (int u = 0; u <= LC; ++u)
    d[u] = interior && t.K0 + 1 + u <= KE + 1 ? a.dvo[base + u * pl] : 0.;
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    const bool ok = t.K0 + 1 + u <= KE;
    x[0][u] = valid && ok ? T[base + u * pl] : 0.;
    th[u] = interior && ok ? a.ddpo[base + u * pl] : 0.;
    wt[u] = interior && ok ? a.weto[base + u * pl] : 0.;
  }
  const bool above = interior && t.K0 > 0 && t.K0 < KE;
  const double thp = above ? a.ddpo[base - pl] : 0.;
  const double zo = interior ? a.zo[p2(a, i, j)] : 0.;
  auto den = [&](int K, double dd) {
    const double zzsurf = K == 1 ? 1. : 0.;
    return dd + zzsurf * (zo) + a.almzer;
  };
#pragma unroll
  for (int u = 0; u < LC; ++u) {
    const int K = t.K0 + 1 + u;
    ta[u] = tc[u] = 0.;
    tb[u] = 1.;
    if (interior && K <= KE) {
      const double dn = den(K, th[u]), rd = div_nr(1., dn);
      ta[u] = quotient(-a.dt * d[u] * wt[u] * a.di[K - 1], dn, rd);
      tc[u] = quotient(-a.dt * d[u + 1] * a.di[K], dn, rd);
      tb[u] = 1. - ta[u] - tc[u];
      if (K == 1) ta[u] = 0.;
    }
  }
  const double cprev = above ? -a.dt * d[0] * a.di[t.K0] / den(t.K0, thp) : 0.;
  if (valid && !interior) {
#pragma unroll
    for (int u = 0; u < LC; ++u)
      if (t.K0 + 1 + u <= KE) O[base + u * pl] = x[0][u];
  }
  tri_solve<Ln, 1>(t, scan, ta, tb, tc, cprev, x);
  if (interior) {
#pragma unroll
    for (int u = 0; u < LC; ++u)
      if (t.K0 + 1 + u <= KE) O[base + u * pl] = x[0][u];
  }
}

// The horizontal passes: a thread takes kNaLevels levels of a column, so that
// the divisions by the metrics are made once for them.
constexpr int kNaLevels = 6;

// masked Laplacian (octdiff_ts.f90:346-362); halo cells are written as 0
__global__ void __launch_bounds__(128) k_na_lap(NaArgs a, const double* __restrict__ T,
                                                double* __restrict__ L1) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int IE = a.IE, JE = a.JE, pl = IE * JE, K0 = blockIdx.z * kNaLevels;
  if (i > IE || j > JE) return;
  const bool inner = i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  double rxw = 0., rxe = 0., rxp = 0., ryn = 0., rys = 0., ryp = 0.;
  if (inner) {
    rxw = 1. / a.dlxu[u2(a, i - 1, j)];
    rxe = 1. / a.dlxu[u2(a, i, j)];
    rxp = 1. / a.dlxp[p2(a, i, j)];
    ryn = 1. / a.dlyv[v2(a, i, j - 1)];
    rys = 1. / a.dlyv[v2(a, i, j)];
    ryp = 1. / a.dlyp[p2(a, i, j)];
  }
  const int c = (int)p3(a, i, j, K0 + 1);
#pragma unroll
  for (int q = 0; q < kNaLevels; ++q) {
    const int o = c + q * pl;
    if (K0 + q >= a.KE) break;
    double r = 0.0;
    if (inner) {
      const double t = T[o];
      r = a.weto[o] * ((a.weto[o - 1] * (T[o - 1] - t) * rxw + a.weto[o + 1] * (T[o + 1] - t) * rxe) * rxp +
                       (a.weto[o - IE] * (T[o - IE] - t) * ryn + a.weto[o + IE] * (T[o + IE] - t) * rys) * ryp);
    }
    L1[o] = r;
  }
}

// biharmonic update (octdiff_ts.f90:369-399)
__global__ void __launch_bounds__(128) k_na_bih(NaArgs a, const double* __restrict__ T,
                                                const double* __restrict__ L1,
                                                double* __restrict__ O) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int IE = a.IE, JE = a.JE, pl = IE * JE, K0 = blockIdx.z * kNaLevels;
  if (i > IE || j > JE) return;
  const bool inner = i >= 2 && i <= IE - 1 && j >= 2 && j <= JE - 1;
  double fw = 0., fe = 0., fn = 0., fs = 0., area = 0., z = 0.;
  if (inner) {
    // AULX DLYU / DLXU and AULY DLXV / DLYV of the four faces
    auto fx = [&](int ii) {
      const double x = a.dlxu[u2(a, ii, j)];
      return a.aulapts * ((x * x) * (x * x)) * a.dlyu[u2(a, ii, j)] / x;
    };
    auto fy = [&](int jj) {
      const double y = a.dlyv[v2(a, i, jj)];
      return a.aulapts * ((y * y) * (y * y)) * a.dlxv[v2(a, i, jj)] / y;
    };
    fw = fx(i - 1);
    fe = fx(i);
    fn = fy(j - 1);
    fs = fy(j);
    area = a.dlxp[p2(a, i, j)] * a.dlyp[p2(a, i, j)];
    z = a.zo[p2(a, i, j)];
  }
  const int o0 = (int)p3(a, i, j, K0 + 1);
#pragma unroll
  for (int q = 0; q < kNaLevels; ++q) {
    const int o = o0 + q * pl, K = K0 + q + 1;
    if (K > a.KE) break;
    const double t = T[o];
    double r = t;
    if (inner) {
      const double zzsurf = K == 1 ? 1. : 0.;
      const double c = L1[o];
      const double den = (a.ddpo[o] + a.almzer + zzsurf * (z)) * area;
      r = t - (a.weto[o] / den) * a.dzw[K - 1] *
                  (a.weto[o - 1] * fw * (L1[o - 1] - c) + a.weto[o + 1] * fe * (L1[o + 1] - c) +
                   a.weto[o - IE] * fn * (L1[o - IE] - c) + a.weto[o + IE] * fs * (L1[o + IE] - c));
    }
    O[o] = r;
  }
}

// Device address of the scratch array on the current device.  The first call
// on a device looks it up (cudaGetSymbolAddress, with that device current).
// Later calls look it up again when their stream is not being captured, so
// an address cached before a cudaDeviceReset (which unloads the module and
// may place the array elsewhere) is not reused; a call on a capturing stream
// uses the cached address, so the first call on a device must come before
// any capture, and a device reset must be followed by one call outside a
// capture before the next capture.
int scratch_for_current_device(cudaStream_t s, double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_status(e);
  if (dev < 0 || dev >= kNoAllocMaxDevices) {
    set_unbound_error("device ordinal beyond the no-allocation table");
    return ORCTM_E_ARG;
  }
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  const bool capturing = cudaStreamIsCapturing(s, &cs) != cudaSuccess ||
                         cs != cudaStreamCaptureStatusNone;
  std::lock_guard<std::mutex> lk(g_na_mutex);
  if (!g_na_ptr[dev] || !capturing) {
    if (capturing) {
      set_unbound_error("the first call on a device must not be made under stream capture");
      return ORCTM_E_ARG;
    }
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      const int st = cuda_status(e);
      set_unbound_error((std::string("cudaGetSymbolAddress failed: ") + cudaGetErrorString(e)).c_str());
      return st;
    }
    g_na_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_na_ptr[dev];
  return ORCTM_OK;
}

}  // namespace
}  // namespace orctm

using namespace orctm;

extern "C" int orctm_octdiff_noalloc(const orctm_octdiff_noalloc_args* in) {
  clear_unbound_errors();
  if (!in) {
    set_unbound_error("null argument block");
    return ORCTM_E_ARG;
  }
  const long long cells = (long long)in->ie * in->je * in->ke;
  if (in->ie < 3 || in->je < 3 || in->ke < 2 || in->ke > kMaxKe) {
    set_unbound_error("grid size out of range");
    return ORCTM_E_ARG;
  }
  if (cells > kNoAllocMaxCells) {
    set_unbound_error("IE*JE*KE exceeds the no-allocation limit of 2097152 cells");
    return ORCTM_E_TOO_LARGE;
  }
  const void* req[] = {in->tracer_in, in->tracer_out, in->dvo, in->ddpo, in->weto, in->di,
                       in->dzw, in->dlxp, in->dlyp, in->dlxu, in->dlyu, in->dlxv, in->dlyv,
                       in->zo};
  for (const void* p : req)
    if (!p) {
      set_unbound_error("missing device pointer");
      return ORCTM_E_ARG;
    }
  if (in->tracer_in == in->tracer_out) {
    set_unbound_error("tracer_in and tracer_out must be different buffers");
    return ORCTM_E_ARG;
  }
  if (in->ah00 > in->almzer) {
    set_unbound_error("harmonic tracer diffusion (AH00 > ALMZER) is not implemented");
    return ORCTM_E_UNSUPPORTED;
  }
  cudaStream_t s = static_cast<cudaStream_t>(in->stream);
  double* scratch = nullptr;
  int st = scratch_for_current_device(s, &scratch);
  if (st != ORCTM_OK) return st;
  double* vdiff = scratch;                     // vertically diffused tracer
  double* lap = scratch + kNoAllocMaxCells;    // first Laplacian T1O
  NaArgs a{in->ie, in->je, in->ke, in->dt, in->almzer, in->aulapts, in->dvo, in->ddpo, in->weto,
           in->di, in->dzw, in->dlxp, in->dlyp, in->dlxu, in->dlyu, in->dlxv, in->dlyv, in->zo};
  const dim3 b3(32, 4);
  const dim3 g3((in->ie + 31) / 32, (in->je + 3) / 4, (in->ke + kNaLevels - 1) / kNaLevels);
  const bool bih = in->aulapts > in->almzer;
  with_tri_split(in->ke, [&](auto* l) {
    using Ln = std::remove_pointer_t<decltype(l)>;
    const int gc = (in->ie + Ln::W - 1) / Ln::W * in->je;  // rows in x: y ends at 65535
    k_na_vert<Ln><<<gc, Ln::NT, 0, s>>>(a, in->tracer_in, bih ? vdiff : in->tracer_out);
  });
  count_launch();
  if (bih) {
    k_na_lap<<<g3, b3, 0, s>>>(a, vdiff, lap);
    count_launch();
    k_na_bih<<<g3, b3, 0, s>>>(a, vdiff, lap, in->tracer_out);
    count_launch();
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e);
  return ORCTM_OK;
}
