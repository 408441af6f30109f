// ggb_observables_noalloc: dipole, acceleration and norm of a set of orbitals without any device
// allocation.
//
// Some callers cannot call cudaMalloc: code that runs inside another framework's memory pool or
// allocator (which must own every device allocation), code on a path that is being captured into a
// CUDA graph after its set-up, or a process that has reserved all device memory up front.  This
// entry point computes the same per-(l, orbital) dipole and acceleration sums and per-orbital norm
// that the time step records (dipoleMoment.cuh / dipoleAcceleration.cuh plus the norm), from
// caller-provided device-accessible buffers only.  The norm's partial sums over l live in a file-scope
// __device__ array of fixed size.
#include <cuda_runtime.h>

#include <mutex>

#include "../../include/ggbtddft.h"
#include "ggb_angular.cuh"

namespace ggb {

// Limits of a call: n_orb * N_l * ceil(N_r / 32) and n_orb * ceil(N_r / 32).
constexpr int NA_MAX_PARTIALS = 65536;
constexpr int NA_MAX_NORM = 16384;
constexpr int NA_MAX_NL = 256;

// Norm partials (dd), one per (orbital, l): n_orb * N_l <= NA_MAX_PARTIALS (1 MiB).
static __device__ __align__(256) double2 g_norm_scratch[NA_MAX_PARTIALS];

// T threads per (l, orbital) row, NA_THREADS / T rows a block.  The rows l - 1, l and l + 1 of the orbital come
// straight from L2 (each is read three times: 25 MB of L2 traffic for nine orbitals on 600 radii, 97 l), a
// thread sums its radii in double-double, and one reduction over the row's threads ends it: no partial sums
// per tile of radii, no second pass over them, and one reduction per row where the tile form (a warp
// reduction of every row for every 32 radii) made ceil(N_r / 32).  T = 128: a row of 600 radii is five loads
// per thread, all rows of a call are resident at once; bound by the latency of one load, the five sums
// and the reduction (N_r 600, N_l 97, nine orbitals: 12.3 us a call with the norm kernel, 44.7 us as tiles and
// a reduction kernel).  T = 32 up to 128 radii, where the reductions are the work: 65536 rows of 32 radii
// 60 us (128 threads: 189; tiles: 119), 25854 of 31 radii 27 (78; 43); a few hundred rows take the 6.5 us of
// the launches either way.
constexpr int NA_THREADS = 128;

template <int T>
__global__ void __launch_bounds__(NA_THREADS)
k_obs_rows(const double2* __restrict__ x, const double* __restrict__ r, const double* __restrict__ coef,
           const int* __restrict__ m_of, int n_l, int n_orb, int n_r, double2* __restrict__ dip,
           double2* __restrict__ acc, double2* __restrict__ norm_part) {
  asm volatile("griddepcontrol.launch_dependents;");
  const int row_id = blockIdx.x * (NA_THREADS / T) + threadIdx.x / T, tid = threadIdx.x % T;
  if (T < NA_THREADS && row_id >= n_l * n_orb) return;   // whole warps
  const int l = row_id / n_orb, k = row_id - l * n_orb;
  int m = m_of[k];
  if (m < 0 || m > n_l) m = n_l;   // an invalid m contributes nothing (no l satisfies l >= m)
  // dipole (re, im), acceleration (re, im), norm
  dd s[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) s[q] = dd{0.0, 0.0};
  if (l >= m) {   // here m < NA_MAX_NL
    // the first row has no lower, the last no upper neighbour (dipoleMoment.cuh:19-43)
    const bool up = l + 1 < n_l, down = l > m;
    const double c_u = (l == m || l != n_l - 1) ? coef[((size_t)CF_CU * NA_MAX_NL + m) * NA_MAX_NL + l] : 0.0;
    const double c_d = down ? coef[((size_t)CF_CD * NA_MAX_NL + m) * NA_MAX_NL + l] : 0.0;
    const size_t ls = (size_t)n_orb * n_r;
    const double2* row = x + (size_t)l * ls + (size_t)k * n_r;
    for (int i = tid; i < n_r; i += T) {
      const double2 xl = row[i];
      const double2 xu = up ? row[ls + i] : make_double2(0.0, 0.0);
      const double2 xd = down ? (row - ls)[i] : make_double2(0.0, 0.0);
      const double rr = r[i], fr2 = 1.0 / (rr * rr);
      const double zx = c_u * xu.x + c_d * xd.x, zy = c_u * xu.y + c_d * xd.y;
      // conj(x_l) . z
      const double px = xl.x * zx + xl.y * zy, py = xl.x * zy - xl.y * zx;
      s[0] = dd_add(s[0], dd{rr * px, 0.0});
      s[1] = dd_add(s[1], dd{rr * py, 0.0});
      s[2] = dd_add(s[2], dd{fr2 * px, 0.0});
      s[3] = dd_add(s[3], dd{fr2 * py, 0.0});
      s[4] = dd_add(s[4], dd{xl.x * xl.x + xl.y * xl.y, 0.0});
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 5; ++q)
      s[q] = dd_add(s[q], dd{__shfl_xor_sync(0xffffffffu, s[q].hi, o), __shfl_xor_sync(0xffffffffu, s[q].lo, o)});
  const size_t o = (size_t)l * n_orb + k;
  auto store = [&](int q, dd t) {
    if (q < 2) reinterpret_cast<double*>(dip + o)[q] = t.hi + t.lo;
    else if (q < 4) reinterpret_cast<double*>(acc + o)[q - 2] = t.hi + t.lo;
    else norm_part[(size_t)k * n_l + l] = make_double2(t.hi, t.lo);
  };
  if constexpr (T == 32) {
    if (tid == 0)
#pragma unroll
      for (int q = 0; q < 5; ++q) store(q, s[q]);
  } else {
    __shared__ dd part[T / 32][5];
    if ((tid & 31) == 0)
#pragma unroll
      for (int q = 0; q < 5; ++q) part[tid >> 5][q] = s[q];
    __syncthreads();
    if (tid < 5) {
      dd t = part[0][tid];
#pragma unroll
      for (int w = 1; w < T / 32; ++w) t = dd_add(t, part[w][tid]);
      store(tid, t);
    }
  }
}

// One warp per orbital sums the norm partials of its l.  Launched as a programmatic dependent of
// k_obs_rows: its launch overlaps that kernel, it reads after the wait.
__global__ void __launch_bounds__(32)
k_obs_norm(const double2* norm_part, int n_l, double* __restrict__ norm) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const double2* p = norm_part + (size_t)blockIdx.x * n_l;
  dd s{0.0, 0.0};
  for (int l = threadIdx.x; l < n_l; l += 32) s = dd_add(s, dd{p[l].x, p[l].y});
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    s = dd_add(s, dd{__shfl_xor_sync(0xffffffffu, s.hi, o), __shfl_xor_sync(0xffffffffu, s.lo, o)});
  if (threadIdx.x == 0) norm[blockIdx.x] = s.hi + s.lo;
}

// Angular coefficient rows c_u, c_d (l, m < NA_MAX_NL) of the observables, [coef][m][l] with rows
// NA_MAX_NL long (independent of a call's N_l, so filled once per device): the same closed forms
// as the context's tables (angularCoefficients.cuh:57-111).
static __device__ __align__(256) double g_coef[2 * NA_MAX_NL * NA_MAX_NL];

__global__ void k_fill_coef(double* coef) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NA_MAX_NL * NA_MAX_NL) return;
  const int n_l = NA_MAX_NL;
  const int m = i / n_l, l = i - m * n_l;
  const double dl = l, dm = m;
  const double cu = (l >= m) ? sqrt((pow(dl + 1.0, 2.0) - pow(dm, 2.0)) / ((2.0 * dl + 1.0) * (2.0 * dl + 3.0))) : 0.0;
  const double cd = (l >= 1 && l - 1 >= m) ? sqrt((pow(dl, 2.0) - pow(dm, 2.0)) / ((2.0 * dl + 1.0) * (2.0 * dl - 1.0)))
                                           : 0.0;
  coef[((size_t)CF_CU * NA_MAX_NL + m) * n_l + l] = cu;
  coef[((size_t)CF_CD * NA_MAX_NL + m) * n_l + l] = cd;
}

// Per-device addresses of the file-scope arrays, resolved on a device's first call.
struct NoallocDevice {
  bool ready = false;
  double2* norm = nullptr;
  double* coef = nullptr;
};
static NoallocDevice g_dev[64];
static std::mutex g_setup_mutex;

// Resolves the arrays' device addresses with `dev` current and fills the coefficient table, once
// per device (synchronously); serialised across host threads.
static int noalloc_setup(int dev) {
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  NoallocDevice& d = g_dev[dev];
  if (d.ready) return GGB_OK;
  if (cudaGetSymbolAddress((void**)&d.norm, g_norm_scratch) != cudaSuccess) return GGB_ERR_CUDA;
  if (cudaGetSymbolAddress((void**)&d.coef, g_coef) != cudaSuccess) return GGB_ERR_CUDA;
  k_fill_coef<<<(NA_MAX_NL * NA_MAX_NL + 255) / 256, 256>>>(d.coef);
  if (cudaStreamSynchronize(0) != cudaSuccess) return GGB_ERR_CUDA;
  d.ready = true;
  return GGB_OK;
}

}  // namespace ggb

extern "C" int ggb_observables_noalloc(const double* x, const double* r, const int* m, int n_l, int n_orb, int n_r,
                                       double* dip, double* acc, double* norm, void* stream) {
  using namespace ggb;
  if (!x || !r || !m || !dip || !acc || !norm) return GGB_ERR_ARG;
  if (n_l < 2 || n_l > NA_MAX_NL || n_orb < 1 || n_r < 1) return GGB_ERR_ARG;
  const int n_tiles = (n_r + TR - 1) / TR;
  if ((long long)n_orb * n_l * n_tiles > NA_MAX_PARTIALS || (long long)n_orb * n_tiles > NA_MAX_NORM)
    return GGB_ERR_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GGB_ERR_CUDA;
  const int rc = noalloc_setup(dev);
  if (rc) return rc;
  const NoallocDevice& d = g_dev[dev];
  cudaStream_t s = (cudaStream_t)stream;
  const int rows = n_l * n_orb;
  const double2* xs = reinterpret_cast<const double2*>(x);
  double2 *ds = reinterpret_cast<double2*>(dip), *as = reinterpret_cast<double2*>(acc);
  if (n_r <= NA_THREADS)
    k_obs_rows<32><<<(rows + NA_THREADS / 32 - 1) / (NA_THREADS / 32), NA_THREADS, 0, s>>>(xs, r, d.coef, m, n_l, n_orb, n_r, ds, as,
                                                                                           d.norm);
  else
    k_obs_rows<NA_THREADS><<<rows, NA_THREADS, 0, s>>>(xs, r, d.coef, m, n_l, n_orb, n_r, ds, as, d.norm);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute after{};
  after.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  after.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(n_orb);
  cfg.blockDim = dim3(32);
  cfg.stream = s;
  cfg.attrs = &after;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_obs_norm, (const double2*)d.norm, n_l, norm);
  return cudaGetLastError() == cudaSuccess ? GGB_OK : GGB_ERR_CUDA;
}
