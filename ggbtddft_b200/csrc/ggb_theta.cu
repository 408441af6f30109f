// Hartree potential of the theta form from every multipole L = 0 .. 2 l_max (GGB_RUN_THETA with
// n_har > 4; not in the reference, whose density multipoles stop at L = 3,
// hartreePotentialDensity.cuh:1-181, and whose Hartree sum is the O(N_r^2) loop of
// h_calculateHartreePotential.cuh:1-56).
//
// Per run and step, from the orbitals x[l][col][r] at the end of the step:
//  k_theta_density  the density on a Gauss-Legendre grid of 2 N_l nodes +-x_q, exact for every
//                   multipole up to 2 l_max: per orbital f(+-x_q) = E_q +- O_q with E (O) the sum over
//                   l - m even (odd) of x_l Theta_l^m(x_q); summed over the run's orbitals,
//                   S_q = sum occ 2 (|E|^2 + |O|^2) = rho(x_q) + rho(-x_q) and
//                   D_q = sum occ 4 Re(E conj O)  = rho(x_q) - rho(-x_q);
//                   then rho_L(r) = sum_q w_q P_L(x_q) (S_q for even L, D_q for odd L).
//  k_theta_hartree  v_L(r_a) = sum_b rho_L(b) r_<^L / r_>^(L+1) as two linear recurrences with ratios
//                   of radii (no power of r over- or underflows):
//                     A_a = (r_(a-1)/r_a)^L A_(a-1) + rho_a,  B_a = (r_a/r_(a+1))^(L+1) (B_(a+1) + rho_(a+1)),
//                     v_L(r_a) = (A_a + B_a) / r_a,
//                   each evaluated by a warp: sequential over a chunk of radii per lane, then a warp
//                   scan of the chunks' affine maps.
//  k_theta_table    htab[m][j][r] = sum_{L>=1} v_L(r) P_L(x_j^m): the multipoles' potential at the
//                   nodes of the angular phase (the monopole and exchange changes come from k_finalize
//                   and enter the phase as in the theta form with n_har <= 4).
// k_finalize runs beside them (they share no buffer): in the step's graph it is a parallel branch.
#include <cuda_runtime.h>

#include <algorithm>

#include "ggb_internal.cuh"

namespace ggb {

// Blocks own TH_R radii: everything of those radii (the l-vectors, the densities at the nodes, the
// potentials' multipoles) sits in shared memory, so that a single run (the helium configuration: 400
// radii) is 100 blocks.  The tables come through shared memory too, TH_ROWS rows at a time into one of
// two buffers by cp.async: all of a chunk's lines are in flight at once.  (Read from L2 in the loops,
// eight loads ahead, the projection and the table waited a memory latency for every eight terms.)
// Lanes: radius fastest, then eight nodes, multipoles or channels.  One output per thread and round.
// Latency bound.  Helium configuration (N_r 400, N_l 65, 129 multipoles), with k_finalize beside them:
// 27 us a step; as four kernels of a warp per (32 radii, node or multipole) that read every row
// from L2, and k_finalize after them: 73.
constexpr int TH_R = 4;
constexpr int TH_ILP = 8;         // independent partial sums of the projection and table loops
constexpr int TH_ROWS = 32;       // table rows per chunk (a multiple of TH_ILP)

// pairwise sum of the partial sums
__device__ __forceinline__ double sum_partials(const double (&a)[TH_ILP]) {
  return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// body(row0, n, rows in shared memory) for the chunks of `rows` table rows of `cols` doubles (row stride
// ld in memory, cols in shared memory), the next chunk on its way meanwhile.  Every thread of the block
// takes part; body must not synchronise the block.
template <class Body>
__device__ __forceinline__ void table_chunks(const double* table, int rows, int cols, int ld, double* buf, Body body) {
  auto fetch = [&](int c) {
    const int row0 = c * TH_ROWS, n = min(TH_ROWS, rows - row0);
    double* dst = buf + (c & 1) * TH_ROWS * cols;
    for (int i = threadIdx.x; i < n * cols; i += blockDim.x) {
      const int row = i / cols, col = i - row * cols;
      cp_async8(dst + i, table + (size_t)(row0 + row) * ld + col);
    }
    cp_async_commit();
  };
  const int chunks = (rows + TH_ROWS - 1) / TH_ROWS;
  __syncthreads();                   // the buffers are free
  if (chunks > 0) fetch(0);
  for (int c = 0; c < chunks; ++c) {
    if (c + 1 < chunks) fetch(c + 1);
    else cp_async_commit();
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    body(c * TH_ROWS, min(TH_ROWS, rows - c * TH_ROWS), (const double*)(buf + (c & 1) * TH_ROWS * cols));
    __syncthreads();
  }
}

// S and D of the run's orbitals at the positive fine nodes, accumulated over the orbitals in order, then
// the projections
__global__ void __launch_bounds__(1024) k_theta_density(GroupArgs g, ThetaArgs t, const double2* __restrict__ x) {
  extern __shared__ __align__(16) double th_sm[];
  const int nq = t.nq, n_l = g.n_l, n_r = g.n_r, n_mp = t.n_mp;
  double2* xs = reinterpret_cast<double2*>(th_sm);              // [N_l][TH_R]
  double* fs = th_sm + 2 * (size_t)n_l * TH_R;                  // [2][nq][TH_R]
  double* buf = fs + 2 * (size_t)nq * TH_R;                     // two table chunks
  const int tiles = (n_r + TH_R - 1) / TH_R;
  const int ri = blockIdx.x / tiles, r0 = (blockIdx.x - ri * tiles) * TH_R;
  const RunDev run = g.runs[ri];
  const int tid = threadIdx.x, p = tid % TH_R, item = tid / TH_R;   // this thread's node, then its multipole
  double S = 0.0, D = 0.0;
  for (int k = 0; k < run.n_orb; ++k) {
    const int col = run.col0 + k;
    const int m = g.col_m[col];
    const double occ = (double)g.col_occ[col];
    __syncthreads();                                            // the tile of the orbital before is done with
    for (int i = tid; i < n_l * TH_R; i += blockDim.x) {
      const int l = i / TH_R, r = r0 + i % TH_R;
      xs[i] = r < n_r ? x[((size_t)l * g.n_cols + col) * n_r + r] : make_double2(0.0, 0.0);
    }
    double2 e = make_double2(0.0, 0.0), o = make_double2(0.0, 0.0);
    // rows l = m .. N_l - 1 of Theta_l^m at every node (chunks start at even l - m)
    table_chunks(t.T + ((size_t)m * n_l + m) * nq, n_l - m, nq, nq, buf, [&](int row0, int n, const double* T) {
      if (item < nq) {
        const double2* xl = xs + (m + row0) * TH_R + p;
        int u = 0;
        for (; u + 1 < n; u += 2) {
          const double te = T[u * nq + item], to = T[(u + 1) * nq + item];
          const double2 xe = xl[u * TH_R], xo = xl[(u + 1) * TH_R];
          e.x = fma(te, xe.x, e.x);
          e.y = fma(te, xe.y, e.y);
          o.x = fma(to, xo.x, o.x);
          o.y = fma(to, xo.y, o.y);
        }
        if (u < n) {
          const double te = T[u * nq + item];
          const double2 xe = xl[u * TH_R];
          e.x = fma(te, xe.x, e.x);
          e.y = fma(te, xe.y, e.y);
        }
      }
    });
    S += occ * 2.0 * (e.x * e.x + e.y * e.y + o.x * o.x + o.y * o.y);
    D += occ * 4.0 * (e.x * o.x + e.y * o.y);
  }
  if (item < nq) {
    fs[item * TH_R + p] = S;
    fs[(nq + item) * TH_R + p] = D;
  }
  for (int L0 = 0; L0 < n_mp; L0 += blockDim.x / TH_R) {
    const int L = L0 + item;
    double acc[TH_ILP];
#pragma unroll
    for (int u = 0; u < TH_ILP; ++u) acc[u] = 0.0;
    const int cols = min((int)(blockDim.x / TH_R), n_mp - L0);
    table_chunks(t.wP + L0, nq, cols, n_mp, buf, [&](int row0, int n, const double* w) {
      if (L >= n_mp) return;
      const double* src = fs + ((size_t)(L & 1) * nq + row0) * TH_R + p;
      int q = 0;
      for (; q + TH_ILP - 1 < n; q += TH_ILP)
#pragma unroll
        for (int u = 0; u < TH_ILP; ++u) acc[u] = fma(w[(q + u) * cols + item], src[(q + u) * TH_R], acc[u]);
      for (; q < n; ++q) acc[0] = fma(w[q * cols + item], src[q * TH_R], acc[0]);
    });
    if (L < n_mp && r0 + p < n_r) t.rho[((size_t)ri * n_mp + L) * n_r + r0 + p] = sum_partials(acc);
  }
}

// affine map a -> mul a + add, composed in the order of the recurrence
struct Aff {
  double mul, add;
};
__device__ __forceinline__ Aff aff_then(Aff first, Aff second) {
  return Aff{second.mul * first.mul, fma(second.mul, first.add, second.add)};
}

// one warp (block) per (run, L >= 1), the rows it scans in shared memory
__global__ void __launch_bounds__(32) k_theta_hartree(GroupArgs g, ThetaArgs t) {
  extern __shared__ __align__(16) double th_sm[];
  const int lane = threadIdx.x;
  const int ri = blockIdx.x / (t.n_mp - 1);
  const int L = 1 + blockIdx.x - ri * (t.n_mp - 1);
  const int n = g.n_r;
  // rho_L, (r_(a-1)/r_a)^L and (r_(a-1)/r_a)^(L+1) (the grid's table)
  double *rho = th_sm, *fL = th_sm + n, *gL = th_sm + 2 * n;
  const double* rho_g = t.rho + ((size_t)ri * t.n_mp + L) * n;
  const double* rq_g = t.rq + (size_t)L * n;
  for (int a = lane; a < n; a += 32) {
    cp_async8(rho + a, rho_g + a);
    cp_async8(fL + a, rq_g + a);
    cp_async8(gL + a, rq_g + n + a);
  }
  cp_async_commit();
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  double* v = fL;               // a lane writes v[a] after its last use of fL[a]
  const int C = (n + 31) / 32;
  const int a0 = lane * C, a1 = min(n, a0 + C);
  // forward: A_a = f_a A_(a-1) + rho_a, f_a = (r_(a-1)/r_a)^L, f_0 = 0
  Aff mine{1.0, 0.0};
  for (int a = a0; a < a1; ++a) {
    const double f = a == 0 ? 0.0 : fL[a];
    mine = Aff{f * mine.mul, fma(f, mine.add, rho[a])};
  }
  Aff inc = mine;                       // inclusive scan of the lanes' maps, in lane order
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const Aff o{__shfl_up_sync(0xffffffffu, inc.mul, d), __shfl_up_sync(0xffffffffu, inc.add, d)};
    if (lane >= d) inc = aff_then(o, inc);
  }
  double A = __shfl_up_sync(0xffffffffu, inc.add, 1);   // A_(a0 - 1): the previous lanes' maps applied to 0
  if (lane == 0) A = 0.0;
  for (int a = a0; a < a1; ++a) {
    const double f = a == 0 ? 0.0 : fL[a];
    A = fma(f, A, rho[a]);
    v[a] = A;
  }
  // backward: B_a = g_a (B_(a+1) + rho_(a+1)), g_a = (r_a/r_(a+1))^(L+1), B_(n-1) = 0;
  // lane order reversed: the last chunk first
  const int bl = 31 - lane;
  const int b0 = bl * C, b1 = min(n, b0 + C);
  Aff mb{1.0, 0.0};
  for (int a = b1 - 1; a >= b0; --a) {
    const double gg = a == n - 1 ? 0.0 : gL[a + 1];
    const double rn = a == n - 1 ? 0.0 : rho[a + 1];
    mb = Aff{gg * mb.mul, gg * (mb.add + rn)};
  }
  Aff ib = mb;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const Aff o{__shfl_up_sync(0xffffffffu, ib.mul, d), __shfl_up_sync(0xffffffffu, ib.add, d)};
    if (lane >= d) ib = aff_then(o, ib);
  }
  double B = __shfl_up_sync(0xffffffffu, ib.add, 1);
  if (lane == 0) B = 0.0;
  __syncwarp();
  for (int a = b1 - 1; a >= b0; --a) {
    const double gg = a == n - 1 ? 0.0 : gL[a + 1];
    const double rn = a == n - 1 ? 0.0 : rho[a + 1];
    B = gg * (B + rn);
    v[a] += B;
  }
  __syncwarp();
  double* v_g = t.vmp + ((size_t)ri * t.n_mp + L) * n;
  for (int a = lane; a < n; a += 32) v_g[a] = v[a] / g.r[a];
}

// htab[m][j][r] = sum_{L>=1} v_L(r) P_L(x_j^m), TH_ILP partial sums over L; blocks (run, m, radii)
__global__ void __launch_bounds__(1024) k_theta_table(GroupArgs g, ThetaArgs t) {
  extern __shared__ __align__(16) double th_sm[];
  const int n_r = g.n_r, n_mp = t.n_mp, n_l = g.n_l;
  const int tiles = (n_r + TH_R - 1) / TH_R;
  const int rm = blockIdx.x / tiles, r0 = (blockIdx.x - rm * tiles) * TH_R;
  const int ri = rm / g.n_m, m = rm - ri * g.n_m;
  const RunDev run = g.runs[ri];
  double* vs = th_sm;                                           // [n_mp][TH_R]
  double* buf = th_sm + (size_t)n_mp * TH_R;                    // two table chunks
  const double* v = t.vmp + (size_t)ri * n_mp * n_r;
  for (int i = threadIdx.x; i < n_mp * TH_R; i += blockDim.x) {
    const int L = i / TH_R, r = r0 + i % TH_R;
    vs[i] = L > 0 && r < n_r ? v[(size_t)L * n_r + r] : 0.0;
  }
  const int p = threadIdx.x % TH_R, j = threadIdx.x / TH_R;
  double acc[TH_ILP];
#pragma unroll
  for (int u = 0; u < TH_ILP; ++u) acc[u] = 0.0;
  table_chunks(t.PLj + ((size_t)m * n_mp + 1) * g.ldS, n_mp - 1, n_l, g.ldS, buf, [&](int row0, int n, const double* P) {
    if (j < m || j >= n_l) return;
    const double* vl = vs + (1 + row0) * TH_R + p;
    int q = 0;
    for (; q + TH_ILP - 1 < n; q += TH_ILP)
#pragma unroll
      for (int u = 0; u < TH_ILP; ++u) acc[u] = fma(vl[(q + u) * TH_R], P[(q + u) * n_l + j], acc[u]);
    for (; q < n; ++q) acc[0] = fma(vl[q * TH_R], P[q * n_l + j], acc[0]);
  });
  if (j < n_l && r0 + p < n_r) run.htab[((size_t)m * n_l + j) * n_r + r0 + p] = sum_partials(acc);
}

static int theta_threads(int items) { return std::min(1024, (items * TH_R + 31) / 32 * 32); }
static size_t theta_density_smem(int n_l, int nq, int threads) {
  return ((size_t)(2 * n_l + 2 * nq) * TH_R + 2 * (size_t)TH_ROWS * std::max(nq, threads / TH_R)) * sizeof(double);
}

cudaError_t configure_theta(int optin) {
  for (const void* fn : {(const void*)k_theta_density, (const void*)k_theta_hartree, (const void*)k_theta_table}) {
    const cudaError_t e = set_max_dynamic_smem(fn, optin);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

void launch_theta_potentials(const GroupArgs& g, const ThetaArgs& t, const double2* x, cudaStream_t s) {
  const int tiles = (g.n_r + TH_R - 1) / TH_R;
  const int threads = theta_threads(std::max(t.nq, t.n_mp));    // >= nq TH_R: N_l <= 220
  k_theta_density<<<g.n_runs * tiles, threads, theta_density_smem(g.n_l, t.nq, threads), s>>>(g, t, x);
  if (t.n_mp > 1) k_theta_hartree<<<g.n_runs * (t.n_mp - 1), 32, 3 * (size_t)g.n_r * sizeof(double), s>>>(g, t);
  k_theta_table<<<g.n_runs * g.n_m * tiles, theta_threads(g.n_l),
                  ((size_t)t.n_mp * TH_R + 2 * (size_t)TH_ROWS * g.n_l) * sizeof(double), s>>>(g, t);
}

}  // namespace ggb
