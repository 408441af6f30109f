// FP64 (parity form) kernels of the split-operator step.
//
//  k_angular_fp64  one half of the angular step for a tile of radii of one orbital column: the
//                  whole l-vector of every radius is held in shared memory while the chain
//                  (rotate -> phase -> [pre-multiplied rotate pair] -> phase ... -> rotate back,
//                  plus the l-diagonal S phase) is applied, each product on the FP64 tensor cores
//                  (mma.sync m8n8k4).  Replaces, per half-step, the 3 launches of each of
//                  h_couplingFF/FP/D/P (couplingP.cuh:108-125, couplingD.cuh, couplingF.cuh) and
//                  h_couplingS (couplingS.cuh:43-57).  The second half also produces the
//                  density-multipole partial sums of the new orbitals
//                  (hartreePotentialDensity.cuh:1-181).  k_angular_fp64_small: the same for groups of
//                  many tiles and up to 104 channels, in smaller blocks.
//  k_radial_fp64   x_l <- A_l x_l for every l with A_l(a,b) = W[l][b][a]: the batched ZGEMM of
//                  h_propagationH0 (h_timePropagation.cuh:1-30), out of place.  More than nine
//                  columns, and large grids of one, two and six (radial_tiles): persistent, two CTAs
//                  per SM; a producer warp streams the W rows and x
//                  segments of each 16-wide k chunk into a 3-stage shared-memory ring with
//                  cp.async.bulk (mbarrier transaction counts), so that ~200 KB per SM are in flight
//                  whatever the occupancy; four consumer warps run the product on the FP64 tensor
//                  cores.  Else, up to nine columns (one run): k_radial_fp64_rows.
//  k_finalize      per run: observables of the step from the partials, density multipoles
//                  (occupation-weighted sum over orbitals), Hartree potentials by compensated
//                  prefix scans (h_calculateHartreePotential.cuh:1-136), LDA exchange
//                  (h_calculateExchangeCorrelationPotential.cuh:1-56), step counter.
#include <algorithm>
#include <cstdio>
#include "ggb_internal.cuh"
#include "ggb_angular.cuh"
#include "ggb_mixed.cuh"
#include "ggb_tc_common.cuh"

namespace ggb {

// ---------------------------------------------------------------------------------------------
// angular chain
// ---------------------------------------------------------------------------------------------

// A tile is P radii of one orbital column.  Its l-vectors sit in shared memory as a [rows][2 P + 4]
// FP64 matrix (column 2 p + 0/1 = real/imaginary part of radius p; rows N_l rounded up to 8, zero beyond
// N_l; the odd multiple of four doubles puts the fragment loads' 4 rows on different banks), and every
// product of the chain y_j = sum_l S[l][j] x_l is a small real GEMM  Y (N_l x 2 P) = S^T X  on the FP64
// tensor cores: mma.sync m8n8k4 (8 channels x 8 columns x 4 l per instruction).  The warps form 8 row
// groups x WN column groups; a warp owns the 8-channel tiles rt = group, group + 8, ... (R of them) over
// NT 8-column tiles, all of whose accumulators it holds, so that the product goes back in place: one
// copy of the tile in shared memory.  Each S element is used by one row group, so it comes straight
// from L2 into registers, laid out in fragment order (a warp's two k steps are 512 contiguous bytes),
// AM_D pairs of k steps ahead of the products; the first product's are requested before the orbitals.
// The phases are a pass over the tile by all threads (sincos per element), since the row tiles do not
// divide evenly over the warps.
//
// P follows the number of tiles (angular_points): the smallest tile while all fit on the SMs at once
// (one column on 200 radii: 50 blocks of 4 radii, where 16-radius tiles made 13 blocks), up to 40 radii
// when that fills the SMs exactly once (nine columns on 600 radii: 135 blocks; at 16 radii 342 blocks,
// 2.3 per SM, left a third of them waiting).  FP64-tensor bound at the large end (2 products x 4 N_l^2
// flop per radius and column), latency bound at the small one.
constexpr int AM_ROW_GROUPS = 8;
__host__ __device__ constexpr int angular_ldx(int points) { return 2 * points + 4; }
__host__ __device__ constexpr int angular_rows(int n_l) { return (n_l + 7) / 8 * 8; }
// lane groups of the density's partial sums
__host__ __device__ constexpr int angular_den_groups(int threads, int points) { return threads / points; }

__device__ __forceinline__ void mma_f64_8x8x4(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Density multipoles L = 0 .. n_den - 1 at one radius over l in [l0, l1) (rows of this m, l0 >= m),
// every product x_l.x_(l+d) taken once: c_u(l) serves the terms (l, l+1) and (l+1, l) of the literal
// sums, c_d(l+1) being c_u(l), and likewise for the other couplings.  For N_l >= m + 7 the literal l
// ranges cover every l once, but for l = N_l - 4 of the octupole, counted twice without its upper
// coupling (the reference's tail loop restarts there, hartreePotentialDensity.cuh:150).
template <int STRIDE>
__device__ __forceinline__ void density_window(int n_den, int n_l, const double2* xs, const double* rows, size_t rs,
                                               int l0, int l1, double (&d)[N_DEN]) {
  const double *cu = rows + CF_CU * rs, *pp = rows + CF_P * rs, *qu = rows + CF_QU * rs, *p3 = rows + CF_P3 * rs,
               *f3 = rows + CF_F3 * rs;
  auto at = [&](int l) { return l < n_l ? xs[(size_t)l * STRIDE] : make_double2(0.0, 0.0); };
  auto dot = [](double2 a, double2 b) { return a.x * b.x + a.y * b.y; };
  double2 x0 = at(l0), x1 = at(l0 + 1), x2 = at(l0 + 2);
  for (int l = l0; l < l1; ++l) {
    const double2 x3 = at(l + 3);
    const double d0 = dot(x0, x0);
    d[0] += d0;
    if (n_den > 1) {
      const double d1 = dot(x0, x1);
      d[1] += 2.0 * cu[l] * d1;
      if (n_den > 2) d[2] += pp[l] * d0 + 2.0 * qu[l] * dot(x0, x2);
      if (n_den > 3) {
        d[3] += 2.0 * (p3[l] * d1 + f3[l] * dot(x0, x3));
        if (l == n_l - 4)
          d[3] += f3[l - 3] * dot(xs[(size_t)(l - 3) * STRIDE], x0) + p3[l - 1] * dot(xs[(size_t)(l - 1) * STRIDE], x0) +
                  p3[l] * d1;
      }
    }
    x0 = x1;
    x1 = x2;
    x2 = x3;
  }
}

// One half of the angular step (or, with the empty chain of half 2, only the density): replaces, per
// half-step, the 3 launches of each of h_couplingFF/FP/D/P (couplingP.cuh:108-125, couplingD.cuh,
// couplingF.cuh) and h_couplingS (couplingS.cuh:43-57); the second half also produces the
// density-multipole partial sums of the new orbitals (hartreePotentialDensity.cuh:1-181).
template <int NT, int WN, int R>
__global__ void __launch_bounds__(AM_ROW_GROUPS * WN * 32)
k_angular_fp64(GroupArgs g, int half, const double2* __restrict__ xin, double2* xout, int do_den) {
  constexpr int P = 4 * NT * WN;
  constexpr int LD = angular_ldx(P);
  constexpr int THREADS = AM_ROW_GROUPS * WN * 32;
  constexpr int AM_D = R * NT <= 2 ? 4 : 2;
  extern __shared__ __align__(16) double xs[];
  __shared__ double s_rE[P], s_v1[P], s_v2[P], s_v3[P], s_sb[P];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, q = lane & 3;      // fragment row group, thread in group
  const int wr = warp % AM_ROW_GROUPS, wn = warp / AM_ROW_GROUPS;
  const int n_l = g.n_l, n8 = (n_l + 7) / 8;
  const int tilesN = (g.n_r + P - 1) / P;
  const int col = blockIdx.x / tilesN;
  const int r0 = (blockIdx.x - col * tilesN) * P;
  const int m = g.col_m[col];
  const Chain& ch = g.chain[half];

  // S^T fragments of row tile rt, k steps 2 kp and 2 kp + 1 (rows l < m are zero, as the reference's
  // couplings start at l = m)
  double2 fa[AM_D][R];
  const double2* Sm = reinterpret_cast<const double2*>(g.frag) + (size_t)m * n8 * n8 * 32 + lane;
  const size_t mat_stride = (size_t)g.n_m * n8 * n8 * 32;
  auto load_a = [&](const double2* S, int kp, double2 (&dst)[R]) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int rt = wr + AM_ROW_GROUPS * i;
      if (rt < n8 && kp < n8) dst[i] = __ldg(S + ((size_t)rt * n8 + kp) * 32);
    }
  };
  if (ch.n_ops > 0)
#pragma unroll
    for (int d = 0; d < AM_D; ++d) load_a(Sm + ch.ops[0].mat * mat_stride, d, fa[d]);

  const RunDev run = g.runs[g.col_run[col]];
  int step = *g.step;
  if (step >= run.n_t) step = run.n_t - 1;  // overflow is flagged by k_finalize
  // the tile's orbitals (zero beyond N_l and beyond N_r)
  for (int i = tid; i < 8 * n8 * P; i += THREADS) {
    const int l = i / P, p = i - l * P, r = r0 + p;
    const double2 v = (l < n_l && r < g.n_r) ? xin[((size_t)l * g.n_cols + col) * g.n_r + r] : make_double2(0.0, 0.0);
    *reinterpret_cast<double2*>(xs + (size_t)l * LD + 2 * p) = v;
  }
  // per-radius potentials
  if (tid < P) {
    const int r = r0 + tid;
    const bool rv = r < g.n_r;
    const int rc = rv ? r : 0;
    const double rr = rv ? g.r[r] : 1.0;
    double v1 = 0.0, v2 = 0.0, v3 = 0.0, sbase = 0.0;
    if (g.hartree_on) {
      v1 = run.v[1 * g.n_r + rc];
      v2 = run.v[2 * g.n_r + rc];
      v3 = run.v[3 * g.n_r + rc];
      // couplingS.cuh:20-21, evaluated left to right
      sbase = run.v[rc] - run.v0[rc] + run.vexc[rc] - run.vexc0[rc];
    }
    s_rE[tid] = rr * run.E[step];
    s_v1[tid] = v1;
    s_v2[tid] = v2;
    s_v3[tid] = v3;
    s_sb[tid] = sbase;
  }
  const double hdt = 0.5 * g.dt;
  const double* pco = g.coef + ((size_t)CF_P * g.n_m + m) * n_l;
  __syncthreads();

  if (ch.pre_s) {
    for (int i = tid; i < n_l * P; i += THREADS) {
      const int l = i / P, p = i - l * P;
      double eta = s_sb[p] + pco[l] * s_v2[p];
      eta *= hdt;
      double2* x = reinterpret_cast<double2*>(xs + (size_t)l * LD + 2 * p);
      *x = cmul_conj_phase(*x, eta);
    }
    __syncthreads();
  }

  for (int o = 0; o < ch.n_ops; ++o) {
    const ChainOp op = ch.ops[o];
    const double2* S = Sm + op.mat * mat_stride;
    const bool last = (o == ch.n_ops - 1);
    double acc[R][NT][2];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) acc[i][nt][0] = acc[i][nt][1] = 0.0;
    const double* xb = xs + (size_t)q * LD + wn * NT * 8 + gid;
    for (int kp0 = 0; kp0 < n8; kp0 += AM_D) {
#pragma unroll
      for (int d = 0; d < AM_D; ++d) {
        if (kp0 + d < n8 && wr < n8) {
          const double* xr = xb + (size_t)(kp0 + d) * 8 * LD;
          double fb[2][NT];
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) fb[e][nt] = xr[e * 4 * LD + nt * 8];
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int i = 0; i < R; ++i)
              if (i == 0 || wr + AM_ROW_GROUPS * i < n8)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                  mma_f64_8x8x4(acc[i][nt][0], acc[i][nt][1], e ? fa[d][i].y : fa[d][i].x, fb[e][nt]);
          load_a(S, kp0 + d + AM_D, fa[d]);
        }
      }
    }
    if (!last)   // the next product's first fragments, under the phase pass
#pragma unroll
      for (int d = 0; d < AM_D; ++d) load_a(Sm + ch.ops[o + 1].mat * mat_stride, d, fa[d]);
    // thread (gid, q) holds channel 8 rt + gid of radius 4 (wn NT + nt) + q: real and imaginary part
    const bool direct = last && !ch.post_s;
    const bool keep = !direct || do_den;
    if (keep) __syncthreads();          // every warp has read the tile
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int j = 8 * (wr + AM_ROW_GROUPS * i) + gid;
      if (j >= n_l) continue;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int p = 4 * (wn * NT + nt) + q;
        const double2 y = make_double2(acc[i][nt][0], acc[i][nt][1]);
        if (keep) *reinterpret_cast<double2*>(xs + (size_t)j * LD + 2 * p) = y;
        if (direct && xout && r0 + p < g.n_r) xout[((size_t)j * g.n_cols + col) * g.n_r + r0 + p] = y;
      }
    }
    if (keep) __syncthreads();
    if (direct) break;
    // phases (couplingP.cuh:61-106 and twins); the last product's is the S phase
    const double* Dv = g.dph + ((size_t)op.coupling * g.n_m + m) * g.ldS;
    for (int i = tid; i < n_l * P; i += THREADS) {
      const int j = i / P, p = i - j * P;
      double2* x = reinterpret_cast<double2*>(xs + (size_t)j * LD + 2 * p);
      double2 y = *x;
      if (op.phase == PH_THETA && j >= m) {
        // the theta form: the whole angular potential at node x_j
        const double dj = Dv[j];
        double eta = (s_rE[p] + s_v1[p]) * dj + s_v2[p] * legendre_p2(dj) + s_v3[p] * legendre_p3(dj) + s_sb[p];
        // n_har > 4: the multipoles L >= 1 at this node come from the exact-quadrature table
        if (g.theta_tab && r0 + p < g.n_r) eta += run.htab[((size_t)m * n_l + j) * g.n_r + r0 + p];
        eta *= hdt;
        y = cmul_conj_phase(y, eta);
      } else if (op.phase != PH_NONE && j >= m) {
        double eta;
        if (op.phase == PH_P) eta = g.p_hartree ? (s_rE[p] + s_v1[p]) : s_rE[p];
        else if (op.phase == PH_D) eta = s_v2[p];
        else eta = s_v3[p];   // FP and FF
        eta *= hdt * Dv[j];
        y = cmul_conj_phase(y, eta);
      }
      if (last) {
        double eta = s_sb[p] + pco[j] * s_v2[p];
        eta *= hdt;
        y = cmul_conj_phase(y, eta);
        if (xout && r0 + p < g.n_r) xout[((size_t)j * g.n_cols + col) * g.n_r + r0 + p] = y;
      }
      *x = y;
    }
    __syncthreads();
  }

  if (do_den) {
    // density multipoles: lane groups of P threads, one radius per thread, a range of l per group,
    // then the groups summed in order (the tile's memory holds the groups' partials)
    const double2* x2 = reinterpret_cast<const double2*>(xs);
    const int n_den = g.n_den > 0 ? g.n_den : 1;  // L = 0 is always needed for the norm
    const int n_sub = g.den_groups > 0 ? g.den_groups : angular_den_groups(THREADS, P);
    const int sub = tid / P, p = tid - sub * P;
    double d[N_DEN] = {0.0, 0.0, 0.0, 0.0};
    if (sub < n_sub) {
      if (g.den_groups > 0 || n_l < m + 7) {
        // the literal l loops strided over the groups
        density_partials<double2, LD / 2>(n_den, m, n_l, x2, p, g.coef + (size_t)m * n_l, sub, n_sub, d, g.n_m * n_l);
      } else {
        const int per = (n_l - m + n_sub - 1) / n_sub, l0 = m + sub * per;
        density_window<LD / 2>(n_den, n_l, x2 + p, g.coef + (size_t)m * n_l, (size_t)g.n_m * n_l, l0, min(n_l, l0 + per), d);
      }
    }
    __syncthreads();
    if (sub < n_sub)
#pragma unroll
      for (int L = 0; L < N_DEN; ++L) xs[(sub * N_DEN + L) * P + p] = d[L];
    __syncthreads();
    for (int i = tid; i < n_den * P; i += THREADS) {
      const int L = i / P, pp = i - L * P, rl = r0 + pp;
      double sum = 0.0;
      for (int w = 0; w < n_sub; ++w) sum += xs[(w * N_DEN + L) * P + pp];
      if (rl < g.n_r) g.dens[((size_t)col * N_DEN + L) * g.n_r + rl] = sum;
    }
  }
}

// The same half-step for groups of many tiles: blocks of four warps on 16 radii, so that several share an SM
// and one's products run under another's phases and waits (with eight row groups a block's sixteen warps wait
// for one another three times per product, and one or two blocks fill an SM).  The tile is held twice, a
// product reads one copy and writes the other: one barrier per product.  A warp takes pairs of 8-channel
// tiles one after the other over all 32 columns, its S fragments AS_KU pairs of k steps ahead, and the
// phases are applied to its accumulators.  Bound by the FP64 pipe, which the products share with the phases'
// sines: 575 radii, N_l 70, 120 columns, five products 450 us, 15 TFLOP/s of products alone.
constexpr int AS_WARPS = 4, AS_P = 16, AS_LD = 2 * AS_P + 8, AS_NT = 2 * AS_P / 8, AS_KU = 2;
__global__ void __launch_bounds__(AS_WARPS * 32)
k_angular_fp64_small(GroupArgs g, int half, const double2* __restrict__ xin, double2* xout, int do_den) {
  extern __shared__ __align__(16) double smd[];
  __shared__ double s_rE[AS_P], s_v1[AS_P], s_v2[AS_P], s_v3[AS_P], s_sb[AS_P];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, q = lane & 3;
  const int n_l = g.n_l, n8 = (n_l + 7) / 8;
  const int tilesN = (g.n_r + AS_P - 1) / AS_P;
  const int col = blockIdx.x / tilesN;
  const int r0 = (blockIdx.x - col * tilesN) * AS_P;
  const int m = g.col_m[col];
  const Chain& ch = g.chain[half];
  double* xs = smd;
  double* ys = smd + (size_t)8 * n8 * AS_LD;
  const RunDev run = g.runs[g.col_run[col]];
  int step = *g.step;
  if (step >= run.n_t) step = run.n_t - 1;  // overflow is flagged by k_finalize
  for (int i = tid; i < 8 * n8 * AS_P; i += AS_WARPS * 32) {
    const int l = i / AS_P, p = i - l * AS_P, r = r0 + p;
    const double2 v = (l < n_l && r < g.n_r) ? xin[((size_t)l * g.n_cols + col) * g.n_r + r] : make_double2(0.0, 0.0);
    *reinterpret_cast<double2*>(xs + (size_t)l * AS_LD + 2 * p) = v;
    if (l >= n_l) *reinterpret_cast<double2*>(ys + (size_t)l * AS_LD + 2 * p) = make_double2(0.0, 0.0);
  }
  if (tid < AS_P) {
    const int r = r0 + tid;
    const bool rv = r < g.n_r;
    const int rc = rv ? r : 0;
    const double rr = rv ? g.r[r] : 1.0;
    double v1 = 0.0, v2 = 0.0, v3 = 0.0, sbase = 0.0;
    if (g.hartree_on) {
      v1 = run.v[1 * g.n_r + rc];
      v2 = run.v[2 * g.n_r + rc];
      v3 = run.v[3 * g.n_r + rc];
      sbase = run.v[rc] - run.v0[rc] + run.vexc[rc] - run.vexc0[rc];
    }
    s_rE[tid] = rr * run.E[step];
    s_v1[tid] = v1;
    s_v2[tid] = v2;
    s_v3[tid] = v3;
    s_sb[tid] = sbase;
  }
  const double hdt = 0.5 * g.dt;
  const double* pco = g.coef + ((size_t)CF_P * g.n_m + m) * n_l;
  __syncthreads();
  if (ch.pre_s) {
    for (int i = tid; i < n_l * AS_P; i += AS_WARPS * 32) {
      const int l = i / AS_P, p = i - l * AS_P;
      double eta = s_sb[p] + pco[l] * s_v2[p];
      eta *= hdt;
      double2* x = reinterpret_cast<double2*>(xs + (size_t)l * AS_LD + 2 * p);
      *x = cmul_conj_phase(*x, eta);
    }
    __syncthreads();
  }
  const double2* Sm = reinterpret_cast<const double2*>(g.frag) + (size_t)m * n8 * n8 * 32 + lane;
  const size_t mat_stride = (size_t)g.n_m * n8 * n8 * 32;
  for (int o = 0; o < ch.n_ops; ++o) {
    const ChainOp op = ch.ops[o];
    const double2* S = Sm + op.mat * mat_stride;
    const bool last = (o == ch.n_ops - 1);
    const double* Dv = g.dph + ((size_t)op.coupling * g.n_m + m) * g.ldS;
    for (int pr = warp; 2 * pr < n8; pr += AS_WARPS) {
      double acc[2][AS_NT][2];
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int nt = 0; nt < AS_NT; ++nt) acc[t][nt][0] = acc[t][nt][1] = 0.0;
      double2 fa[AS_KU][2], fn[AS_KU][2];
      auto load_a = [&](int kp0, double2 (&dst)[AS_KU][2]) {
#pragma unroll
        for (int u = 0; u < AS_KU; ++u)
#pragma unroll
          for (int t = 0; t < 2; ++t)
            dst[u][t] = kp0 + u < n8 && 2 * pr + t < n8 ? __ldg(S + ((size_t)(2 * pr + t) * n8 + kp0 + u) * 32) : make_double2(0.0, 0.0);
      };
      load_a(0, fa);
      for (int kp0 = 0; kp0 < n8; kp0 += AS_KU) {
        load_a(kp0 + AS_KU, fn);
#pragma unroll
        for (int u = 0; u < AS_KU; ++u) {
          if (kp0 + u < n8) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const double* xr = xs + (size_t)((kp0 + u) * 8 + 4 * e + q) * AS_LD + gid;
              double fb[AS_NT];
#pragma unroll
              for (int nt = 0; nt < AS_NT; ++nt) fb[nt] = xr[nt * 8];
#pragma unroll
              for (int nt = 0; nt < AS_NT; ++nt) {
                mma_f64_8x8x4(acc[0][nt][0], acc[0][nt][1], e ? fa[u][0].y : fa[u][0].x, fb[nt]);
                mma_f64_8x8x4(acc[1][nt][0], acc[1][nt][1], e ? fa[u][1].y : fa[u][1].x, fb[nt]);
              }
            }
          }
        }
#pragma unroll
        for (int u = 0; u < AS_KU; ++u) { fa[u][0] = fn[u][0]; fa[u][1] = fn[u][1]; }
      }
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int j = pr * 16 + 8 * t + gid;
        if (j >= n_l) continue;
        const double dj = Dv[j];
#pragma unroll
        for (int nt = 0; nt < AS_NT; ++nt) {
          const int p = 4 * nt + q;
          double2 y = make_double2(acc[t][nt][0], acc[t][nt][1]);
          // the phases of the kernel above
          if (op.phase == PH_THETA && j >= m) {
            double eta = (s_rE[p] + s_v1[p]) * dj + s_v2[p] * legendre_p2(dj) + s_v3[p] * legendre_p3(dj) + s_sb[p];
            if (g.theta_tab && r0 + p < g.n_r) eta += run.htab[((size_t)m * n_l + j) * g.n_r + r0 + p];
            eta *= hdt;
            y = cmul_conj_phase(y, eta);
          } else if (op.phase != PH_NONE && j >= m) {
            double eta;
            if (op.phase == PH_P) eta = g.p_hartree ? (s_rE[p] + s_v1[p]) : s_rE[p];
            else if (op.phase == PH_D) eta = s_v2[p];
            else eta = s_v3[p];   // FP and FF
            eta *= hdt * dj;
            y = cmul_conj_phase(y, eta);
          }
          if (last && ch.post_s) {
            double eta = s_sb[p] + pco[j] * s_v2[p];
            eta *= hdt;
            y = cmul_conj_phase(y, eta);
          }
          *reinterpret_cast<double2*>(ys + (size_t)j * AS_LD + 2 * p) = y;
        }
      }
    }
    __syncthreads();
    double* t = xs; xs = ys; ys = t;
  }
  const double2* x2 = reinterpret_cast<const double2*>(xs);
  if (xout)
    for (int i = tid; i < n_l * AS_P; i += AS_WARPS * 32) {
      const int l = i / AS_P, p = i - l * AS_P, r = r0 + p;
      if (r < g.n_r) xout[((size_t)l * g.n_cols + col) * g.n_r + r] = x2[(size_t)l * (AS_LD / 2) + p];
    }
  if (do_den) {
    // density multipoles as above, the groups' partials in the free copy of the tile
    const int n_den = g.n_den > 0 ? g.n_den : 1;
    const int n_sub = g.den_groups > 0 ? g.den_groups : AS_WARPS * 32 / AS_P;
    const int sub = tid / AS_P, p = tid - sub * AS_P;
    double d[N_DEN] = {0.0, 0.0, 0.0, 0.0};
    if (sub < n_sub) {
      if (g.den_groups > 0 || n_l < m + 7) {
        density_partials<double2, AS_LD / 2>(n_den, m, n_l, x2, p, g.coef + (size_t)m * n_l, sub, n_sub, d, g.n_m * n_l);
      } else {
        const int per = (n_l - m + n_sub - 1) / n_sub, l0 = m + sub * per;
        density_window<AS_LD / 2>(n_den, n_l, x2 + p, g.coef + (size_t)m * n_l, (size_t)g.n_m * n_l, l0, min(n_l, l0 + per), d);
      }
#pragma unroll
      for (int L = 0; L < N_DEN; ++L) ys[(sub * N_DEN + L) * AS_P + p] = d[L];
    }
    __syncthreads();
    for (int i = tid; i < n_den * AS_P; i += AS_WARPS * 32) {
      const int L = i / AS_P, pp = i - L * AS_P, rl = r0 + pp;
      double sum = 0.0;
      for (int w = 0; w < n_sub; ++w) sum += ys[(w * N_DEN + L) * AS_P + pp];
      if (rl < g.n_r) g.dens[((size_t)col * N_DEN + L) * g.n_r + rl] = sum;
    }
  }
}

static int g_angular_sms = 0;
static constexpr int ANGULAR_POINTS[] = {4, 8, 16, 24, 32, 40};

static int angular_warps_n(int points) { return points == 4 ? 1 : 2; }
static size_t angular_smem_points(int n_l, int points) {
  const int threads = AM_ROW_GROUPS * angular_warps_n(points) * 32;
  return std::max((size_t)angular_rows(n_l) * angular_ldx(points),
                  (size_t)angular_den_groups(threads, points) * N_DEN * points) * sizeof(double);
}
// accumulators of a warp's row tiles and column tiles, in registers (512 threads: 128 each)
static bool angular_points_ok(int n_l, int points) {
  const int r = ((n_l + 7) / 8 + AM_ROW_GROUPS - 1) / AM_ROW_GROUPS;
  return r <= 2 || (r == 3 && points <= 32) || points <= 24;
}
size_t angular_smem_fp64(int n_l) {
  size_t most = 0;
  for (int p : ANGULAR_POINTS)
    if (angular_points_ok(n_l, p)) most = std::max(most, angular_smem_points(n_l, p));
  return most;
}

static size_t angular_small_smem(int n_l) { return 2 * (size_t)angular_rows(n_l) * AS_LD * sizeof(double); }

// Radii per block: the least rounds over the SMs x (radii + the time of a block that does not depend
// on them, about that of 12 radii).  0: the four-warp blocks, by the same measure: four of them share an SM
// (three above 88 channels), and a round of 148 x 4 takes as long as 62 of those units (80 below 30
// channels).  They are the faster ones from about 2.5 tiles of 16 radii per SM on, where the last round is
// not nearly empty; eight-warp form -> this one, both halves: the five products of the coupling chain at
// N_r 253, N_l 49, 24 columns 97 -> 76 us, 575/70/120 1332 -> 927, 425/35/18 87 -> 64; the theta form at
// 225/30/78 62 -> 46.  Few tiles: 253/49/3 28 against 54 us, 600/97/9 66 against 82.  From 105 channels on
// two blocks fit an SM or fewer and the eight-warp form is the better one (300/220/9 128 against 278 us), at
// 9 channels too (the blocks are all set-up).
static int angular_points(const GroupArgs& g) {
  int best = 4;
  long best_cost = -1;
  for (int p : ANGULAR_POINTS) {
    if (!angular_points_ok(g.n_l, p)) continue;
    const long tiles = (long)g.n_cols * ((g.n_r + p - 1) / p);
    const long cost = (tiles + g_angular_sms - 1) / g_angular_sms * (p + 12);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = p;
    }
  }
  if (g.n_l >= 17 && g.n_l <= 104) {
    const long tiles = (long)g.n_cols * ((g.n_r + AS_P - 1) / AS_P), resident = (long)g_angular_sms * (g.n_l <= 88 ? 4 : 3);
    if ((tiles + resident - 1) / resident * (g.n_l < 30 ? 80 : 62) < best_cost) return 0;
  }
  return best;
}

// The kernel that a group's half-steps run on.
struct AngularLaunch {
  void (*fn)(GroupArgs, int, const double2*, double2*, int);
  int points, threads;
  size_t smem;
};
template <int NT, int WN, int R>
static AngularLaunch angular_tile(int n_l) {
  constexpr int P = 4 * NT * WN;
  return {k_angular_fp64<NT, WN, R>, P, AM_ROW_GROUPS * WN * 32, angular_smem_points(n_l, P)};
}
template <int R>
static AngularLaunch angular_launch_rows(int n_l, int points) {
  switch (points) {
    case 4: return angular_tile<1, 1, R>(n_l);
    case 8: return angular_tile<1, 2, R>(n_l);
    case 16: return angular_tile<2, 2, R>(n_l);
    case 32: if constexpr (R <= 3) return angular_tile<4, 2, R>(n_l); break;
    case 40: if constexpr (R <= 2) return angular_tile<5, 2, R>(n_l); break;
    default: break;
  }
  return angular_tile<3, 2, R>(n_l);
}
static AngularLaunch angular_launch(const GroupArgs& g) {
  const int points = angular_points(g);
  if (points == 0) return {k_angular_fp64_small, AS_P, AS_WARPS * 32, angular_small_smem(g.n_l)};
  switch (((g.n_l + 7) / 8 + AM_ROW_GROUPS - 1) / AM_ROW_GROUPS) {
    case 1: return angular_launch_rows<1>(g.n_l, points);
    case 2: return angular_launch_rows<2>(g.n_l, points);
    case 3: return angular_launch_rows<3>(g.n_l, points);
    default: return angular_launch_rows<4>(g.n_l, points);
  }
}

void launch_angular_fp64(const GroupArgs& g, int half, const double2* xin, double2* xout, int do_den, cudaStream_t s) {
  const AngularLaunch k = angular_launch(g);
  k.fn<<<g.n_cols * ((g.n_r + k.points - 1) / k.points), k.threads, k.smem, s>>>(g, half, xin, xout, do_den);
}

// ---------------------------------------------------------------------------------------------
// radial propagator, FP64
// ---------------------------------------------------------------------------------------------

constexpr int RAD_CW = 4;                 // consumer warps: one output radius per thread
constexpr int RAD_TI = 32 * RAD_CW;       // rows (output radii) per tile
constexpr int RAD_KC = 16;                // k per stage (3 stages of ~35 KB: two CTAs per SM)
constexpr int RAD_STAGES = 3;
constexpr int RAD_THREADS = 32 * (RAD_CW + 1);

// Tiles (l, radius tile, column tile), the column tile fastest so that CTAs running side by side
// read the same W rows (one HBM read, the others from L2).
template <int TC>
__global__ void __launch_bounds__(RAD_THREADS, 2)
k_radial_fp64(int n_r, int n_cols, int n_l, const double2* __restrict__ W, const double2* __restrict__ xin,
              double2* __restrict__ xout, unsigned* status) {
  constexpr int W_STAGE = RAD_KC * RAD_TI;        // double2 per stage: [k][row]
  constexpr int X_STAGE = TC * RAD_KC;            // [col][k]
  extern __shared__ __align__(128) double2 rsm[];
  __shared__ uint64_t full_bar[RAD_STAGES], empty_bar[RAD_STAGES];
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_it = (n_r + RAD_TI - 1) / RAD_TI, n_ct = (n_cols + TC - 1) / TC;
  const int total = n_it * n_ct * n_l;
  const int n_kc = (n_r + RAD_KC - 1) / RAD_KC;
  if (threadIdx.x == 0) {
    for (int s = 0; s < RAD_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], RAD_CW);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  volatile int* abort_p = &abort_flag;
  if (warp == RAD_CW) {
    // producer: one thread issues the bulk copies of every stage
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
        const int ct = tile % n_ct, rest = tile / n_ct, itile = rest % n_it, l = rest / n_it;
        const int i0 = itile * RAD_TI, rows = min(RAD_TI, n_r - i0);
        const int c0 = ct * TC, nc = min(TC, n_cols - c0);
        const double2* Wl = W + (size_t)l * n_r * n_r;
        const double2* Xl = xin + (size_t)l * n_cols * n_r;
        for (int kc = 0; kc < n_kc; ++kc, ++it) {
          const int s = it % RAD_STAGES;
          if (it >= RAD_STAGES && !mbar_wait(&empty_bar[s], ((it / RAD_STAGES) & 1) ^ 1, abort_p)) {
            ok = false;
            break;
          }
          const int k0 = kc * RAD_KC, kn = min(RAD_KC, n_r - k0);
          double2* ws = rsm + (size_t)s * (W_STAGE + X_STAGE);
          double2* xs = ws + W_STAGE;
          mbar_expect_tx(&full_bar[s], (uint32_t)(kn * rows + nc * kn) * 16u);
          for (int kk = 0; kk < kn; ++kk)
            bulk_g2s(ws + kk * RAD_TI, Wl + (size_t)(k0 + kk) * n_r + i0, (uint32_t)rows * 16u, &full_bar[s]);
          for (int c = 0; c < nc; ++c)
            bulk_g2s(xs + c * RAD_KC, Xl + (size_t)(c0 + c) * n_r + k0, (uint32_t)kn * 16u, &full_bar[s]);
        }
      }
      if (!ok) {
        // let the copies already issued land before the CTA exits
        for (int q = (it > RAD_STAGES ? it - RAD_STAGES : 0); q < it; ++q)
          mbar_drain(&full_bar[q % RAD_STAGES], (q / RAD_STAGES) & 1);
      }
    }
  } else {
    // consumers on the FP64 tensor cores: warp w computes output radii i0 + 32 w .. + 31 (four 8-row
    // MMA tiles) for the tile's TC columns.  Real form of the complex product, columns interleaved
    // (2 c + 0/1 = real/imaginary part of column c):  [Yr Yi] = Wr B + Wi B'  with B = [Xr Xi] and
    // B' = [-Xi Xr] per column, so that a thread's two accumulators of an 8-column tile are one
    // complex output.  A (i, k) = W[l][k][i] from the W rows in shared memory (one 16-byte load
    // gives the Wr and Wi fragments), B and B' from one 16-byte load of x.  k beyond the row (the
    // last chunk) contributes zero on both sides.
    constexpr int NT = (2 * TC + 7) / 8;            // 8-column MMA tiles
    const int g8 = lane >> 2, q = lane & 3;
    int it = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const int ct = tile % n_ct, rest = tile / n_ct, itile = rest % n_it, l = rest / n_it;
      const int i0 = itile * RAD_TI;
      const int c0 = ct * TC, nc = min(TC, n_cols - c0);
      // separate accumulators for the Wr and Wi products (up to 24 columns; beyond, the registers
      // would spill): the 2 x 4 x NT MMAs of a k step are independent, where one accumulator chain
      // makes every second MMA wait for the first
      constexpr bool SPLIT = NT <= 3;
      double acc[4][NT][2], acd[4][NT][2];
      auto& adst = SPLIT ? acd : acc;
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = acd[mt][nt][0] = acd[mt][nt][1] = 0.0;
      bool ok = true;
      for (int kc = 0; kc < n_kc; ++kc, ++it) {
        const int s = it % RAD_STAGES;
        if (!mbar_wait(&full_bar[s], (it / RAD_STAGES) & 1, abort_p)) {
          ok = false;
          break;
        }
        const int kn = min(RAD_KC, n_r - kc * RAD_KC);
        const double2* ws = rsm + (size_t)s * (W_STAGE + X_STAGE);
        const double2* xs = ws + W_STAGE;
#pragma unroll
        for (int ks = 0; ks < RAD_KC / 4; ++ks) {
          const int kk = 4 * ks + q;
          const bool kv = kk < kn;
          double ar[4], ai[4], bp[NT], bq[NT];
#pragma unroll
          for (int mt = 0; mt < 4; ++mt) {
            const double2 w = kv ? ws[kk * RAD_TI + 32 * warp + 8 * mt + g8] : make_double2(0.0, 0.0);
            ar[mt] = w.x;
            ai[mt] = w.y;
          }
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const int c = 4 * nt + (g8 >> 1);
            const double2 x = (kv && c < TC) ? xs[c * RAD_KC + kk] : make_double2(0.0, 0.0);
            bp[nt] = (g8 & 1) ? x.y : x.x;
            bq[nt] = (g8 & 1) ? x.x : -x.y;
          }
#pragma unroll
          for (int mt = 0; mt < 4; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              mma_f64_8x8x4(acc[mt][nt][0], acc[mt][nt][1], ar[mt], bp[nt]);
              mma_f64_8x8x4(adst[mt][nt][0], adst[mt][nt][1], ai[mt], bq[nt]);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);
      }
      if (!ok) break;
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        const int i = i0 + 32 * warp + 8 * mt + g8;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const int c = 4 * nt + q;
          if (i < n_r && c < nc)
            xout[((size_t)l * n_cols + c0 + c) * n_r + i] =
                make_double2(acc[mt][nt][0] + acd[mt][nt][0], acc[mt][nt][1] + acd[mt][nt][1]);
        }
      }
    }
  }
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicOr(status, ST_TC_TIMEOUT);
}

template <int TC>
static constexpr size_t radial_fp64_smem() {
  return (size_t)RAD_STAGES * (RAD_KC * RAD_TI + TC * RAD_KC) * sizeof(double2);
}

// Few orbital columns (up to RF_MAX_COLS): one block per (l, 32 output radii), k split over the block's
// warps.  A warp streams its k slice of W straight into registers (per k step of 4: four loads, each
// 4 k x 8 radii = four 128-byte segments, RF_D steps ahead of the products), the x values of RF_KC k at
// a time come by cp.async into a double buffer of its own, so that no warp waits for another before
// the slices' sums are added, in slice order, at the end.  Groups of four columns run on the FP64
// tensor pipe as in the tile form above; the columns left over (one of nine) as plain FMAs on the same
// fragments, each lane over its own k: an 8-column MMA tile would pad nine columns (18 real) to 24,
// and the two units share one peak.  The many small blocks keep every SM supplied to the end, where
// tiles of 128 radii leave the last wave a third full (485 tiles on 296 resident blocks).
// Bound by HBM (W, 16 N_r^2 N_l bytes) and, at nine columns, as much by the FP64 pipe.  Tile form ->
// this form: N_r 200, N_l 33, one column 16.9 -> 8.5 us; 400/65/1 35.5 -> 29.0 us (5.7 TB/s of W);
// 253/49/3 22.8 -> 11.5 us; 600/97/9 164 -> 131 us (4.3 TB/s of W, 19 TFLOP/s).
constexpr int RF_MAX_COLS = 9;
constexpr int RF_KC = 16;                 // k per x chunk
constexpr int RF_LDX = RF_KC + 4;         // row of a chunk: four columns' four k fall on 256 different bytes

__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}

// The first RF_KEEP bytes of W stay in L2 from step to step (normal priority), the rest streams
// through it (evict first), so that W does not push itself out of L2 before it comes round again.
// The helium step (166 MB of W) takes 70.2 us with none kept, 66.7 with 48 MB, 74.6 with 96 MB; one argon
// run's (559 MB) 212.9, 205.8 and 219.3.
constexpr size_t RF_KEEP = 48u << 20;

template <int TC, int RF_WARPS, bool KEEP>
__device__ __forceinline__ void radial_rows_block(int n_r, const double2* __restrict__ W,
                                                  const double2* __restrict__ xin, double2* __restrict__ xout,
                                                  double2* sm) {
  // MMA tiles of four columns and FMA columns (three left over: one padded tile, for its registers)
  constexpr int NT = (TC + 1) / 4, NF = TC > 4 * NT ? TC - 4 * NT : 0;
  // k steps of W in flight: four where the registers allow it (three columns: 14.5 -> 11.5 us)
  constexpr int RF_D = TC == 3 || TC == 4 ? 4 : 2;
  constexpr int XC = 4 * NT > TC ? 4 * NT : TC;     // columns of the x buffers (a padded tile's last: unused)
  constexpr int XW = 2 * XC * RF_LDX;               // x buffers of a warp
  constexpr int PL = TC | 1, PW = PL * 32;          // partial sums of a warp, [32 radii][PL]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, q = lane & 3;
  const int n_it = (n_r + 31) / 32;
  const int l = blockIdx.x / n_it, i0 = (blockIdx.x - l * n_it) * 32;
  const int ks = (n_r + 4 * RF_WARPS - 1) / (4 * RF_WARPS) * 4;
  const int k0 = min(n_r, warp * ks), k1 = min(n_r, k0 + ks);
  double2* xs = sm + warp * XW;
  const double2* Xl = xin + (size_t)l * TC * n_r;
  auto load_x = [&](int kc, int buf) {
    for (int e = lane; e < TC * RF_KC; e += 32) {
      const int c = e / RF_KC, kk = e - c * RF_KC, k = kc + kk;
      const bool v = k < k1;
      cp_async16_zfill(xs + buf * XC * RF_LDX + c * RF_LDX + kk, Xl + (size_t)c * n_r + (v ? k : 0), v);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // W[l][k + q][i0 + 8 mt + gid] of the next k step, zero past the slice and past the last radius
  const double2* wp = W + ((size_t)l * n_r + k0 + q) * n_r + i0 + gid;
  const size_t wstep = 4 * (size_t)n_r;
  int kw = k0 + q;
  const int rows_left = n_r - i0 - gid;
  auto load_w = [&](double2 (&w)[4]) {
    const bool kv = kw < k1;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      w[mt] = make_double2(0.0, 0.0);
      if (kv && 8 * mt < rows_left) w[mt] = KEEP ? __ldg(wp + 8 * mt) : __ldcs(wp + 8 * mt);
    }
    wp += wstep;
    kw += 4;
  };
  double acc[4][NT > 0 ? NT : 1][2];
  double2 accf[4][NF > 0 ? NF : 1];
#pragma unroll
  for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;
#pragma unroll
    for (int f = 0; f < NF; ++f) accf[mt][f] = make_double2(0.0, 0.0);
  }
  double2 w[RF_D][4];
#pragma unroll
  for (int d = 0; d < RF_D; ++d) load_w(w[d]);
  load_x(k0, 0);
  int buf = 0;
#pragma unroll 1
  for (int kc = k0; kc < k1; kc += RF_KC, buf ^= 1) {
    load_x(kc + RF_KC, buf ^ 1);          // past the slice: zeros, never read
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const double2* xb = xs + buf * XC * RF_LDX + q;
#pragma unroll
    for (int st = 0; st < RF_KC / 4; ++st) {
      double2 (&ww)[4] = w[st % RF_D];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int c = 4 * nt + (gid >> 1);
        const double2 x = (4 * NT <= TC || c < TC) ? xb[c * RF_LDX + 4 * st] : make_double2(0.0, 0.0);
        const double bp = (gid & 1) ? x.y : x.x, bq = (gid & 1) ? x.x : -x.y;
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) mma_f64_8x8x4(acc[mt][nt][0], acc[mt][nt][1], ww[mt].x, bp);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) mma_f64_8x8x4(acc[mt][nt][0], acc[mt][nt][1], ww[mt].y, bq);
      }
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const double2 x = xb[(4 * NT + f) * RF_LDX + 4 * st];
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
          accf[mt][f].x = fma(ww[mt].x, x.x, accf[mt][f].x);
          accf[mt][f].y = fma(ww[mt].x, x.y, accf[mt][f].y);
          accf[mt][f].x = fma(-ww[mt].y, x.y, accf[mt][f].x);
          accf[mt][f].y = fma(ww[mt].y, x.x, accf[mt][f].y);
        }
      }
      load_w(ww);
    }
    __syncwarp();                         // the buffer is refilled in the next round
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                        // every warp is done with its x buffers
  double2* part = sm + warp * PW;
#pragma unroll
  for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      if (4 * NT <= TC || 4 * nt + q < TC) part[(8 * mt + gid) * PL + 4 * nt + q] = make_double2(acc[mt][nt][0], acc[mt][nt][1]);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      double2 v = accf[mt][f];
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if (q == mt) part[(8 * mt + gid) * PL + 4 * NT + f] = v;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < TC * 32; e += RF_WARPS * 32) {
    const int c = e >> 5, rl = e & 31, r = i0 + rl;
    double2 s = sm[rl * PL + c];
#pragma unroll
    for (int p = 1; p < RF_WARPS; ++p) {
      const double2 v = sm[p * PW + rl * PL + c];
      s.x += v.x;
      s.y += v.y;
    }
    if (r < n_r) xout[((size_t)l * TC + c) * n_r + r] = s;
  }
}

template <int TC>
constexpr int rf_smem(int warps) {    // double2: x buffers or partial sums
  constexpr int xc = (TC + 1) / 4 * 4 > TC ? (TC + 1) / 4 * 4 : TC;
  return warps * (2 * xc * RF_LDX > (TC | 1) * 32 ? 2 * xc * RF_LDX : (TC | 1) * 32);
}

template <int TC, int RF_WARPS>
__global__ void __launch_bounds__(RF_WARPS * 32, (TC == 1 ? 24 : 16) / RF_WARPS)
k_radial_fp64_rows(int n_r, int l_keep, const double2* __restrict__ W, const double2* __restrict__ xin,
                   double2* __restrict__ xout) {
  __shared__ __align__(16) double2 sm[rf_smem<TC>(RF_WARPS)];
  if ((int)blockIdx.x / ((n_r + 31) / 32) < l_keep) radial_rows_block<TC, RF_WARPS, true>(n_r, W, xin, xout, sm);
  else radial_rows_block<TC, RF_WARPS, false>(n_r, W, xin, xout, sm);
}

static int g_radial_sms = 0;

// The tile form also for one, two and six columns on large grids whose tiles of 128 radii fill their rounds
// over the resident CTAs: there it streams W at 5.5 - 7 TB/s, the row form at 4.6 - 6.3 (one column, many
// rounds of short blocks), 3.8 - 5.5 (two, plain FMAs) and 4.8 - 5.5 (six, padded to eight).  Row -> tile
// form, a step in the graph: N_r 2000, N_l 17, one column 267 -> 188 us; 1000/33/1 139 -> 107; 1000/97/2
// 352 -> 292; 1000/33/6 153 -> 142.  Below 640 radii (much of W or of a round in L2, latency) the row form's
// step is the faster one (250/145/1 14 %, 350/129/2 16 %), in part-empty rounds too (600/65/1 90 -> 73 us alone).
static bool radial_tiles(int n_cols, int n_r, int n_l) {
  if (n_cols > RF_MAX_COLS) return true;
  if (n_r < 640 || !(n_cols <= 2 || n_cols == 6)) return false;
  const long tiles = (long)((n_r + RAD_TI - 1) / RAD_TI) * n_l, resident = 2 * g_radial_sms;
  const double fill = n_cols == 2 ? 0.58 : 0.77;    // of the rounds, by rows of W
  return (double)n_r * n_l >= fill * RAD_TI * resident * ((tiles + resident - 1) / resident);
}

struct RadialTile {
  void (*fn)(int, int, int, const double2*, const double2*, double2*, unsigned*);
  int cols;
  size_t smem;
};
template <int TC>
static RadialTile radial_tile() { return {k_radial_fp64<TC>, TC, radial_fp64_smem<TC>()}; }
static RadialTile radial_tile_of(int n_cols) {
  return n_cols == 1 ? radial_tile<1>() : n_cols == 2 ? radial_tile<2>() : n_cols <= 6 ? radial_tile<6>()
       : n_cols <= 12 ? radial_tile<12>() : radial_tile<16>();
}

void launch_radial_fp64(const GroupArgs& g, const double2* W, const double2* xin, double2* xout, cudaStream_t s) {
  const int nc = g.n_cols;
  if (radial_tiles(nc, g.n_r, g.n_l)) {
    const RadialTile k = radial_tile_of(nc);
    const int tiles = ((g.n_r + RAD_TI - 1) / RAD_TI) * ((nc + k.cols - 1) / k.cols) * g.n_l;
    k.fn<<<std::min(tiles, 2 * g_radial_sms), RAD_THREADS, k.smem, s>>>(g.n_r, nc, g.n_l, W, xin, xout, g.status);
    return;
  }
  const int blocks = g.n_l * ((g.n_r + 31) / 32);
  const int l_keep = (int)(RF_KEEP / (sizeof(double2) * g.n_r * g.n_r));
  // eight warps a block until four blocks an SM are there, then four (fewer k slices to start and
  // to add: 138 -> 133 us at 600/97/9; below, the smaller blocks leave the SMs emptier)
  const bool wide = blocks < 4 * g_radial_sms;
#define GGB_RF_CASE(C)                                                                       \
  case C:                                                                                    \
    if (wide) k_radial_fp64_rows<C, 8><<<blocks, 256, 0, s>>>(g.n_r, l_keep, W, xin, xout);  \
    else k_radial_fp64_rows<C, 4><<<blocks, 128, 0, s>>>(g.n_r, l_keep, W, xin, xout);       \
    break;
  switch (nc) {
    GGB_RF_CASE(1) GGB_RF_CASE(2) GGB_RF_CASE(3) GGB_RF_CASE(4) GGB_RF_CASE(5)
    GGB_RF_CASE(6) GGB_RF_CASE(7) GGB_RF_CASE(8) GGB_RF_CASE(9)
    default: break;
  }
#undef GGB_RF_CASE
}

// ---------------------------------------------------------------------------------------------
// finalize: observables, Hartree multipoles (compensated scans), exchange, step counter
// ---------------------------------------------------------------------------------------------

constexpr int FIN_THREADS = 256;

// Compensated scans of two rows in shared memory, in place and side by side (one chain of latencies):
// F[a] <- sum_{b <= a} F[b] (inclusive), G[a] <- sum_{b > a} G[b] (suffix, exclusive).
__device__ void block_scans_dd(double* F, double* G, int n, dd (*wsum)[2]) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = FIN_THREADS / 32;
  const int per = (n + FIN_THREADS - 1) / FIN_THREADS;
  const int b0 = tid * per;
  // local inclusive sums in the scan direction
  dd loc[2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int q = 0; q < per; ++q) {
    const int k = b0 + q;
    if (k < n) {
      loc[0] = dd_add(loc[0], dd{F[k], 0.0});
      loc[1] = dd_add(loc[1], dd{G[n - 1 - k], 0.0});
    }
  }
  // warp inclusive scan of thread totals
  dd inc[2] = {loc[0], loc[1]};
#pragma unroll
  for (int d = 1; d < 32; d <<= 1)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const dd o = dd_shfl_up(inc[c], d);
      if (lane >= d) inc[c] = dd_add(o, inc[c]);
    }
  if (lane == 31) {
    wsum[warp][0] = inc[0];
    wsum[warp][1] = inc[1];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      dd w = lane < nw ? wsum[lane][c] : dd{0.0, 0.0};
#pragma unroll
      for (int d = 1; d < nw; d <<= 1) {
        const dd o = dd_shfl_up(w, d);
        if (lane >= d) w = dd_add(o, w);
      }
      if (lane < nw) wsum[lane][c] = w;
    }
  }
  __syncthreads();
  // exclusive prefix of this thread = inclusive value of the previous lane + earlier warps
  dd run[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const dd prev = dd_shfl_up(inc[c], 1);
    run[c] = lane == 0 ? dd{0.0, 0.0} : prev;
    if (warp > 0) run[c] = dd_add(wsum[warp - 1][c], run[c]);
  }
  for (int q = 0; q < per; ++q) {
    const int k = b0 + q;
    if (k < n) {
      run[0] = dd_add(run[0], dd{F[k], 0.0});
      F[k] = run[0].hi + run[0].lo;                 // inclusive (sum over b <= a)
      const double tv = G[n - 1 - k];
      G[n - 1 - k] = run[1].hi + run[1].lo;         // exclusive (sum over b > a)
      run[1] = dd_add(run[1], dd{tv, 0.0});
    }
  }
  __syncthreads();
}

__device__ __forceinline__ double ipow(double x, int L) {
  double p = 1.0;
  for (int i = 0; i < L; ++i) p *= x;
  return p;
}

// Dipole, acceleration and norm of orbital row (l, column col) by one warp, the lanes striding over
// the radii, in double-double: <x_l | r (c_u x_(l+1) + c_d x_(l-1))>, the same with r^-2, and |x_l|^2
// (dipoleMoment.cuh:19-43, dipoleAcceleration.cuh:17-41 and their cublasZdotc).  Every lane gets the sums.
__device__ __forceinline__ void observe_row(const GroupArgs& g, const double2* x, int col, int l, int lane, dd (&s)[5]) {
#pragma unroll
  for (int q = 0; q < 5; ++q) s[q] = dd{0.0, 0.0};
  const int n_l = g.n_l, n_r = g.n_r, m = g.col_m[col];
  if (l < m) return;
  // the first row has no lower, the last no upper neighbour
  const bool up = l + 1 < n_l, down = l > m;
  const double c_u = up ? g.coef[((size_t)CF_CU * g.n_m + m) * n_l + l] : 0.0;
  const double c_d = down ? g.coef[((size_t)CF_CD * g.n_m + m) * n_l + l] : 0.0;
  const size_t ls = (size_t)g.n_cols * n_r;
  const double2* row = x + (size_t)l * ls + (size_t)col * n_r;
#pragma unroll 4
  for (int i = lane; i < n_r; i += 32) {
    const double2 xl = row[i];
    const double2 xu = up ? row[ls + i] : make_double2(0.0, 0.0);
    const double2 xd = down ? (row - ls)[i] : make_double2(0.0, 0.0);
    const double rr = g.r[i], fr2 = 1.0 / (rr * rr);
    const double zx = c_u * xu.x + c_d * xd.x, zy = c_u * xu.y + c_d * xd.y;
    const double px = xl.x * zx + xl.y * zy, py = xl.x * zy - xl.y * zx;   // conj(x_l) . z
    sum2_add(s[0], rr * px);
    sum2_add(s[1], rr * py);
    sum2_add(s[2], fr2 * px);
    sum2_add(s[3], fr2 * py);
    sum2_add(s[4], xl.x * xl.x + xl.y * xl.y);
  }
#pragma unroll
  for (int q = 0; q < 5; ++q) sum2_warp(s[q]);
}

// exchange blocks per run: one radius per thread; without Hartree the density is the frozen one, and
// the potential stays what mode 0 wrote, until another grid is set (mode 3)
__host__ __device__ inline int fin_xc_blocks(const GroupArgs& g, int mode) {
  return (g.n_den > 0 || mode == 0 || mode == 3) ? (g.n_r + FIN_THREADS - 1) / FIN_THREADS : 0;
}

// Blocks: for each run of the group, n_den Hartree blocks (L = 0..n_den-1), the exchange blocks and
// g.fin_ob observables blocks.  mode 0 = initial potentials (no observables,
// no step increment), mode 1 = end of step, mode 2 = end of step without the step increment and the
// watchdog checks (the per-phase timing), mode 3 = the exchange potential alone (without Hartree).
//
// Observables: one warp per row (l, orbital) of the run.  ROWS (the FP64 angular kernel): from the
// orbitals, straight from L2 where those of a run still are (the angular kernel's tiles summed them
// before: a double-double warp reduction of every row for every 16 radii, 8 us of its second half for
// one column on 200 radii and 25 us for nine on 600).  Otherwise from the partial sums per tile of
// radii that the int8 and BF16 angular kernels leave (an eighth of the orbitals' bytes: the orbitals
// of an ensemble are not in L2), with one more row per orbital for the norm, from the density.  The
// rows' sums go to a scratch array, and the last of an orbital's rows to finish (a counter per orbital)
// adds them over l, writes the totals and runs the NaN / norm-growth watchdog.  (Blocks that took a slice of
// l with one warp per orbital walked its rows one after another: 27 us for nine orbitals, N_l 97, and
// 88 us for 21 such runs at N_l 161, now 10 and 48 us.)
// ROWS: the observables come from the orbitals x (the partial sums' kernel needs half its registers).
template <bool ROWS>
__global__ void __launch_bounds__(FIN_THREADS) k_finalize(GroupArgs g, const double2* x, int mode) {
  extern __shared__ double fsm[];  // [2][N_r]
  __shared__ dd wsum[FIN_THREADS / 32][2];
  const int n_xc = fin_xc_blocks(g, mode);
  const int nb = g.n_den + n_xc + g.fin_ob;
  const int ri = blockIdx.x / nb;
  const int role = blockIdx.x - ri * nb;  // Hartree L = role, then exchange, then observables blocks
  const int n_r = g.n_r, n_l = g.n_l, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const bool obs_block = role >= g.n_den + n_xc;
  const int ob = role - g.n_den - n_xc;
  const int step = *g.step;
  const RunDev run = g.runs[ri];
  // the step counter advances once every thread of every block has read it
  asm volatile("" ::"r"(step) : "memory");
  __syncthreads();
  if (mode == 1 && tid == 0) {
    __threadfence();
    if (atomicAdd(g.done, 1u) == gridDim.x - 1) {
      *g.done = 0u;
      *g.step = step + 1;
    }
  }

  if (obs_block && mode != 0 && step >= run.n_t) {
    if (mode == 1 && ob == 0 && tid == 0) atomicOr(g.status, ST_STEP_OVERFLOW);
  } else if (obs_block && mode != 3) {
    const int n_orb = run.n_orb;
    double2* scr = reinterpret_cast<double2*>(g.fin_scr);     // [col][N_l + 1][5]; row N_l: the norm
    const int rows = n_l * n_orb + (ROWS ? 0 : n_orb);
    auto sum_rows = [&](int k) {
      const int col = run.col0 + k;
      double2* o = scr + (size_t)col * (n_l + 1) * 5;
      dd s[5];
      int last = 0;
      if (lane == 0) last = atomicAdd(g.fin_cnt + col, 1u) == (unsigned)(n_l - (ROWS ? 1 : 0));
      if (__shfl_sync(0xffffffffu, last, 0)) {
        __threadfence();
        __syncwarp();                           // lane 0 counted; the shuffle alone orders no memory
#pragma unroll
        for (int q = 0; q < 5; ++q) s[q] = dd{0.0, 0.0};
        for (int lp = lane; lp < n_l + (ROWS ? 0 : 1); lp += 32)
#pragma unroll
          for (int q = 0; q < 5; ++q) {
            const double2 v = __ldcg(o + (size_t)lp * 5 + q);
            sum2_add(s[q], dd{v.x, v.y});
          }
#pragma unroll
        for (int q = 0; q < 5; ++q) sum2_warp(s[q]);
        // a sum that overflowed is a NaN in hi + lo only (hi stays infinite)
        const double nrm = s[4].hi + s[4].lo, dip = s[0].hi + s[0].lo, acc = s[2].hi + s[2].lo;
        if (lane == 0) {
          if (mode == 0) {
            run.norm0[k] = nrm;                 // for the growth watchdog
          } else {
            run.dip_tot[(size_t)k * run.n_t + step] = make_double2(dip, s[1].hi + s[1].lo);
            run.acc_tot[(size_t)k * run.n_t + step] = make_double2(acc, s[3].hi + s[3].lo);
            run.norm[(size_t)k * run.n_t + step] = nrm;
            if (mode == 1) {
              if (!(nrm == nrm) || isinf(nrm) || !(dip == dip) || !(acc == acc)) atomicOr(g.status, ST_NAN);
              if (nrm > run.norm0[k] * (1.0 + g.norm_tol) + 1e-300) atomicOr(g.status, ST_NORM_GROWTH);
            }
          }
          g.fin_cnt[col] = 0u;                  // for the next launch (stream-ordered after this one)
        }
      }
    };
    const int i0 = ob * (FIN_THREADS / 32) + warp, stride = g.fin_ob * (FIN_THREADS / 32);
    for (int i = i0; i < rows; i += stride) {
      const int l = i / n_orb, k = i - l * n_orb;
      dd s[5];
      if constexpr (ROWS) {
        observe_row(g, x, run.col0 + k, l, lane, s);
      } else {
#pragma unroll
        for (int q = 0; q < 5; ++q) s[q] = dd{0.0, 0.0};
        if (l == n_l) {
          const double* dn = g.dens + (size_t)(run.col0 + k) * N_DEN * n_r;  // L = 0 row
          for (int q = lane; q < n_r; q += 32) sum2_add(s[4], dn[q]);
          sum2_warp(s[4]);
        } else {
          const double4* p = g.obs + ((size_t)(run.col0 + k) * n_l + l) * g.n_tiles * g.obs_parts;
          for (int t = lane; t < g.n_tiles * g.obs_parts; t += 32) {   // low parts are terms like the others
            const double4 h = p[t];
            sum2_add(s[0], h.x);
            sum2_add(s[1], h.y);
            sum2_add(s[2], h.z);
            sum2_add(s[3], h.w);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) sum2_warp(s[q]);
        }
      }
      const int col = run.col0 + k;
      double2* o = scr + (size_t)col * (n_l + 1) * 5;
      if (lane == 0) {
        if (mode != 0 && g.per_l && l < n_l) {
          run.dip[((size_t)l * n_orb + k) * run.n_t + step] = make_double2(s[0].hi + s[0].lo, s[1].hi + s[1].lo);
          run.acc[((size_t)l * n_orb + k) * run.n_t + step] = make_double2(s[2].hi + s[2].lo, s[3].hi + s[3].lo);
        }
#pragma unroll
        for (int q = 0; q < 5; ++q) o[l * 5 + q] = make_double2(s[q].hi, s[q].lo);
      }
      if (i + stride < rows) continue;
      // one fence for this warp's rows, then each counts; the last of an orbital's rows adds the totals
      if (lane == 0) __threadfence();
      for (int ii = i0; ii <= i; ii += stride) {
        const int kk = ii == i ? k : ii % n_orb;
        sum_rows(kk);
      }
    }
  }

  // rho_L(r) = sum_kso occ * density_kso (hartreePotentialDensity.cuh:58-60, orbital order)
  auto multipole = [&](int L, int q) {
    double s = 0.0;
    for (int k = 0; k < run.n_orb; ++k)
      s += (double)g.col_occ[run.col0 + k] * g.dens[((size_t)(run.col0 + k) * N_DEN + L) * n_r + q];
    return s;
  };

  if (role < g.n_den) {
    const int L = role;
    double* F = fsm;              // [N_r] forward partial sums
    double* G = fsm + n_r;        // backward partial sums
    // v_L(r_a) = r_a^-(L+1) sum_{b<=a} rho(b) r_b^L + r_a^L sum_{b>a} rho(b) r_b^-(L+1)
    for (int q = tid; q < n_r; q += FIN_THREADS) {
      const double rb = g.r[q], rho = multipole(L, q);
      F[q] = rho * ipow(rb, L);
      G[q] = rho / ipow(rb, L + 1);
    }
    __syncthreads();
    block_scans_dd(F, G, n_r, wsum);
    for (int q = tid; q < n_r; q += FIN_THREADS) {
      const double ra = g.r[q];
      const double v = F[q] / ipow(ra, L + 1) + ipow(ra, L) * G[q];
      run.v[(size_t)L * n_r + q] = v;
      if (mode == 0 && L == 0) run.v0[q] = v;
    }
  }

  if (role >= g.n_den && !obs_block) {
    const bool pw92 = (run.flags & RUN_FLAG_PW92) != 0;
    const int q = (role - g.n_den) * FIN_THREADS + tid;
    if (q < n_r) {
      const double rho0 = g.n_den > 0 ? multipole(0, q) : 0.0;
      // h_calculateExchangeCorrelationPotential.cuh:33-44
      double den = g.n_g_fac * (rho0 / 4.0 / M_PI + run.rho_frozen[q]) / g.drdx[q] * pow(g.P[q], 2.0);
      const double rq = g.r[q];
      if (mode == 0) {
        double vx0 = -pow(3.0 / M_PI * den, 1.0 / 3.0);
        vx0 /= pow(rq, 2.0 / 3.0);
        if (pw92) {
          // PW92 correlation of n = den / r^2 (not in the reference)
          const double n = fmax(den / (rq * rq), 1e-300);
          const double a = 0.031091, a1 = 0.21370, b1 = 7.5957, b2 = 3.5876, b3 = 1.6382, b4 = 0.49294;
          const double rs = cbrt(3.0 / (4.0 * M_PI * n)), srs = sqrt(rs);
          const double q0 = -2.0 * a * (1.0 + a1 * rs);
          const double q1 = 2.0 * a * (b1 * srs + b2 * rs + b3 * rs * srs + b4 * rs * rs);
          const double q1p = a * (b1 / srs + 2.0 * b2 + 3.0 * b3 * srs + 4.0 * b4 * rs);
          const double lg = log1p(1.0 / q1);
          vx0 += q0 * lg - rs / 3.0 * (-2.0 * a * a1 * lg - q0 * q1p / (q1 * q1 + q1));
        }
        run.vexc0[q] = vx0;
      }
      if (den < 0.0) den = 0.0;
      double vx = -pow(3.0 / M_PI * den, 1.0 / 3.0);
      vx /= pow(rq, 2.0 / 3.0);
      if (pw92) {
        const double n = fmax(den / (rq * rq), 1e-300);
        const double a = 0.031091, a1 = 0.21370, b1 = 7.5957, b2 = 3.5876, b3 = 1.6382, b4 = 0.49294;
        const double rs = cbrt(3.0 / (4.0 * M_PI * n)), srs = sqrt(rs);
        const double q0 = -2.0 * a * (1.0 + a1 * rs);
        const double q1 = 2.0 * a * (b1 * srs + b2 * rs + b3 * rs * srs + b4 * rs * rs);
        const double q1p = a * (b1 / srs + 2.0 * b2 + 3.0 * b3 * srs + 4.0 * b4 * rs);
        const double lg = log1p(1.0 / q1);
        vx += q0 * lg - rs / 3.0 * (-2.0 * a * a1 * lg - q0 * q1p / (q1 * q1 + q1));
      }
      // GGB_RUN_XC_FROZEN: the exchange-correlation potential stays at its t = 0 value
      run.vexc[q] = (run.flags & RUN_FLAG_XC_FROZEN) ? run.vexc0[q] : vx;
    }
  }
}

void launch_finalize(const GroupArgs& g, const double2* x, int mode, cudaStream_t s) {
  const dim3 grid(g.n_runs * (g.n_den + fin_xc_blocks(g, mode) + g.fin_ob)), block(FIN_THREADS);
  const size_t smem = g.n_den > 0 ? 2 * (size_t)g.n_r * sizeof(double) : 0;
  if (x) k_finalize<true><<<grid, block, smem, s>>>(g, x, mode);
  else k_finalize<false><<<grid, block, smem, s>>>(g, x, mode);
}

// Allow a kernel the largest dynamic shared memory the device offers beyond its static part.
cudaError_t set_max_dynamic_smem(const void* fn, int optin) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
}

cudaError_t configure_kernels_fp64(int n_l_max, int n_r_max) {
  int dev = 0, optin = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (angular_smem_fp64(n_l_max) > (size_t)optin || 3 * (size_t)n_r_max * sizeof(double) > (size_t)optin)
    return cudaErrorInvalidValue;
  g_angular_sms = g_radial_sms = sms;
  return cudaSuccess;
}

// The attribute is global per function: set to the device's opt-in maximum, so that contexts of different
// sizes can coexist.  Callers check their own sizes against it.  Only for the kernels that the group
// launches: the first mention of a kernel in a process loads it (all of this file's forms: 3 ms of the first
// context of 33 channels, more with more).
cudaError_t configure_group_fp64(const GroupArgs& g, bool radial, bool angular, bool obs_rows) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess && angular) e = set_max_dynamic_smem((const void*)angular_launch(g).fn, optin);
  if (e == cudaSuccess && radial && radial_tiles(g.n_cols, g.n_r, g.n_l))
    e = set_max_dynamic_smem((const void*)radial_tile_of(g.n_cols).fn, optin);
  if (e == cudaSuccess && g.theta_tab) e = configure_theta(optin);
  if (e == cudaSuccess) e = set_max_dynamic_smem(obs_rows ? (const void*)k_finalize<true> : (const void*)k_finalize<false>, optin);
  return e;
}

}  // namespace ggb
