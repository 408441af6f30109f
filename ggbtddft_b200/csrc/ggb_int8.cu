// Integer-split form of the step (GGB_SPLIT_INT8): exact accumulation on tcgen05.
//
// Why: the tensor cores' FP32 accumulators do not round to nearest.  Every accumulator update
// shrinks |acc| by a fraction of an ulp, always in the same direction, and a time step makes a few
// hundred updates per orbital value: the norm then decays geometrically (measured: ~1.4e-8 per
// update, 2.4 % over the 8,826 steps of the hydrogen pulse).  Integer products accumulate exactly.
//
// Representation (Ozaki-style split, base 256):
//   every operand row (a row of W_l, of a chain matrix S^T, of orbital values) is scaled by a power
//   of two 2^e that puts its largest |value| in [63, 126), rounded once to an integer T ~ v 2^e 2^24
//   (to nearest for orbital values; dithered for the constant operators, below)
//   (|T| < 2^31) and cut into its four balanced base-256 digits, the bytes of T + 0x80808080 each
//   less 128 (an int8 in [-128, 127]):
//       v 2^e = a1 + a2 2^-8 + a3 2^-16 + a4 2^-24 (+ at most 2^-25)
//   A row is resolved to ~2^-31 of its own maximum.  The constant operators (W_l, the chain
//   matrices) are applied every step, so a fixed rounding error of theirs compounds linearly over
//   the pulse (measured: W rounded to nearest alone moves the helium harmonics by 6e-4).  They are
//   therefore held as several dithered variants, rounded with offsets that cycle through
//   (j + 1/2) / n_var, and the step counter picks variant (step mod n_var): over n_var steps the
//   variants average to the exact operator to within 2^-24 / (2 n_var) of the row scale, and what
//   is left of the rounding is a zero-mean oscillation.  The orbital values are rounded to nearest
//   afresh at every product, which is already zero-mean.
//   product: the ten slice pairs (j, m) with j + m <= 3 (0-based; the rest weigh < 2^-32 of the
//   row maxima and are zero-mean), accumulated exactly in int32 tensor memory, one accumulator per
//   weight 2^-8(j+m); the epilogue combines the four accumulators exactly (int64 shifts), undoes the
//   two row scales exactly and rounds once to FP64.  The orbitals stay complex128 between products.
//   int32 range: |a b| <= 2^14, at most 8 products per k and accumulator, K <= 8192: <= 2^30.
//
//  k_slice_w_i8      W[l][k][i] -> A(i,k) stages [variant][l][row tile][k block][8][128][32] (Wr a1..a4, Wi a1..a4) + exponents
//  k_build_st_i8     chain matrices -> S^T stage images [variant n_mats + mat][m] + exponents
//  k_slice_x         orbitals (complex128) -> radial B operand stages (Xr, Xi, -Xi) + exponents
//  k_radial_i8       persistent radial product, kind::i8, 32-byte swizzle, 16 MMAs per 32-wide k block
//                    (each covers all x slices m of one W slice j):
//                      Re_s += Wr_j Xr_m + Wi_j (-Xi)_m,  Im_s += Wr_j Xi_m + Wi_j Xr_m   (j + m = s)
//  k_angular_i8      the angular chain with int8 operands, exact accumulation and per-point scales
#include <cuda.h>

#include <algorithm>
#include <cstdio>

#include "../../include/ggbtddft.h"
#include "ggb_angular.cuh"
#include "ggb_mixed.cuh"
#include "ggb_tc_common.cuh"

namespace ggb {

constexpr int I8_SLICES = 4;

// ---------------------------------------------------------------------------------------------
// slicing
// ---------------------------------------------------------------------------------------------


// exponent e with max 2^e in [63, 126) (0 for an all-zero row): with max = f 2^E, f in [0.5, 1),
// f 2^7 lies in [64, 126) unless f >= 126 / 128, and then f 2^6 lies in [63, 64).  Below 126 the
// top slice never exceeds 126 (see slice_int).  Clamped to e <= 1000 (rows below 1e-290 are
// resolved less finely; 2^e stays a normal double).
__device__ __forceinline__ int row_exponent(double mx) {
  if (!(mx > 0.0) || !(mx < 1e300)) return 0;
  int ex;
  const double f = frexp(mx, &ex);
  return min(1000, 7 - ex - (f >= 126.0 / 128.0 ? 1 : 0));
}

// The four balanced base-256 digits of T = rint(t3), t3 = t 2^24 with |t| < 126 (|T| < 2^31): the
// bytes of (T + 0x80808080) xor 0x80808080, each an int8 in [-128, 127], T = sum_k a_k 2^(8(3-k)).
__device__ __forceinline__ uint32_t slice_word(double t3) {
  return ((uint32_t)__double2int_rn(t3) + 0x80808080u) ^ 0x80808080u;
}
// byte (3 - k) of four slice words as one word per plane k (the first word's byte lowest)
__device__ __forceinline__ void plane_words(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t (&p)[4]) {
  const uint32_t a = __byte_perm(w0, w1, 0x6273), b = __byte_perm(w2, w3, 0x6273);
  const uint32_t c = __byte_perm(w0, w1, 0x4051), d = __byte_perm(w2, w3, 0x4051);
  p[0] = __byte_perm(a, b, 0x5410);
  p[1] = __byte_perm(a, b, 0x7632);
  p[2] = __byte_perm(c, d, 0x5410);
  p[3] = __byte_perm(c, d, 0x7632);
}
// the four slices of t3 stored one byte at dst + k * PLANE, most significant first
template <uint32_t PLANE>
__device__ __forceinline__ void store_slices(uint8_t* dst, double t3) {
  const uint32_t v = slice_word(t3);
  dst[0] = (uint8_t)(v >> 24);
  dst[PLANE] = (uint8_t)(v >> 16);
  dst[2 * PLANE] = (uint8_t)(v >> 8);
  dst[3 * PLANE] = (uint8_t)v;
}
// Dithered variants of the constant operators: variant v of element (a, b, c) rounds t 2^24 down
// after adding ((v + h(a, b, c)) mod n_var + 1/2) / n_var.  Over the n_var variants the offsets
// take every value once, so their mean is t 2^24 to within 1 / (2 n_var); the hash h staggers the
// cycle from element to element, so that one step's errors are as uncorrelated as rounding to
// nearest.  n_var is a power of two.
constexpr int I8_W_VARIANTS = 8;
constexpr int I8_S_VARIANTS = 16;

__device__ __forceinline__ uint32_t dither_hash(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t h = a * 0x9E3779B1u ^ b * 0x85EBCA77u ^ c * 0xC2B2AE3Du;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 13;
  return h;
}
__device__ __forceinline__ double dither_offset(int v, int n_var, uint32_t h) {
  return ((double)((v + (int)(h >> 8)) & (n_var - 1)) + 0.5) / (double)n_var;
}
// the four slices of floor(t 2^24 + d) (|t| < 126, 0 < d < 1) as int8 values, most significant first
__device__ __forceinline__ void slice4_dithered(double t, double d, int8_t* s) {
  const uint32_t v = ((uint32_t)__double2int_rd(fma(t, 16777216.0, d)) + 0x80808080u) ^ 0x80808080u;
#pragma unroll
  for (int q = 0; q < I8_SLICES; ++q) s[q] = (int8_t)(uint8_t)(v >> (24 - 8 * q));
}

// row maxima of A(i,k) = W[l][k][i] over k (re and im)
__global__ void k_w_rowmax(const double2* __restrict__ W, int* __restrict__ wexp, int n_r, int rows_pad) {
  const int l = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows_pad) return;
  double mx = 0.0;
  if (i < n_r)
    for (int k = 0; k < n_r; ++k) {
      const double2 w = W[((size_t)l * n_r + k) * n_r + i];
      mx = fmax(mx, fmax(fabs(w.x), fabs(w.y)));
    }
  wexp[(size_t)l * rows_pad + i] = row_exponent(mx);
}

// Operand tiles of the radial product in memory are the shared-memory image of a pipeline stage: per
// (tile of rows, 32-wide k block) the slice planes one after the other, each [rows][32 bytes] with the
// 32-byte swizzle already applied (the two 16-byte halves of a row change places in rows 4 .. 7 of every
// eight), so that a stage is one contiguous copy.  The last tiles are only as high as the matrix needs:
// N_r rounded up to 8 rows of W (the product's further rows are what follows in the buffer, never
// read from the accumulators), the orbital columns rounded up to 16 (the MMAs' N follows).  As a [rows][k]
// matrix a stage was a TMA box of 32-byte rows, 1024 and more of them, which paced the copies: 69 -> 53 us for
// one argon run (N_r 600, N_l 97: 283 MB of W, 5.3 TB/s), 176 -> 155 us for ten (123 with the trimmed tiles
// and 32 columns a tile), 990 -> 859 us for 21 at N_r 1000, N_l 161.
__host__ __device__ __forceinline__ uint32_t r8_row_off(int row, int k) {
  return (uint32_t)(row * 32 + ((((k >> 4) & 1) ^ ((row >> 2) & 1)) << 4) + (k & 15));
}

// A(i,k) tiles, transposed through shared memory (read along i, write along k)
__global__ void k_slice_w_i8(const double2* __restrict__ W, const int* __restrict__ wexp, int8_t* __restrict__ Wi8,
                             int n_r, int rows8, int rows_pad, int k_pad, int variant, int n_var) {
  __shared__ double2 t[32][33];
  const int l = blockIdx.z;
  const int i0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int q = ty; q < 32; q += 8) {
    const int k = k0 + q, i = i0 + tx;
    t[q][tx] = (k < n_r && i < n_r) ? W[((size_t)l * n_r + k) * n_r + i] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int n_kb = k_pad / 32;
  for (int q = ty; q < 32; q += 8) {
    const int i = i0 + q, k = k0 + tx;
    // the last row tile is rows8 - 128 mt rows high
    const int mt = i / 128, plane = min(128, rows8 - 128 * mt) * 32;
    int8_t* base = Wi8 + ((size_t)l * rows8 + 128 * mt) * n_kb * (2 * I8_SLICES * 32) + (size_t)(k0 / 32) * (2 * I8_SLICES) * plane +
                   r8_row_off(i % 128, tx);
    if (i < rows8 && k < k_pad) {
      const double sc = ldexp(1.0, wexp[(size_t)l * rows_pad + i]);
      const double2 w = t[tx][q];
      const uint32_t h = dither_hash((uint32_t)l, (uint32_t)i, (uint32_t)k);
      int8_t sr[I8_SLICES], si[I8_SLICES];
      slice4_dithered(w.x * sc, dither_offset(variant, n_var, h), sr);
      slice4_dithered(w.y * sc, dither_offset(variant, n_var, h * 0x165667B1u), si);
#pragma unroll
      for (int p = 0; p < I8_SLICES; ++p) {
        base[p * plane] = sr[p];
        base[(I8_SLICES + p) * plane] = si[p];
      }
    }
  }
}

// S^T planes of the chain matrices as the shared-memory images of the angular kernel's stages: per
// (variant, mat, m), per M tile of 128 rows (channels j) and k atom of 128 (l), the four slice planes
// [rows][pitch bytes], K-major, the swizzle of that pitch applied.  Only what the products need: the rows
// rounded up to 8, the k atom's 32-wide steps (pitch 32, 64 or 128; three steps take 128).  N_l = 161:
// 126 KB a matrix where full 128 x 128 tiles are 256, and these copies (one matrix per 16 radii, product
// and orbital) were at what L2 delivers to the SMs.
struct StGeom {
  int rows8, k_steps, psum;           // rows, 32-wide k steps, sum of the atoms' pitches
  __host__ __device__ int rows(int mt) const { return rows8 - 128 * mt < 128 ? rows8 - 128 * mt : 128; }
  __host__ __device__ int pitch(int ka) const {
    const int nk = k_steps - 4 * ka;
    return nk <= 0 ? 0 : nk == 1 ? 32 : nk == 2 ? 64 : 128;
  }
  __host__ __device__ size_t tile(int mt, int ka) const {   // offset of a tile's first plane
    return (size_t)4 * (128 * mt * psum + (ka ? rows(mt) * pitch(0) : 0));
  }
  __host__ __device__ size_t bytes() const { return (size_t)4 * rows8 * psum; }
  static StGeom of(int n_l) {
    StGeom g{(n_l + 7) & ~7, (n_l + 31) / 32, 0};
    g.psum = g.pitch(0) + g.pitch(1);
    return g;
  }
};
// A product's tiles (i = M tile, k atom) pass through the four stages (one per slice plane, 16 KB) in
// rounds: the first tile, then the three others at once where their planes fit a stage together (N_l = 161:
// 15.5 KB), else one by one.  A stage is refilled when its products are done, and the copy's latency is
// waited for between rounds.
static bool st_one_round(const StGeom& g) {
  return g.rows(0) * g.pitch(1) + g.rows(1) * (g.pitch(0) + g.pitch(1)) <= 128 * 128;
}
// byte of (row, k) in a plane of this pitch
__device__ __forceinline__ int st_off(int pitch, int row, int k) {
  const int x = pitch == 128 ? row & 7 : pitch == 64 ? (row >> 1) & 3 : (row >> 2) & 1;
  return row * pitch + (((k >> 4) ^ x) << 4) + (k & 15);
}

// S^T images with the row (j) exponents
__global__ void k_build_st_i8(const double* __restrict__ mats, int8_t* __restrict__ St, int* __restrict__ sexp,
                              int n_mm, int n_m, int n_l, int ldS, int rows, StGeom geo, int variant, int n_var) {
  const int row = blockIdx.x;                 // (mat * n_m + m) * rows + j
  const int mm = row / rows, j = row - mm * rows;
  if (mm >= n_mm) return;
  __shared__ double red[256];
  double mx = 0.0;
  for (int l = threadIdx.x; l < n_l; l += blockDim.x)
    if (j < n_l) mx = fmax(mx, fabs(mats[((size_t)mm * n_l + l) * ldS + j]));
  red[threadIdx.x] = mx;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  const int e = row_exponent(red[0]);
  if (threadIdx.x == 0 && variant == 0) sexp[row] = e;
  const double sc = ldexp(1.0, e);
  if (j >= geo.rows8) return;
  const int mt = j / 128;
  for (int l = threadIdx.x; l < 32 * geo.k_steps; l += blockDim.x) {
    const double v = (j < n_l && l < n_l) ? mats[((size_t)mm * n_l + l) * ldS + j] * sc : 0.0;
    int8_t s[I8_SLICES];
    // the hash leaves out m, so that a matrix gets the same variants in any group of runs
    slice4_dithered(v, dither_offset(variant, n_var, dither_hash((uint32_t)(mm / n_m), (uint32_t)j, (uint32_t)l)), s);
    const int ka = l / 128, pitch = geo.pitch(ka);
    int8_t* t = St + (size_t)mm * geo.bytes() + geo.tile(mt, ka) + st_off(pitch, j - 128 * mt, l - 128 * ka);
#pragma unroll
    for (int p = 0; p < I8_SLICES; ++p) t[(size_t)p * geo.rows(mt) * pitch] = s[p];
  }
}

// ---------------------------------------------------------------------------------------------
// radial product, kind::i8
// ---------------------------------------------------------------------------------------------

constexpr int R8_BM = 128, R8_BK = 32, R8_THREADS = 192;
constexpr int R8_W_PLANES = 8;      // Wr a1..a4, Wi a1..a4
constexpr int R8_X_PLANES = 12;     // Xr b1..b4, Xi b1..b4, -Xi b1..b4

__host__ __device__ constexpr uint32_t idesc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void tc_mma_i8_if(uint32_t elected, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(elected));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

// 2^k as a double (0 below the normal range)
__device__ __forceinline__ double pow2i(int k) {
  return k < -1022 ? 0.0 : __longlong_as_double((long long)(k + 1023) << 52);
}
// sum_s D_s 2^(8(3-s)) of the four int32 accumulators of column u, exactly (|D_s| <= 2^30: < 2^55)
template <int W>
__device__ __forceinline__ long long combine_int(const uint32_t (&d)[4][W], int u) {
  return (long long)(int)d[0][u] * 16777216LL + (long long)(int)d[1][u] * 65536LL + (long long)(int)d[2][u] * 256LL +
         (long long)(int)d[3][u];
}
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, uint32_t (&v)[2]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(taddr));
}

template <int BN>
struct R8Tile {
  static constexpr int A_PLANE = R8_BM * R8_BK;     // 4 KB
  static constexpr int B_PLANE = BN * R8_BK;
  static constexpr int A_STAGE = R8_W_PLANES * A_PLANE;
  static constexpr int STAGE = A_STAGE + R8_X_PLANES * B_PLANE;
  static constexpr int ACC_COLS = 8 * BN;           // Re s=2..5, Im s=2..5
  static constexpr int NBUF = (2 * ACC_COLS <= 512) ? 2 : 1;
  static constexpr int TMEM_COLS = NBUF * ACC_COLS <= 32 ? 32 : NBUF * ACC_COLS <= 64 ? 64
                                 : NBUF * ACC_COLS <= 128 ? 128 : NBUF * ACC_COLS <= 256 ? 256 : 512;
};

template <int BN>
__global__ void __launch_bounds__(R8_THREADS, 1)
k_radial_i8(const int8_t* __restrict__ W, size_t w_variant, const int8_t* __restrict__ X,
            const int* __restrict__ wexp, const int* __restrict__ xexp, int n_r, int rows_pad, int n_cols,
            int cols_pad, int n_l, int n_k_blocks, int stages, const int* __restrict__ step, int n_var,
            double2* __restrict__ Y, unsigned* status) {
  using T = R8Tile<BN>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t full_bar[8], empty_bar[8], accf_bar[2], acce_bar[2], drain_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  // aligned by an offset from the __shared__ array itself, so that the compiler keeps the shared
  // address space (shared loads and stores, not generic ones) for every access through it
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = (n_r + R8_BM - 1) / R8_BM, n_tiles = (n_cols + BN - 1) / BN;
  const int total = m_tiles * n_tiles * n_l;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf_bar[b], 1);
      mbar_init(&acce_bar[b], 4);
    }
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_slot, T::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* abort_p = &abort_flag;
  // rows of a W stage and columns of an x stage: full tiles but for the last ones
  const int rows8 = (n_r + 7) & ~7, cols16 = (n_cols + 15) & ~15;
  auto tile_rows = [&](int mt) { return min(R8_BM, rows8 - mt * R8_BM); };
  auto tile_cols = [&](int nt) { return min(BN, cols16 - nt * BN); };
  // tile order: N tile fastest, so CTAs that share a W tile run side by side (one HBM read)
  auto decode = [&](int tile, int& mt, int& nt, int& l) {
    // (rotated from round to round where every round would give a CTA the same N tile: the last one
    // is narrower)
    nt = (tile + (gridDim.x % n_tiles == 0 ? tile / (int)gridDim.x : 0)) % n_tiles;
    const int rest = tile / n_tiles;
    mt = rest % m_tiles;
    l = rest / m_tiles;
  };

  if (warp == 0) {
    if (lane == 0) {
      const int var = *step & (n_var - 1);     // this step's variant of W
      const int8_t* Wv = W + (size_t)var * w_variant;
      // W streams through L2 once a step (its variants alternate): read by one CTA only, it must not push
      // the orbitals, the chain matrices and the kept vectors out; read by several, it stays for them
      const uint64_t w_policy = l2_evict_first();
      int it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
        int mt, nt, l;
        decode(tile, mt, nt, l);
        const uint32_t wb = R8_W_PLANES * R8_BK * tile_rows(mt), xb = R8_X_PLANES * R8_BK * tile_cols(nt);
        const int8_t* wsrc = Wv + ((size_t)l * rows8 + mt * R8_BM) * n_k_blocks * (R8_W_PLANES * R8_BK);
        const int8_t* xsrc = X + ((size_t)l * cols16 + nt * BN) * n_k_blocks * (R8_X_PLANES * R8_BK);
        for (int kb = 0; kb < n_k_blocks; ++kb, ++it, wsrc += wb, xsrc += xb) {
          const int s = it % stages;
          if (it >= stages && !mbar_wait(&empty_bar[s], ((it / stages) & 1) ^ 1, abort_p)) {
            ok = false;
            break;
          }
          uint8_t* st = smem + (size_t)s * T::STAGE;
          mbar_expect_tx(&full_bar[s], wb + xb);
          if (n_tiles == 1) bulk_g2s_hint(st, wsrc, wb, &full_bar[s], w_policy);
          else bulk_g2s(st, wsrc, wb, &full_bar[s]);
          bulk_g2s(st + T::A_STAGE, xsrc, xb, &full_bar[s]);
        }
      }
      if (!ok)
        for (int q = (it > stages ? it - stages : 0); q < it; ++q) mbar_drain(&full_bar[q % stages], (q / stages) & 1);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // descriptors: those of stage 0 plus the byte offset / 16 in the start-address field (this
      // thread's issue rate paces the products)
      const uint64_t desc0 = sdesc_kmajor(smem_u32(smem), 32, 6);
      int local = 0, s = 0, ph = 0;
      for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++local) {
        const int buf = (T::NBUF == 2) ? (local & 1) : 0;
        const int use = (T::NBUF == 2) ? (local >> 1) : local;
        if (use >= 1 && !mbar_wait(&acce_bar[buf], (use - 1) & 1, abort_p)) break;
        tc_fence_after();
        const uint32_t d0 = tmem + buf * T::ACC_COLS;
        int mt, nt, l;
        decode(tile, mt, nt, l);
        const uint32_t bn = tile_cols(nt), wp = tile_rows(mt) * R8_BK, xp = bn * R8_BK;   // columns, plane sizes
        const uint32_t idesc[I8_SLICES] = {idesc_i8(R8_BM, 4 * bn), idesc_i8(R8_BM, 3 * bn), idesc_i8(R8_BM, 2 * bn),
                                           idesc_i8(R8_BM, bn)};
        bool ok = true;
        for (int kb = 0; kb < n_k_blocks; ++kb) {
          if (!mbar_wait(&full_bar[s], ph, abort_p)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t da = desc0 + (uint64_t)(((uint32_t)s * T::STAGE) >> 4);
          // one 32-wide k block: for each W slice j, one MMA per real product covers the x slices
          // m = 0 .. 3 - j at once (the x planes of each kind are contiguous rows), N = (4 - j) bn,
          // written from accumulator group j on, so that column group m lands on weight 2^-8(j+m)
          const uint64_t xr = da + (T::A_STAGE >> 4);
          const uint64_t xi = xr + ((I8_SLICES * xp) >> 4);
          const uint64_t xn = xr + ((2 * I8_SLICES * xp) >> 4);
#pragma unroll
          for (int j = 0; j < I8_SLICES; ++j) {
            const uint64_t wr = da + ((j * wp) >> 4);
            const uint64_t wi = da + (((I8_SLICES + j) * wp) >> 4);
            const uint32_t dre = d0 + j * bn, dim = d0 + (4 + j) * bn;
            const uint32_t first = (kb == 0 && j == 0) ? 0u : 1u;
            tc_mma_i8(dre, wr, xr, idesc[j], first);
            tc_mma_i8(dre, wi, xn, idesc[j], 1u);
            tc_mma_i8(dim, wr, xi, idesc[j], first);
            tc_mma_i8(dim, wi, xr, idesc[j], 1u);
          }
          tc_commit(&empty_bar[s]);
          if (++s == stages) {
            s = 0;
            ph ^= 1;
          }
        }
        tc_commit(&accf_bar[buf]);
        if (!ok) break;
      }
    }
  } else {
    const int q = warp & 3;
    const uint32_t lane_base = (uint32_t)(32 * q) << 16;
    int local = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++local) {
      const int buf = (T::NBUF == 2) ? (local & 1) : 0;
      const int use = (T::NBUF == 2) ? (local >> 1) : local;
      int mt, nt, l;
      decode(tile, mt, nt, l);
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&accf_bar[buf], use & 1, abort_p));
      tc_fence_after();
      if (!ok) break;
      const int i = mt * R8_BM + 32 * q + lane, c0 = nt * BN;
      const int ew = (i < n_r) ? wexp[(size_t)l * rows_pad + i] : 0;
      const uint32_t d0 = tmem + buf * T::ACC_COLS + lane_base;
      const int bn = tile_cols(nt), used = min(bn, n_cols - c0);
#pragma unroll 1
      for (int cc = 0; cc < used; cc += 8) {
        uint32_t re[4][8], im[4][8];
#pragma unroll
        for (int sidx = 0; sidx < 4; ++sidx) {
          tmem_ld8(d0 + sidx * bn + cc, re[sidx]);
          tmem_ld8(d0 + (4 + sidx) * bn + cc, im[sidx]);
        }
        tmem_ld_wait();
#pragma unroll
        for (int sidx = 0; sidx < 4; ++sidx) {
          tmem_regs_ready(re[sidx]);
          tmem_regs_ready(im[sidx]);
        }
        if (i < n_r) {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int c = c0 + cc + u;
            if (c < n_cols) {
              const double sc = pow2i(-ew - xexp[(size_t)l * cols_pad + c] - 24);
              Y[((size_t)l * n_cols + c) * n_r + i] =
                  make_double2((double)combine_int(re, u) * sc, (double)combine_int(im, u) * sc);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acce_bar[buf]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicOr(status, ST_TC_TIMEOUT);
  if (warp == 1) {
    if (abort_flag && lane == 0) {
      tc_commit(&drain_bar);
      mbar_drain(&drain_bar, 0);
    }
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, T::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------
// angular chain, kind::i8
// ---------------------------------------------------------------------------------------------

constexpr int A8_THREADS = 576;          // TMA warp, MMA warp, 16 epilogue warps
constexpr int A8_EPI_WARP0 = 2;
constexpr int A8_BLOCKS_PER_SM = 2;
constexpr int A8_KATOM = 128;            // int8 per 128-byte swizzled row
constexpr int A8_A_TILE = 128 * 128;     // one S^T slice plane: 128 rows (j) x 128 k (l), one stage
constexpr int A8_PTS = 8;                // points per epilogue thread and product
constexpr int A8_DEN_WARPS = 10;         // warps of the density's partial sums (fixes their order)
constexpr int A8_TMEM_COLS = 256;        // 4 accumulators x 2 NP columns x m_tiles: two CTAs per SM

struct Ang8Args {
  int k_atoms;            // ceil(N_l / 128)
  int m_tiles;            // ceil(N_l / 128)
  int k_steps;            // ceil(N_l / 32): 32-wide K steps that carry data
  int stages;
  const int8_t* St;       // S^T images [variant n_mats + mat][m], geo.bytes() each
  StGeom geo;
  int one_round;          // tiles 1 .. 3 pass through the stages together
  const int* sexp;        // S^T row exponents [mat][m][rows]
  int rows;               // m_tiles * 128
  int sms;
  int n_mats;             // chain matrices per variant
  int n_var;              // dithered variants of the chain matrices (a power of two)
  // theta form: the node-basis vectors of the second half after its phase, [N_l][n_cols][N_r]
  // (nullptr: not kept); g.yth_step says which step's first half may start from them
  double2* yth;
};

// descriptor of a K-major operand of this row pitch with its swizzle
__device__ __forceinline__ uint64_t a8_sdesc(uint32_t saddr, int pitch) {
  return sdesc_kmajor(saddr, (uint32_t)pitch, pitch == 128 ? 2u : pitch == 64 ? 4u : 6u);
}

// Byte offset of (row n, k) of slice plane 0 in the B operand: per 128-wide k atom, the four slice
// planes of nrows K-major 128-byte-swizzled rows each, one after the other (plane q at + q nrows 128),
// so that for one k atom the planes form one operand of 4 nrows rows.
__device__ __forceinline__ uint32_t a8_off(int nrows, int n, int k) {
  const int chunk = ((k & 127) >> 4) ^ (n & 7);
  return (uint32_t)((k >> 7) * I8_SLICES * nrows * 128 + n * 128 + chunk * 16 + (k & 15));
}

// sin and cos of e in FP64: for |e| <= 1/2 the Maclaurin series through e^11 (sine) and e^12
// (cosine), evaluated by Estrin's scheme (short dependency chains); truncation below 2e-14 at
// |e| = 1/2 and far less for the small angles of most phases.  The length-gauge phase r E dt/2 of a
// step stays below 1/2 for the configurations here (r_max E_0 dt/2 <= 0.4); larger angles take the
// library sincos.
__device__ __forceinline__ void sincos_series(double e, double* s, double* c) {
  if (fabs(e) <= 0.5) {
    const double z = e * e, z2 = z * z, z4 = z2 * z2;
    const double s01 = fma(z, -1.0 / 6, 1.0), s23 = fma(z, -1.0 / 5040, 1.0 / 120);
    const double s45 = fma(z, -1.0 / 39916800, 1.0 / 362880);
    *s = e * fma(z4, s45, fma(z2, s23, s01));
    const double c01 = fma(z, -1.0 / 2, 1.0), c23 = fma(z, -1.0 / 720, 1.0 / 24);
    const double c45 = fma(z, -1.0 / 3628800, 1.0 / 40320);
    *c = fma(z4 * z2, 1.0 / 479001600.0, fma(z4, c45, fma(z2, c23, c01)));
  } else {
    sincos(e, s, c);
  }
}
// x exp(-i e), FP64
__device__ __forceinline__ double2 rotd(double2 x, double e) {
  double s, c;
  sincos_series(e, &s, &c);
  return make_double2(c * x.x + s * x.y, c * x.y - s * x.x);
}

template <int V>
struct I8c {
  static constexpr int value = V;
};
// One CTA per (orbital column, NP radii): NP = 32 for N_l <= 128 (one M tile of 128 channels),
// NP = 16 for N_l <= 256 (two M tiles), so that every CTA holds 256 TMEM columns and two CTAs share
// an SM (one CTA's epilogue overlaps the other's products and loads).
//
// The B operand (the l-vectors of the CTA's points, Re rows then Im rows) stays in shared memory
// as four int8 slice planes.  Every point carries one power-of-two scale for its Re and Im rows,
// chosen from the 2-norm of its l-vector: each product of the chain is an orthogonal matrix and
// each phase unitary, so that norm bounds every entry of every intermediate vector and one
// exponent serves the whole chain.  The chain matrices S^T stream through a pipeline of bulk
// copies, one slice plane (or the row tiles of one that fit, a round) per stage.  Orbitals in and out are complex128 (xout may alias xin: each CTA reads
// its whole tile before it writes).
//
// Basis reuse (theta form, t.yth set): a half-step is x <- V diag(phase) V^T x with V orthogonal,
// and nothing acts on the orbitals between the second half of one step and the first half of the
// next (the potentials only change the phase).  So V^T x at the start of the next first half is
// the second half's node-basis vector after its phase, which the second half keeps (t.yth, one
// FP64 copy); the next first half loads it, applies its own phase in the prologue and runs only
// its last product, one product instead of two.  The skipped pair V^T V is the identity up to the
// int8 operands' rounding (~2^-31 of each row), which is then not applied.  g.yth_step names the
// step that may start from the kept vectors; setting orbitals clears it.
template <int NP, bool SECOND_HALF, bool THETA>
__global__ void __launch_bounds__(A8_THREADS, A8_BLOCKS_PER_SM)
k_angular_i8(GroupArgs g, Ang8Args t, const double2* xin, double2* xout) {
  constexpr int NB = 2 * NP;                 // B rows: Re of NP points, then Im
  constexpr int B_TILE = NB * 128;           // one slice plane, one k atom
  constexpr int K_ATOMS = NP == 32 ? 1 : 2;  // = M tiles = ceil(N_l / 128)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t full_bar[4], empty_bar[4], acc_bar, xb_bar, drain_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ double pbase[5][NP];
  __shared__ double pnorm2[A8_THREADS / NP][NP];
  __shared__ double sdl[MAX_NL];
  __shared__ double prr[2][NP];               // second half: r and r^-2 of each point (0 past N_r)
  __shared__ double pscale3[NP], pinv[NP];    // 2^e(p) 2^24 and 2^-e(p) of each point's B rows
  // aligned by an offset from the __shared__ array itself, so that the compiler keeps the shared
  // address space (shared loads and stores, not generic ones) for every access through it
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  // stages of 16 KB, then the operand: the MMAs read 128 rows of a stage's tile whatever its height, up to
  // 16 KB past the last stage, which is the operand's memory (what they read there is never used)
  uint8_t* sst = smem;
  uint8_t* xb = smem + I8_SLICES * A8_A_TILE;                       // 4 planes x k_atoms x B_TILE, 32 KB
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_l = g.n_l;
  const int tilesN = (g.n_r + NP - 1) / NP;
  const int col = blockIdx.x / tilesN;
  const int r0 = (blockIdx.x - col * tilesN) * NP;
  const Chain& ch = g.chain[SECOND_HALF ? 1 : 0];
  const int n_ops = ch.n_ops;
  const int acc_cols = 4 * NB;                // per M tile: weights 2^0 .. 2^-24
  const int step_raw = *g.step;
  const int m = g.col_m[col], col_run = g.col_run[col];
  // basis reuse: the second half keeps its node-basis vectors, the first half of the step they
  // were kept for starts from them at its last product (o0 = 1, the theta chain having two)
  const bool keep_theta = THETA && SECOND_HALF && t.yth != nullptr;
  const bool from_theta = THETA && !SECOND_HALF && t.yth != nullptr && *g.yth_step == step_raw + 1;
  const int o0 = from_theta ? 1 : 0;

  // the x tile (all l, NP points): point fp = tid % NP, the l quads fg, fg + FG, ... of this thread, all
  // requested here, so that the rest of the set-up runs under their latency
  constexpr int FG = A8_THREADS / NP;          // l quads per round
  constexpr int FR = 2;                        // rounds: 32 quads (N_l <= 128, FG = 18) or 56 (N_l <= 220, FG = 36)
  const int fp = threadIdx.x % NP, fg = threadIdx.x / NP;
  double2 xv[FR][4];
  {
    const double2* src = (from_theta ? t.yth : xin) + (size_t)col * g.n_r + r0 + fp;
    const size_t ls = (size_t)g.n_cols * g.n_r;
    const bool rv = r0 + fp < g.n_r;
#pragma unroll
    for (int f = 0; f < FR; ++f)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int l = 4 * (fg + f * FG) + u;
        xv[f][u] = (l < n_l && rv) ? src[(size_t)l * ls] : make_double2(0.0, 0.0);
      }
  }
  const RunDev run = g.runs[col_run];
  const int step = step_raw < run.n_t ? step_raw : run.n_t - 1;
  const double hdt = 0.5 * g.dt;
  const double* pco = g.coef + ((size_t)CF_P * g.n_m + m) * n_l;

  if (threadIdx.x == 0) {
    for (int s = 0; s < t.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    mbar_init(&xb_bar, A8_THREADS / 32 - A8_EPI_WARP0);
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_slot, A8_TMEM_COLS);
  if (threadIdx.x < NP) {
    const int p = threadIdx.x, r = r0 + p;
    const bool rv = r < g.n_r;
    const int rc = rv ? r : 0;
    const double rr = rv ? g.r[r] : 1.0, E = run.E[step];
    double v1 = 0.0, v2 = 0.0, v3 = 0.0, sb = 0.0;
    if (g.hartree_on) {
      v1 = run.v[1 * g.n_r + rc];
      v2 = run.v[2 * g.n_r + rc];
      v3 = run.v[3 * g.n_r + rc];
      sb = run.v[rc] - run.v0[rc] + run.vexc[rc] - run.vexc0[rc];
    }
    pbase[0][p] = rr;
    pbase[1][p] = ((g.p_hartree || g.theta) ? (rr * E + v1) : (rr * E)) * hdt;
    pbase[2][p] = v2 * hdt;
    pbase[3][p] = v3 * hdt;
    pbase[4][p] = sb * hdt;
    if (SECOND_HALF) {
      prr[0][p] = rv ? rr : 0.0;
      prr[1][p] = rv ? 1.0 / (rr * rr) : 0.0;
    }
  }
  // what the fill's phase takes per l: the first product's eigenvalue (basis reuse) or the S coefficient
  for (int l = threadIdx.x; l < n_l; l += A8_THREADS)
    sdl[l] = SECOND_HALF ? (ch.pre_s ? pco[l] : 0.0) : g.dph[((size_t)ch.ops[0].coupling * g.n_m + m) * g.ldS + l];
  __syncthreads();
  // the first S^T slice planes are on their way while the operand is filled
  const int mat0 = ch.ops[o0].mat + (step_raw & (t.n_var - 1)) * t.n_mats;   // this step's variant
  if (threadIdx.x == 0) {
    const uint32_t plane = (uint32_t)(t.geo.rows(0) * t.geo.pitch(0));
    const int8_t* src = t.St + ((size_t)mat0 * g.n_m + m) * t.geo.bytes();
#pragma unroll
    for (int pa = 0; pa < I8_SLICES; ++pa) {
      mbar_expect_tx(&full_bar[pa], plane);
      bulk_g2s(sst + pa * A8_A_TILE, src + pa * plane, plane, &full_bar[pa]);
    }
  }

  // operand: phases of the tile in registers (second half: the l-diagonal S phase; basis reuse: the
  // first product's phase, the same angle as its epilogue's), the per-point norms, then the slices
  const int lk = t.k_atoms * A8_KATOM;
  {
    double part = 0.0;
#pragma unroll
    for (int f = 0; f < FR; ++f)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int l = 4 * (fg + f * FG) + u;
        double2 w = xv[f][u];
        if (l < n_l) {
          if (SECOND_HALF && ch.pre_s) w = rotd(w, pbase[4][fp] + sdl[l] * pbase[2][fp]);
          if (!SECOND_HALF && THETA && from_theta && l >= m) {
            const double dj = sdl[l], p2j = legendre_p2(dj), p3j = legendre_p3(dj);
            double ang = pbase[1][fp] * dj + pbase[2][fp] * p2j + pbase[3][fp] * p3j + pbase[4][fp];
            if (g.theta_tab && r0 + fp < g.n_r) ang += run.htab[((size_t)m * n_l + l) * g.n_r + r0 + fp] * hdt;
            w = rotd(w, ang);
          }
        }
        xv[f][u] = w;
        part += w.x * w.x + w.y * w.y;
      }
    pnorm2[fg][fp] = part;
  }
  __syncthreads();
  if (threadIdx.x < NP) {
    // |Re y_j|, |Im y_j| <= |y| = |x| for every vector of the chain; the margin covers the chain's
    // rounding and the non-orthogonality of the sliced matrices (both ~2^-31)
    double n2 = 0.0;
#pragma unroll
    for (int q = 0; q < FG; ++q) n2 += pnorm2[q][threadIdx.x];
    const int e = row_exponent(sqrt(n2) * (1.0 + 0x1p-20));
    pscale3[threadIdx.x] = pow2i(e + 24);
    pinv[threadIdx.x] = pow2i(-e);
  }
  __syncthreads();
  // four consecutive l per thread: one word per slice plane, Re in row fp and Im in row NP + fp (the
  // same swizzle chunk, NP being a multiple of 8); zero beyond N_l up to the K steps that are read
  {
    const double sc3 = pscale3[fp];
#pragma unroll
    for (int f = 0; f < FR; ++f) {
      const int quad = fg + f * FG;
      if (quad < 8 * t.k_steps) {
        uint8_t* dst = xb + a8_off(2 * NP, fp, 4 * quad);
        uint32_t pr[I8_SLICES], pi[I8_SLICES];
        plane_words(slice_word(xv[f][0].x * sc3), slice_word(xv[f][1].x * sc3), slice_word(xv[f][2].x * sc3),
                    slice_word(xv[f][3].x * sc3), pr);
        plane_words(slice_word(xv[f][0].y * sc3), slice_word(xv[f][1].y * sc3), slice_word(xv[f][2].y * sc3),
                    slice_word(xv[f][3].y * sc3), pi);
#pragma unroll
        for (int k = 0; k < I8_SLICES; ++k) {
          *reinterpret_cast<uint32_t*>(dst + k * B_TILE) = pr[k];
          *reinterpret_cast<uint32_t*>(dst + k * B_TILE + NP * 128) = pi[k];
        }
      }
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // bring the x tile of the block that follows on this SM to L2, one row (NP radii of one l) per thread
  if (const unsigned nb = blockIdx.x + A8_BLOCKS_PER_SM * t.sms; nb < gridDim.x && (int)threadIdx.x < n_l) {
    const int ncol = nb / tilesN, nr0 = (nb - ncol * tilesN) * NP;
    const double2* row = (from_theta ? t.yth : xin) + ((size_t)threadIdx.x * g.n_cols + ncol) * g.n_r + nr0;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row), "r"(min(NP, g.n_r - nr0) * 16) : "memory");
  }
  const uint32_t tmem = tmem_slot;
  volatile int* abort_p = &abort_flag;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      // per tile: bytes of a slice plane and offset of the first one.  Worked out here and the rounds unrolled:
      // this thread shares its SM sub-partition with busy epilogue warps, so what it does per refill is
      // exposed between the rounds (as a loop over tiles with its index arithmetic: the halves of the coupling
      // chain at N_r 300, 30 columns 151 + 158 us at N_l 161 and 186 + 199 at 220; so: 131 + 140 and 158 + 171)
      uint32_t plane[K_ATOMS * K_ATOMS], off[K_ATOMS * K_ATOMS];
#pragma unroll
      for (int i = 0; i < K_ATOMS * K_ATOMS; ++i) {
        plane[i] = (uint32_t)(t.geo.rows(i / K_ATOMS) * t.geo.pitch(i % K_ATOMS));
        off[i] = (uint32_t)t.geo.tile(i / K_ATOMS, i % K_ATOMS);
      }
      const size_t mat_bytes = t.geo.bytes(), m_stride = mat_bytes * g.n_m;
      const int8_t* mats = t.St + (size_t)((step_raw & (t.n_var - 1)) * t.n_mats) * m_stride + m * mat_bytes;   // this step's variant
      for (int o = o0; o < n_ops && ok; ++o) {
        const int8_t* src = mats + ch.ops[o].mat * m_stride;
        // stage pa takes slice plane pa; the ring turns once per round
        auto load_round = [&](auto I0, auto I1) -> bool {
          uint32_t bytes = 0;
#pragma unroll
          for (int i = decltype(I0)::value; i < decltype(I1)::value; ++i) bytes += plane[i];
          const int round = it / I8_SLICES;
          if (round == 0) {                    // issued before the fill
            it += I8_SLICES;
            return true;
          }
#pragma unroll
          for (int pa = 0; pa < I8_SLICES; ++pa, ++it) {
            if (!mbar_wait(&empty_bar[pa], (round & 1) ^ 1, abort_p)) return false;
            mbar_expect_tx(&full_bar[pa], bytes);
            uint8_t* stage = sst + pa * A8_A_TILE;
#pragma unroll
            for (int i = decltype(I0)::value; i < decltype(I1)::value; ++i) {
              bulk_g2s(stage, src + off[i] + pa * plane[i], plane[i], &full_bar[pa]);
              stage += plane[i];
            }
          }
          return true;
        };
        ok = load_round(I8c<0>(), I8c<1>());
        if constexpr (K_ATOMS == 2) {
          if (t.one_round) {
            ok = ok && load_round(I8c<1>(), I8c<4>());
          } else {
            ok = ok && load_round(I8c<1>(), I8c<2>()) && load_round(I8c<2>(), I8c<3>()) && load_round(I8c<3>(), I8c<4>());
          }
        }
      }
      if (!ok)
        for (int q = (it > t.stages ? it - t.stages : 0); q < it; ++q) mbar_drain(&full_bar[q % t.stages], (q / t.stages) & 1);
    }
  } else if (warp == 1) {
    // one MMA per (S^T slice pa, 32-wide k step): N = (4 - pa) NB rows of the stacked x slice planes
    // 0 .. 3 - pa, written at TMEM column pa NB, so that its column group pb lands on the
    // accumulator of weight 2^-8(pa + pb)
    constexpr uint32_t idesc[I8_SLICES] = {idesc_i8(128, 4 * NB), idesc_i8(128, 3 * NB), idesc_i8(128, 2 * NB),
                                           idesc_i8(128, NB)};
    // The loads come four per round, one per slice plane pa, into a ring of four stages, so stage pa always
    // holds plane pa and the ring turns once per round.  Descriptors are those of stage 0 (or of the B
    // operand's atom) plus the byte offset / 16 in the start-address field.  This warp shares its SM
    // sub-partition with busy epilogue warps, and its issue rate paces the products.  (Rows past the M
    // tile's images, and the accumulator lanes they reach, hold what the buffer held: they only ever meet
    // the zero columns past N_l of the next product.)
    const uint32_t elected = elect_one();
    const uint64_t adesc0 = a8_sdesc(smem_u32(sst), t.geo.pitch(0)), adesc1 = a8_sdesc(smem_u32(sst), t.geo.pitch(1));
    const uint64_t bdesc = sdesc_kmajor(smem_u32(xb), 128, 2);
    uint32_t plane[K_ATOMS * K_ATOMS];
#pragma unroll
    for (int i = 0; i < K_ATOMS * K_ATOMS; ++i) plane[i] = (uint32_t)(t.geo.rows(i / K_ATOMS) * t.geo.pitch(i % K_ATOMS)) >> 4;
    int round = 0;
    for (int o = o0; o < n_ops; ++o) {
      if (o > o0 && !__all_sync(0xffffffffu, mbar_wait(&xb_bar, (o - o0 - 1) & 1, abort_p))) break;
      tc_fence_after();
      // tiles I0 .. I1 - 1 as one round, unrolled
      auto issue_round = [&](auto I0, auto I1) -> bool {
#pragma unroll
        for (int pa = 0; pa < I8_SLICES; ++pa) {
          if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[pa], round & 1, abort_p))) return false;
          tc_fence_after();
          uint32_t off = (pa * A8_A_TILE) >> 4;
#pragma unroll
          for (int i = decltype(I0)::value; i < decltype(I1)::value; ++i) {
            const int mt = i / K_ATOMS, ka = i % K_ATOMS;
            const uint32_t d0 = tmem + acc_cols * mt + pa * NB;
            const uint64_t ak = (ka ? adesc1 : adesc0) + off;
            const uint64_t bk = bdesc + (uint64_t)((ka * I8_SLICES * B_TILE) >> 4);
            const int nk = K_ATOMS == 2 && ka == 0 ? A8_KATOM / 32 : t.k_steps - ka * (A8_KATOM / 32);
#pragma unroll
            for (int kk = 0; kk < A8_KATOM / 32; ++kk)
              if (kk < nk) tc_mma_i8_if(elected, d0, ak + 2 * kk, bk + 2 * kk, idesc[pa], (ka | kk | pa) ? 1u : 0u);
            off += plane[i];
          }
          tc_commit_if(elected, &empty_bar[pa]);
        }
        ++round;
        return true;
      };
      bool ok = issue_round(I8c<0>(), I8c<1>());
      if constexpr (K_ATOMS == 2) {
        if (t.one_round) {
          ok = ok && issue_round(I8c<1>(), I8c<4>());
        } else {
          ok = ok && issue_round(I8c<1>(), I8c<2>()) && issue_round(I8c<2>(), I8c<3>()) && issue_round(I8c<3>(), I8c<4>());
        }
      }
      // one commit for all M tiles: every tile's products read the whole operand, which the
      // epilogue overwrites with the next product's
      tc_commit_if(elected, &acc_bar);
      if (!ok) break;
    }
  } else {
    const int ew = warp - A8_EPI_WARP0;
    const int q = warp & 3;                     // TMEM lane quarter of this warp
    const int grp = ew >> 2;                    // four warps per lane quarter share its (M tile, points)
    const int mt = (t.m_tiles == 2) ? grp >> 1 : 0;
    const int j = 128 * mt + 32 * q + lane;     // eigen-channel (M row) of this thread
    const int p_begin = A8_PTS * ((t.m_tiles == 2) ? grp & 1 : grp);
    // staging of the last product, [N_l][NP + 1] (the odd row length keeps both this write, lanes
    // along l, and the reads below, lanes along the points, free of bank conflicts)
    double2* stage_out = reinterpret_cast<double2*>(smem);
    const uint32_t d0 = tmem + ((uint32_t)(32 * q) << 16) + acc_cols * mt;
    // a warp whose 32 channels are all padding (j >= N_l) does no work: its rows of the next
    // operand stay as the fill left them (zero), and the next product's S^T columns there are zero
    const bool live = 128 * mt + 32 * q < n_l;
    for (int o = o0; o < n_ops; ++o) {
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&acc_bar, (o - o0) & 1, abort_p));
      tc_fence_after();
      if (!ok) break;
      const ChainOp op = ch.ops[o];
      const bool last = (o == n_ops - 1);
      // basis reuse: the second half keeps the first product's result after its phase (row j of
      // this column, from radius r0)
      double2* const ykeep = (keep_theta && o == 0 && j < n_l) ? t.yth + ((size_t)j * g.n_cols + col) * g.n_r + r0 : nullptr;
      if (!live) {
        if (!last) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&xb_bar);
        }
        continue;
      }
      const double* Dv = g.dph + ((size_t)op.coupling * g.n_m + m) * g.ldS;
      const double dj = (op.phase != PH_NONE && j >= m && j < n_l) ? Dv[j] : 0.0;
      const int pb = op.phase == PH_P ? 1 : op.phase == PH_D ? 2 : 3;
      // the theta form: angle = pbase1 x_j + pbase2 P_2(x_j) + pbase3 P_3(x_j) + pbase4 (all x dt/2), zero for
      // channels below m and past N_l
      const bool ph_theta = THETA && op.phase == PH_THETA, act = j >= m && j < n_l;
      const double p2j = legendre_p2(dj), p3j = legendre_p3(dj);
      const bool post_s = last && !SECOND_HALF && ch.post_s && j < n_l;
      const double pj = post_s ? pco[j] : 0.0;
      const double sj = pow2i(-t.sexp[((size_t)op.mat * g.n_m + m) * t.rows + j]);   // S^T row scale
      // software pipeline over chunks of 2 points: the next chunk's accumulators are requested
      // from tensor memory before this chunk is rotated and sliced
      constexpr int CH = 2;
      uint32_t re[4][CH], im[4][CH];
      auto tload = [&](int p0) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          tmem_ld2(d0 + s * NB + p0, re[s]);
          tmem_ld2(d0 + s * NB + NP + p0, im[s]);
        }
      };
      auto tready = [&]() {
        tmem_ld_wait();
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          tmem_regs_ready(re[s]);
          tmem_regs_ready(im[s]);
        }
      };
      tload(p_begin);
      tready();
#pragma unroll 1
      for (int c = 0; c < A8_PTS / CH; ++c) {
        const int p0 = p_begin + CH * c;
        // the accumulators hold y 2^(e_j + e_p) 2^24; rotations commute with the scale, and the
        // next product's slices want y 2^e_p 2^24: one exact power of two in between
        double2 v[CH];
#pragma unroll
        for (int u = 0; u < CH; ++u)
          v[u] = make_double2((double)combine_int(re, u) * sj, (double)combine_int(im, u) * sj);
        if (c + 1 < A8_PTS / CH) tload(p0 + CH);
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          const int p = p0 + u;
          if constexpr (THETA) {
            if (ph_theta) {
              double ang = pbase[1][p] * dj + pbase[2][p] * p2j + pbase[3][p] * p3j + pbase[4][p];
              // n_har > 4: the multipoles L >= 1 at this node come from the exact-quadrature table
              if (g.theta_tab && act && r0 + p < g.n_r) ang += run.htab[((size_t)m * n_l + j) * g.n_r + r0 + p] * hdt;
              v[u] = rotd(v[u], act ? ang : 0.0);
            }
          } else {
            if (dj != 0.0) v[u] = rotd(v[u], pbase[pb][p] * dj);
          }
          if (post_s) v[u] = rotd(v[u], pbase[4][p] + pj * pbase[2][p]);
          if (NP != 32 && ykeep && r0 + p < g.n_r) {
            const double sc = pinv[p] * 0x1p-24;
            ykeep[p] = make_double2(v[u].x * sc, v[u].y * sc);
          }
          if (!last) {
            if (j < lk) {
              const uint32_t o = a8_off(2 * NP, p, j);
              store_slices<B_TILE>(xb + o, v[u].x);
              store_slices<B_TILE>(xb + o + NP * 128, v[u].y);
            }
          } else if (j < n_l) {
            const double sc = pinv[p] * 0x1p-24;
            stage_out[j * (NP + 1) + p] = make_double2(v[u].x * sc, v[u].y * sc);
          }
        }
        if (NP == 32 && ykeep) {
          // two points are 32 bytes: one store where the row starts on them (ten runs, N_l 97: second half
          // 172 -> 164 us; with two M tiles the same form costs 4 %, in registers, and the points are
          // stored one by one above)
          const double s0 = pinv[p0] * 0x1p-24, s1 = pinv[p0 + 1] * 0x1p-24;
          if (!(g.n_r & 1) && r0 + p0 + 1 < g.n_r) {
            asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(ykeep + p0), "d"(v[0].x * s0), "d"(v[0].y * s0),
                         "d"(v[1].x * s1), "d"(v[1].y * s1)
                         : "memory");
          } else {
            if (r0 + p0 < g.n_r) ykeep[p0] = make_double2(v[0].x * s0, v[0].y * s0);
            if (r0 + p0 + 1 < g.n_r) ykeep[p0 + 1] = make_double2(v[1].x * s1, v[1].y * s1);
          }
        }
        if (c + 1 < A8_PTS / CH) tready();
      }
      tc_fence_before();
      if (!last) {
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&xb_bar);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    if (threadIdx.x == 0) atomicOr(g.status, ST_TC_TIMEOUT);
  } else {
    // the kept vectors serve the first half of the next step (the step counter advances once
    // per step, after this kernel)
    if (keep_theta && blockIdx.x == 0 && threadIdx.x == 0) *g.yth_step = step_raw + 2;
    const double2* xs = reinterpret_cast<const double2*>(smem);
    // the observables' thread layout and its coefficients, requested before the store
    const int lw = (n_l + 31) & ~31, parts = A8_THREADS / lw;     // N_l <= 220
    const int part = threadIdx.x / lw, lo = threadIdx.x - part * lw;
    double c_u = 0.0, c_d = 0.0;
    if (SECOND_HALF && part < parts && lo < n_l) {
      if (lo + 1 < n_l) c_u = g.coef[((size_t)CF_CU * g.n_m + m) * n_l + lo];
      if (lo > m) c_d = g.coef[((size_t)CF_CD * g.n_m + m) * n_l + lo];
    }
    for (int idx = threadIdx.x; idx < n_l * NP; idx += A8_THREADS) {
      const int l = idx / NP, p = idx - l * NP, r = r0 + p;
      if (r < g.n_r) xout[((size_t)l * g.n_cols + col) * g.n_r + r] = xs[l * (NP + 1) + p];
    }
    if (SECOND_HALF) {
      // FP64 dipole and acceleration partial sums and density multipoles of the new orbitals, from
      // the staged tile, with the coefficient rows of this m staged after it.
      constexpr int LG = 32 / NP;        // lane groups per warp: lane = (point, l-loop group)
      constexpr int NG = A8_DEN_WARPS * LG;   // groups that stride the density's l loops
      double* rows = reinterpret_cast<double*>(smem + (((size_t)n_l * (NP + 1) * 16 + 255) & ~(size_t)255));
      double* red = rows + ((COEF_N * n_l + 1) & ~1);       // [NG][N_DEN][NP] (and the observables' shares), 16-byte aligned
      const int n_den = g.n_den > 0 ? g.n_den : 1;   // L = 0 is always needed for the norm
      if (n_den > 1)
        for (int i = threadIdx.x; i < COEF_N * n_l; i += A8_THREADS) {
          const int c = i / n_l, l = i - c * n_l;
          rows[i] = g.coef[((size_t)c * g.n_m + m) * n_l + l];
        }
      // dipole and acceleration: `parts` threads per l, each over its share of the CTA's NP radii, then
      // the shares added in order (one partial per (l, NP radii))
      double4* ored = reinterpret_cast<double4*>(red);      // [parts][lw], parts lw <= A8_THREADS
      double4 osum = make_double4(0.0, 0.0, 0.0, 0.0);
      if (part < parts && lo < n_l && lo >= m) {
        // the first row has no lower, the last no upper neighbour
        const bool has_u = lo + 1 < n_l, has_d = lo > m;
        const double2* xl_p = xs + lo * (NP + 1);
        for (int p = part * NP / parts; p < (part + 1) * NP / parts; ++p) {
          const double2 xl = xl_p[p];
          const double2 xu = has_u ? xl_p[p + NP + 1] : make_double2(0.0, 0.0);
          const double2 xd = has_d ? xl_p[p - NP - 1] : make_double2(0.0, 0.0);
          const double zx = c_u * xu.x + c_d * xd.x, zy = c_u * xu.y + c_d * xd.y;
          const double px = xl.x * zx + xl.y * zy, py = xl.x * zy - xl.y * zx;     // conj(x_l) . z
          osum.x = fma(prr[0][p], px, osum.x);
          osum.y = fma(prr[0][p], py, osum.y);
          osum.z = fma(prr[1][p], px, osum.z);
          osum.w = fma(prr[1][p], py, osum.w);
        }
      }
      if (parts > 1) {
        if (part < parts) ored[part * lw + lo] = osum;
        __syncthreads();
        if (part == 0)
          for (int q = 1; q < parts; ++q) {
            const double4 v = ored[q * lw + lo];
            osum.x += v.x; osum.y += v.y; osum.z += v.z; osum.w += v.w;
          }
      }
      if (part == 0 && lo < n_l) g.obs[((size_t)col * n_l + lo) * g.n_tiles + r0 / NP] = osum;
      if (parts > 1) __syncthreads();         // the shares' memory is the density's next
      // density multipoles: every lane works (point lane % NP), the literal l loops strided over the
      // NG lane groups, then the groups summed in order
      const int pt = lane % NP, gi = warp * LG + lane / NP;
      double d[N_DEN] = {0.0, 0.0, 0.0, 0.0};
      if (warp < A8_DEN_WARPS) {
        density_partials<double2, NP + 1>(n_den, m, n_l, xs, pt, rows, gi, NG, d);
#pragma unroll
        for (int L = 0; L < N_DEN; ++L) red[(gi * N_DEN + L) * NP + pt] = d[L];
      }
      __syncthreads();
      if (threadIdx.x < n_den * NP) {
        const int L = threadIdx.x / NP, pp = threadIdx.x - L * NP, rl = r0 + pp;
        double sum = 0.0;
        for (int w = 0; w < NG; ++w) sum += red[(w * N_DEN + L) * NP + pp];
        if (rl < g.n_r) g.dens[((size_t)col * N_DEN + L) * g.n_r + rl] = sum;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (abort_flag) {
      // the lane that issued the products commits them (elect.sync gives the same one every time)
      tc_commit_if(elect_one(), &drain_bar);
      if (lane == 0) mbar_drain(&drain_bar, 0);
    }
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, A8_TMEM_COLS);
  }
}

// Radial B operand of one (l, orbital column) row: exponent f with max(|Re|, |Im|) 2^f in
// [63.75, 127.5) over the row, then Xr, Xi, -Xi as four slices each ([l][column tile][k block][12][bn][32]).
// A thread owns quads of four consecutive radii (one 32-bit store per plane).  QUADS > 0: the row fits
// QUADS quads per thread, which stay in registers between the maximum and the slices; every load is
// issued at once and the row is read once.  QUADS = 0: any length, read twice.  873 rows of 600 radii
// (one argon run) and 30429 of 1000 (21 runs): the first half with them 22.5 -> 21.6 and 910 -> 864 us.
constexpr int SX_THREADS = 128;
template <int QUADS>
__global__ void __launch_bounds__(SX_THREADS)
k_slice_x(const double2* __restrict__ x, int n_r, int n_cols, int cols_pad, int bn, int k_pad, int8_t* __restrict__ X,
          int* __restrict__ xexp) {
  const int row = blockIdx.x;                  // l * n_cols + col
  const int l = row / n_cols, col = row - l * n_cols;
  const double2* xr = x + (size_t)row * n_r;
  constexpr int Q = QUADS > 0 ? QUADS : 1;
  double2 v[Q][4];
  double mx = 0.0;
  if constexpr (QUADS > 0) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = 4 * (threadIdx.x + q * SX_THREADS) + u;
        v[q][u] = r < n_r ? xr[r] : make_double2(0.0, 0.0);
      }
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int u = 0; u < 4; ++u) mx = fmax(mx, fmax(fabs(v[q][u].x), fabs(v[q][u].y)));
  } else {
    for (int r = threadIdx.x; r < n_r; r += SX_THREADS) {
      const double2 w = xr[r];
      mx = fmax(mx, fmax(fabs(w.x), fabs(w.y)));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  __shared__ double wm[SX_THREADS / 32];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = wm[0];
#pragma unroll
  for (int w = 1; w < SX_THREADS / 32; ++w) mx = fmax(mx, wm[w]);
  const int f = row_exponent(mx);
  if (threadIdx.x == 0) xexp[(size_t)l * cols_pad + col] = f;
  const double sc = pow2i(f);
  // stage (l, column tile, k block): 12 planes of [columns of the tile][32 bytes]
  const int cols16 = (n_cols + 15) & ~15;
  const int nt = col / bn, row_in = col - nt * bn, plane = min(bn, cols16 - nt * bn) * 32;
  int8_t* xt = X + ((size_t)l * cols16 + nt * bn) * (k_pad / 32) * (R8_X_PLANES * 32);
  auto put = [&](int r4, const double2 (&w)[4]) {
    uint32_t pr[I8_SLICES], pi[I8_SLICES], pn[I8_SLICES], wr[4], wi[4], wn[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      // -Xi is sliced from -x itself: negating a digit -128 would not fit an int8
      wr[u] = slice_word(w[u].x * sc * 16777216.0);
      wi[u] = slice_word(w[u].y * sc * 16777216.0);
      wn[u] = slice_word(-w[u].y * sc * 16777216.0);
    }
    plane_words(wr[0], wr[1], wr[2], wr[3], pr);
    plane_words(wi[0], wi[1], wi[2], wi[3], pi);
    plane_words(wn[0], wn[1], wn[2], wn[3], pn);
    int8_t* b = xt + (size_t)(r4 >> 5) * (R8_X_PLANES * plane) + r8_row_off(row_in, r4 & 31);
#pragma unroll
    for (int qq = 0; qq < I8_SLICES; ++qq) {
      reinterpret_cast<uint32_t*>(b + qq * plane)[0] = pr[qq];
      reinterpret_cast<uint32_t*>(b + (I8_SLICES + qq) * plane)[0] = pi[qq];
      reinterpret_cast<uint32_t*>(b + (2 * I8_SLICES + qq) * plane)[0] = pn[qq];
    }
  };
  if constexpr (QUADS > 0) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int r4 = 4 * (threadIdx.x + q * SX_THREADS);
      if (r4 < n_r) put(r4, v[q]);
    }
  } else {
    for (int r4 = 4 * threadIdx.x; r4 < n_r; r4 += 4 * SX_THREADS) {
#pragma unroll
      for (int u = 0; u < 4; ++u) v[0][u] = r4 + u < n_r ? xr[r4 + u] : make_double2(0.0, 0.0);
      put(r4, v[0]);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------

template <int BN>
static size_t r8_smem(int stages) { return (size_t)stages * R8Tile<BN>::STAGE + 1024; }

// Columns per tile: the narrowest that takes them all, else 64 (fewest reads of W), but 32 where 64 would
// leave a second tile of 32 or fewer: the 32-column tile has two accumulator buffers, so its epilogue runs
// under the next tile's products (90 columns on 600 radii: 126 against 137 us; 72 on 700: 193 against 199;
// 108 on 900: 556 against 443, 117 on 800: 384 against 348, 189 on 1000: 1011 against 871).
static int r8_bn(int n_cols) { return n_cols <= 16 ? 16 : n_cols <= 32 || (n_cols > 64 && n_cols <= 96) ? 32 : 64; }

static int r8_stages(int bn) {
  const int stage = R8_W_PLANES * R8_BM * R8_BK + R8_X_PLANES * bn * R8_BK;
  int s = (200 * 1024) / stage;
  return s > 8 ? 8 : (s < 2 ? 2 : s);
}

template <int NP>
static size_t a8_smem(int k_atoms, int stages) {
  return (size_t)I8_SLICES * k_atoms * (2 * NP * 128) + (size_t)stages * A8_A_TILE + 1024;
}

#define I8_CK(call)                                                      \
  do {                                                                   \
    cudaError_t e_ = (call);                                             \
    if (e_ != cudaSuccess) {                                             \
      err = std::string(#call) + ": " + cudaGetErrorString(e_);          \
      return GGB_ERR_CUDA;                                               \
    }                                                                    \
  } while (0)

// the W planes and row exponents of these propagators, into the buffers of int8_prepare (legacy stream)
void int8_slice_w(MixedGroup& mg, const GroupArgs& a, const double2* W_fp64) {
  const I8Group& q = mg.i8;
  const int n_r = a.n_r, n_l = a.n_l, rows8 = (n_r + 7) & ~7;
  k_w_rowmax<<<dim3((mg.rows_pad + 127) / 128, n_l), 128>>>(W_fp64, q.wexp, n_r, mg.rows_pad);
  const dim3 tb(32, 8), tg((mg.rows_pad + 31) / 32, (mg.k_pad + 31) / 32, n_l);
  for (int v = 0; v < I8_W_VARIANTS; ++v)
    k_slice_w_i8<<<tg, tb>>>(W_fp64, q.wexp, q.W + q.w_variant * v, n_r, rows8, mg.rows_pad, mg.k_pad, v, I8_W_VARIANTS);
}

int int8_prepare(MixedGroup& mg, GroupArgs& a, const double2* W_fp64, int n_mats, std::string& err) {
  const int n_r = a.n_r, n_l = a.n_l;
  I8Group& q = mg.i8;
  q.bn = q.tune_bn > 0 ? q.tune_bn : r8_bn(a.n_cols);
  q.cols_pad = ((a.n_cols + q.bn - 1) / q.bn) * q.bn;
  q.stages = r8_stages(q.bn);
  if (q.tune_stages > 0) q.stages = std::min(q.tune_stages, q.stages);
  // W planes and row exponents
  const int rows8 = (n_r + 7) & ~7;
  const size_t nw = (size_t)n_l * R8_W_PLANES * rows8 * mg.k_pad;    // one variant
  q.w_variant = nw;
  I8_CK(cudaMalloc(&q.W, nw * I8_W_VARIANTS));
  I8_CK(cudaMalloc(&q.wexp, (size_t)n_l * mg.rows_pad * sizeof(int)));
  int8_slice_w(mg, a, W_fp64);
  I8_CK(cudaGetLastError());
  // radial B operand planes
  const size_t nx = (size_t)n_l * R8_X_PLANES * q.cols_pad * mg.k_pad;
  I8_CK(cudaMalloc(&q.X, nx));
  I8_CK(cudaMemset(q.X, 0, nx));
  I8_CK(cudaMalloc(&q.xexp, (size_t)n_l * q.cols_pad * sizeof(int)));
  I8_CK(cudaMemset(q.xexp, 0, (size_t)n_l * q.cols_pad * sizeof(int)));
  // angular chain: S^T slices
  q.a_m_tiles = (n_l + 127) / 128;
  q.a_k_atoms = (n_l + A8_KATOM - 1) / A8_KATOM;
  if (q.a_m_tiles > 2) {
    err = "N_l > 256 is not supported by the int8 angular chain";
    return GGB_ERR_ARG;
  }
  // two CTAs per SM: 256 TMEM columns each (NP points x {Re, Im} x 4 accumulators x M tiles) and
  // at most ~110 KB of shared memory each
  q.np = q.a_m_tiles == 1 ? 32 : 16;     // the kernel takes k_atoms = m_tiles = (NP == 32 ? 1 : 2)
  q.a_stages = I8_SLICES;   // the MMA issue loop relies on stage = slice plane
  q.a_smem = q.np == 32 ? a8_smem<32>(q.a_k_atoms, q.a_stages) : a8_smem<16>(q.a_k_atoms, q.a_stages);
  // FP64 staging of the last product, [N_l][NP + 1], over the operand planes and stage buffers
  // the second half's tail: output tile, coefficient rows and the multipoles' warp partials
  const size_t tail = (((size_t)n_l * (q.np + 1) * 16 + 255) & ~(size_t)255) + ((size_t)COEF_N * n_l + 1) * 8 +
                      (size_t)A8_THREADS * 4 * 8 + 2 * (size_t)q.np * 8;
  if (tail > q.a_smem - 1024 || q.a_smem > 110 * 1024) {
    err = "int8 angular chain: shared memory";
    return GGB_ERR_ARG;
  }
  if (a.obs_seg != q.np) {
    // the second half writes one observables partial per CTA, so the group's partials are NP radii
    err = "int8 angular chain: observables partials do not match its tile";
    return GGB_ERR_STATE;
  }
  const int rows = 128 * q.a_m_tiles;
  q.a_rows = rows;
  const int n_mm = n_mats * a.n_m;
  const StGeom geo = StGeom::of(n_l);
  const size_t nst = (size_t)n_mm * geo.bytes();    // one variant
  q.n_mats = n_mats;
  I8_CK(cudaMalloc(&q.St, nst * I8_S_VARIANTS));
  I8_CK(cudaMalloc(&q.sexp, (size_t)n_mm * rows * sizeof(int)));
  for (int v = 0; v < I8_S_VARIANTS; ++v)
    k_build_st_i8<<<n_mm * rows, 256>>>(a.mats, q.St + nst * v, q.sexp, n_mm, a.n_m, n_l, a.ldS, rows, geo, v,
                                        I8_S_VARIANTS);
  I8_CK(cudaGetLastError());
  // basis reuse of the theta form (one phase op and one closing product per half); the angular
  // products on the FP64 kernel keep the full chain
  if (q.theta_reuse && a.theta && !mg.angular_fp64 && a.chain[0].n_ops == 2 && a.chain[1].n_ops == 2) {
    I8_CK(cudaMalloc(&q.yth, (size_t)n_l * a.n_cols * n_r * sizeof(double2)));
  }
  int dev = 0, optin = 0, sms = 0;
  I8_CK(cudaGetDevice(&dev));
  I8_CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  I8_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  q.ctas = sms;
  switch (q.bn) {
    case 16: I8_CK(set_max_dynamic_smem((const void*)k_radial_i8<16>, optin)); q.smem = r8_smem<16>(q.stages); break;
    case 32: I8_CK(set_max_dynamic_smem((const void*)k_radial_i8<32>, optin)); q.smem = r8_smem<32>(q.stages); break;
    default: I8_CK(set_max_dynamic_smem((const void*)k_radial_i8<64>, optin)); q.smem = r8_smem<64>(q.stages); break;
  }
  // the two halves that this group launches (a kernel's first mention in a process loads it)
#define GGB_A8(NP, TH)                                                              \
  do {                                                                              \
    I8_CK(set_max_dynamic_smem((const void*)k_angular_i8<NP, false, TH>, optin));   \
    I8_CK(set_max_dynamic_smem((const void*)k_angular_i8<NP, true, TH>, optin));    \
  } while (0)
  if (!mg.angular_fp64) {
    if (q.np == 32) { if (a.theta) GGB_A8(32, true); else GGB_A8(32, false); }
    else { if (a.theta) GGB_A8(16, true); else GGB_A8(16, false); }
  }
#undef GGB_A8
  I8_CK(cudaDeviceSynchronize());
  return GGB_OK;
}

void int8_radial(MixedGroup& mg, const GroupArgs& a, cudaStream_t s) {
  const I8Group& q = mg.i8;
  const int tiles = ((a.n_r + R8_BM - 1) / R8_BM) * ((a.n_cols + q.bn - 1) / q.bn) * a.n_l;
  const dim3 g(tiles < q.ctas ? tiles : q.ctas);
  const int nkb = mg.k_pad / R8_BK;
  switch (q.bn) {
    case 16: k_radial_i8<16><<<g, R8_THREADS, q.smem, s>>>(q.W, q.w_variant, q.X, q.wexp, q.xexp, a.n_r, mg.rows_pad, a.n_cols, q.cols_pad, a.n_l, nkb, q.stages, a.step, I8_W_VARIANTS, mg.Yd, a.status); break;
    case 32: k_radial_i8<32><<<g, R8_THREADS, q.smem, s>>>(q.W, q.w_variant, q.X, q.wexp, q.xexp, a.n_r, mg.rows_pad, a.n_cols, q.cols_pad, a.n_l, nkb, q.stages, a.step, I8_W_VARIANTS, mg.Yd, a.status); break;
    default: k_radial_i8<64><<<g, R8_THREADS, q.smem, s>>>(q.W, q.w_variant, q.X, q.wexp, q.xexp, a.n_r, mg.rows_pad, a.n_cols, q.cols_pad, a.n_l, nkb, q.stages, a.step, I8_W_VARIANTS, mg.Yd, a.status); break;
  }
}

void int8_angular(MixedGroup& mg, const GroupArgs& a, int half, const double2* xin, double2* xout, cudaStream_t s) {
  const I8Group& q = mg.i8;
  Ang8Args t;
  t.k_atoms = q.a_k_atoms;
  t.m_tiles = q.a_m_tiles;
  t.k_steps = (a.n_l + 31) / 32;
  t.stages = q.a_stages;
  t.St = q.St;
  t.geo = StGeom::of(a.n_l);
  t.one_round = q.a_m_tiles == 2 && st_one_round(t.geo);
  t.sexp = q.sexp;
  t.rows = q.a_rows;
  t.sms = q.ctas;
  t.n_mats = q.n_mats;
  t.n_var = I8_S_VARIANTS;
  t.yth = q.yth;
  const dim3 grid(a.n_cols * ((a.n_r + q.np - 1) / q.np));
#define GGB_A8(NP, SH, TH) k_angular_i8<NP, SH, TH><<<grid, A8_THREADS, q.a_smem, s>>>(a, t, xin, xout)
  if (q.np == 32) {
    if (half == 0) { if (a.theta) GGB_A8(32, false, true); else GGB_A8(32, false, false); }
    else { if (a.theta) GGB_A8(32, true, true); else GGB_A8(32, true, false); }
  } else {
    if (half == 0) { if (a.theta) GGB_A8(16, false, true); else GGB_A8(16, false, false); }
    else { if (a.theta) GGB_A8(16, true, true); else GGB_A8(16, true, false); }
  }
#undef GGB_A8
}

void int8_slice_x(MixedGroup& mg, const GroupArgs& a, const double2* x, cudaStream_t s) {
  const I8Group& q = mg.i8;
#define GGB_SX(Q) k_slice_x<Q><<<a.n_l * a.n_cols, SX_THREADS, 0, s>>>(x, a.n_r, a.n_cols, q.cols_pad, q.bn, mg.k_pad, q.X, q.xexp)
  if (a.n_r <= 4 * SX_THREADS) GGB_SX(1);
  else if (a.n_r <= 8 * SX_THREADS) GGB_SX(2);
  else GGB_SX(0);
#undef GGB_SX
}

void int8_release(I8Group& q) {
  cudaFree(q.W);
  cudaFree(q.wexp);
  cudaFree(q.X);
  cudaFree(q.xexp);
  cudaFree(q.St);
  cudaFree(q.sexp);
  cudaFree(q.yth);
  q = I8Group();
}

}  // namespace ggb
