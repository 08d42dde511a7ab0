// Mixed-precision solver of the smoothed TPS subdomain systems.
//
// Upstream (calcul/interpolate/thin_plate_spline.py:168-216,
// thin_plate_spline_subdom.py:236-280) solves [[K + lam I, P], [P^T, 0]] [w; a] =
// [u; 0] with LAPACK gesv in FP64, for x and y and again after each outlier
// replacement.  That saddle-point matrix has condition numbers ~1e13-1e15, but its
// null-space form is benign: with P = Q [R; 0] (Householder, Q = H0 H1 H2),
// w = Q2 z and
//     B z = g = Q2^T u,   B = Q2^T (K + lam I) Q2   (SPD, cond ~1e4 for lam > 0),
//     a = R^-1 (Q1^T u - C z),  C = Q1^T (K + lam I) Q2,   smoothed = u - lam w.
// On this GPU FP32 runs 73x faster than FP64.  B and C are projected once with the
// compact WY form of Q; the projection cancels the large affine part of K, so it
// needs more than FP32: Y = A V and B are computed in double-float (pairs of floats,
// error-free products and sums on the FP32 pipe, ~48 bits), the O(n) parts and C in
// FP64.  B is kept as (hi, lo) pairs and its high terms are factorised (tiled Cholesky
// on the tensor cores, FP16 pairs with FP32 accumulation).  z is refined in double-float:
// rho = g - B z on the FP32 pipe (error-free products and sums), then a solve with the
// factor for the correction.
// Each sweep contracts the error ~1e3-1e4 times; refinement stops when the
// predicted remaining error is below 1e-10 of z, or when it stagnates (then it must
// be below 1e-9).  A subdomain that does not converge (or whose P has rank < 3, or
// whose Cholesky meets a non-positive pivot) is flagged and re-solved by the FP64
// LU kernel (k_tps_solve).
//
// K entries come from a table of phi(r^2) = r^2 log(r^2) / 2 indexed by 4 r^2,
// exact for window centres on the half-integer lattice (the integer window shifts
// put every PIV vector there); other distances use log() directly.  When a
// subdomain's centres lie on a grid of the lattice, the block keeps the (hi, lo)
// values of every grid offset in shared memory (the same table entries).
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <climits>
#include <cmath>

#include "fi_common.cuh"
#include "fi_df.cuh"
#include "fi_lattice.cuh"

namespace fi {

// ------------------------------------------------------------------ phi
__device__ __forceinline__ double phi_direct(double r2) {
  if (r2 == 0.0) return 0.0;
  return __ddiv_rn(__dmul_rn(r2, log(r2)), 2.0);
}

// phi(r^2) for the centre pair (a, b); table lookup when 4 r^2 is an integer in range.
__device__ __forceinline__ double phi_pair(double xa, double ya, double xb, double yb,
                                           const double* table, int64_t tsize) {
  const double dy = __dsub_rn(ya, yb), dx = __dsub_rn(xa, xb);
  const double r2 = __dadd_rn(__dmul_rn(dy, dy), __dmul_rn(dx, dx));
  const double q = 4.0 * r2;
  if (table != nullptr && q < (double)tsize) {
    const int64_t k = (int64_t)q;
    if ((double)k == q) return __ldg(table + k);
  }
  return phi_direct(r2);
}

__global__ void k_phi_table(double* table, int64_t count) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count;
       k += (int64_t)gridDim.x * blockDim.x)
    table[k] = phi_direct((double)k * 0.25);
}

// The same values as (hi, lo) float pairs (double-float evaluation).
__global__ void k_phi_table2(float2* table, int64_t count) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count;
       k += (int64_t)gridDim.x * blockDim.x)
    table[k] = df_split(phi_direct((double)k * 0.25));
}

// ------------------------------------------------------------------ block helpers
// FP64 is narrow on this GPU (an instruction holds its scheduler's FP64 unit for ~70
// cycles), so the block-wide steps below keep FP64 additions, and scalar FP64 work on
// every thread, to a minimum.

// Sums of K values over the block, returned to every thread in out[K] (shared).  The
// warps reduce-scatter: with P = K rounded up to a power of two, P - 1 + 5 - log2 P
// additions instead of 5 K.  sh: BLOCK_SUMS doubles.
constexpr int BLOCK_SUMS = 16 * 16;
template <int NT, int K>
__device__ __forceinline__ void block_sums(const double (&v)[K], double* sh, double* out) {
  constexpr int NW = NT / 32;
  constexpr int P = K <= 1 ? 1 : K <= 2 ? 2 : K <= 4 ? 4 : K <= 8 ? 8 : 16;
  static_assert(K <= 16 && NW <= 16, "block_sums: sh");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double w[P];
#pragma unroll
  for (int k = 0; k < P; ++k) w[k] = k < K ? v[k < K ? k : 0] : 0.0;
#pragma unroll
  for (int st = 0; st < 5; ++st) {
    const int o = 16 >> st, len = P >> (st + 1);
    if (len > 0) {
      const bool up = lane & o;
#pragma unroll
      for (int k = 0; k < len; ++k) {
        const double send = up ? w[k] : w[k + len], keep = up ? w[k + len] : w[k];
        w[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    } else {
      w[0] += __shfl_xor_sync(0xffffffffu, w[0], o);
    }
  }
  constexpr int PARTS = 32 / P;  // lanes that end with the same value
  if (lane % PARTS == 0) sh[wid * P + lane / PARTS] = w[0];
  __syncthreads();
  if (wid == 0) {
    const int idx = lane % P;
    double t = 0.0;
    for (int q = lane / P; q < NW; q += PARTS) t += sh[q * P + idx];
#pragma unroll
    for (int o = P; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane < K) out[lane] = t;
  }
  __syncthreads();
}

// Largest of a and of b (non-negative floats, as their bits: a NaN is the largest) over
// the block.
template <int NT>
__device__ __forceinline__ float2 block_max2(float a, float b, double* sh) {
  constexpr int NW = NT / 32;
  unsigned* u = reinterpret_cast<unsigned*>(sh);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned full = 0xffffffffu;
  const unsigned wa = __reduce_max_sync(full, __float_as_uint(a));
  const unsigned wb = __reduce_max_sync(full, __float_as_uint(b));
  if (lane == 0) {
    u[wid] = wa;
    u[NW + wid] = wb;
  }
  __syncthreads();
  const unsigned ra = __reduce_max_sync(full, lane < NW ? u[lane] : 0u);
  const unsigned rb = __reduce_max_sync(full, lane < NW ? u[NW + lane] : 0u);
  __syncthreads();
  return make_float2(__uint_as_float(ra), __uint_as_float(rb));
}

// Largest of a non-negative double over the warp, by its bits.
__device__ __forceinline__ double warp_max_pos(double v) {
  const unsigned full = 0xffffffffu;
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(full, hi);
  const unsigned ml = __reduce_max_sync(full, hi == mh ? lo : 0u);
  return __hiloint2double((int)mh, (int)ml);
}
template <int NT>
__device__ __forceinline__ double block_max_pos(double v, double* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_max_pos(v);
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  v = warp_max_pos(lane < NT / 32 ? sh[lane] : 0.0);
  __syncthreads();
  return v;
}

// bytes of a block's panel: the chunk sums of Y, the projection's per-warp tiles, then
// the factorisation's staging and the tiles of small subdomains
__host__ __device__ constexpr size_t panel_bytes(int warps) { return (size_t)(2 + warps) * 4608; }

// Start moving [p, p + bytes) from memory into L2 without waiting for it (bulk
// prefetch by the copy engine; p 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// rho = g - B z for two right-hand sides, in double-float; B (m x m, symmetric, both
// triangles, column-major, leading dimension ld, a multiple of 4; 32-byte aligned)
// holds (hi, lo) pairs, read with the streaming hint (B is twice the FP32 factor,
// which should stay in L2).  Each warp takes four columns at a time (one row per
// lane), then reduce-scatters its eight sums over the warp.  B is streamed from
// memory: each warp has the copy engine prefetch its next two column groups into L2
// (contiguous, 32 ld bytes per column) while it works on the current one, so that
// its loads wait on L2 rather than on memory.  rho is rounded to float.
template <int NT>
__device__ __noinline__ void residual_df2(const float2* __restrict__ B, int m, int ld, const float2* zx,
                             const float2* zy, const float2* gx, const float2* gy, float* rx,
                             float* ry) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned full = 0xffffffffu;
  auto prefetch_group = [&](int c) {
    if (lane == 0 && c < m)
      prefetch_l2(B + (int64_t)c * ld, (unsigned)(min(4, m - c) * ld * sizeof(float2)));
  };
  prefetch_group(4 * wid);
  prefetch_group(4 * wid + 4 * NW);
  for (int c0 = 4 * wid; c0 < m; c0 += 4 * NW) {
    prefetch_group(c0 + 8 * NW);
    // column q: x sums in lane .x, y sums in lane .y of the pairs (packed FP32x2)
    float2 H[4], Lo[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) H[q] = Lo[q] = make_float2(0.f, 0.f);
    const float2* col = B + (int64_t)c0 * ld;
    const int nc = min(4, m - c0);
    // two rows per lane and load (16 bytes: twice the bytes in flight per load); ld
    // is a multiple of 4, so row r + 1 < ld; the padding rows past m are masked
#pragma unroll 2
    for (int r = 2 * lane; r < m; r += 64) {
      const float4 a = *reinterpret_cast<const float4*>(zx + r);
      const float4 b = *reinterpret_cast<const float4*>(zy + r);
      const float2 zh0 = make_float2(a.x, b.x), zl0 = make_float2(a.y, b.y);
      const float2 zh1 = make_float2(a.z, b.z), zl1 = make_float2(a.w, b.w);
      const bool two = r + 1 < m;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q < nc) v = __ldcs(reinterpret_cast<const float4*>(col + (int64_t)q * ld + r));
        if (!two) v.z = v.w = 0.f;
        df_mac_x2(make_float2(v.x, v.y), zh0, zl0, H[q], Lo[q]);
        df_mac_x2(make_float2(v.z, v.w), zh1, zl1, H[q], Lo[q]);
      }
    }
    float h[8], l[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      h[q] = H[q].x;
      l[q] = Lo[q].x;
      h[4 + q] = H[q].y;
      l[4 + q] = Lo[q].y;
    }
    // reduce-scatter: lane ends with value 4 b4 + 2 b3 + b2 (b_k = bit k of lane)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool up = lane & 16;
      const float sh_ = up ? h[k] : h[k + 4], sl_ = up ? l[k] : l[k + 4];
      const float2 keep = up ? make_float2(h[k + 4], l[k + 4]) : make_float2(h[k], l[k]);
      const float2 got = make_float2(__shfl_xor_sync(full, sh_, 16), __shfl_xor_sync(full, sl_, 16));
      const float2 s = df_add(keep, got);
      h[k] = s.x;
      l[k] = s.y;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const bool up = lane & 8;
      const float sh_ = up ? h[k] : h[k + 2], sl_ = up ? l[k] : l[k + 2];
      const float2 keep = up ? make_float2(h[k + 2], l[k + 2]) : make_float2(h[k], l[k]);
      const float2 got = make_float2(__shfl_xor_sync(full, sh_, 8), __shfl_xor_sync(full, sl_, 8));
      const float2 s = df_add(keep, got);
      h[k] = s.x;
      l[k] = s.y;
    }
    {
      const bool up = lane & 4;
      const float sh_ = up ? h[0] : h[1], sl_ = up ? l[0] : l[1];
      const float2 keep = up ? make_float2(h[1], l[1]) : make_float2(h[0], l[0]);
      const float2 got = make_float2(__shfl_xor_sync(full, sh_, 4), __shfl_xor_sync(full, sl_, 4));
      const float2 s = df_add(keep, got);
      h[0] = s.x;
      l[0] = s.y;
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
      const float2 got = make_float2(__shfl_xor_sync(full, h[0], o), __shfl_xor_sync(full, l[0], o));
      const float2 s = df_add(make_float2(h[0], l[0]), got);
      h[0] = s.x;
      l[0] = s.y;
    }
    if ((lane & 3) == 0) {
      const int idx = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
      const int c = c0 + (idx & 3);
      if (c < m) {
        const float2 g = (idx >> 2) ? gy[c] : gx[c];
        const float2 d = df_add(g, make_float2(-h[0], -l[0]));
        ((idx >> 2) ? ry : rx)[c] = __fadd_rn(d.x, d.y);
      }
    }
  }
  __syncthreads();
}

// ---- Cholesky preconditioner on the tensor cores ------------------------------------
// The factor of D B D (D: powers of two that bring the diagonal into [1, 4)) by 32 x 32
// tiles, each kept as two FP16 terms hi + lo (22 significant bits, like the TF32 pairs of
// a 3xTF32 product; the scaling bounds every entry of L by 2, so the terms' absolute
// rounding is that of FP32 relative to the row's norm).  Products take three terms
// (lo hi + hi lo + hi hi; Ootomo and Yokota, "Recovering single precision accuracy from
// Tensor Cores while surpassing the FP32 theoretical peak performance", IJHPCA 2022) with
// FP32 accumulation.  The factor only preconditions the double-float refinement.
//
// 400 centres, two 8-warp blocks per SM: 195 us against 410 us of a right-looking
// Cholesky with 3xTF32 products on an FP32 matrix in memory (its tile updates loaded and
// stored their target and split both operands every time; the same sweeps to converge).
// The m16n8k16 FP16 MMA issues in 8 cycles, the same as m16n8k8 TF32 at half the depth.
//
// A tile is stored in the register layout of the m16n8k16 A operand: 16-byte element
// (4 t + 2 mt + ks) * 32 + lane (t = 0: hi, 1: lo; mt: 16 rows; ks: 16 columns).  The
// same registers are the B operand of the transposed tile, so every product is
// D += X Y^T of two stored tiles, read by 16-byte loads without a conversion.  The
// diagonal slots hold W_kk = inv(L_kk), so that the columns below a diagonal tile and the
// substitutions are products too.  Tile (i, j), i >= j, is at 256 (i (i + 1) / 2 + j);
// until it is final its slot holds the FP32 accumulator of its owner warp, lane by lane.
constexpr int TILE16 = 256;   // 16-byte elements per tile
constexpr int WS_LD = 34;     // row stride (floats) of the diagonal tile's staging
constexpr size_t CHOL_SMEM = (size_t)(32 * WS_LD + 64) * sizeof(float);
// tiles of subdomains of at most 96 unknowns (6 tiles, 24 KB) stay in shared memory:
// with the padding to 32 they could exceed the (m + 6)^2 floats of the slot in memory
constexpr int SMALL_T = 3;

__device__ __forceinline__ int tile_at(int i, int j) { return TILE16 * (i * (i + 1) / 2 + j); }

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// (x, y) = hi + lo as two packed FP16 pairs
__device__ __forceinline__ void split_f16(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn(x - hf.x, y - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// transpose of an 8 x 8 block of 16-bit elements held one row pair per lane
__device__ __forceinline__ uint32_t trans8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// a stored tile in registers: u[t][mt][ks]
struct Tile16 {
  uint4 u[2][2][2];
  __device__ __forceinline__ void load(const uint4* p, int lane) {
#pragma unroll
    for (int s = 0; s < 8; ++s) u[s >> 2][(s >> 1) & 1][s & 1] = p[32 * s + lane];
  }
  __device__ __forceinline__ void store(uint4* p, int lane) const {
#pragma unroll
    for (int s = 0; s < 8; ++s) p[32 * s + lane] = u[s >> 2][(s >> 1) & 1][s & 1];
  }
  // the tile of the accumulators sign * c (C layout of the m16n8k16 MMA)
  __device__ __forceinline__ void from_acc(const float (&c)[2][4][4], float sign) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        const float(&p)[4] = c[mt][2 * ks];
        const float(&q)[4] = c[mt][2 * ks + 1];
        uint4 &h = u[0][mt][ks], &l = u[1][mt][ks];
        split_f16(sign * p[0], sign * p[1], h.x, l.x);
        split_f16(sign * p[2], sign * p[3], h.y, l.y);
        split_f16(sign * q[0], sign * q[1], h.z, l.z);
        split_f16(sign * q[2], sign * q[3], h.w, l.w);
      }
  }
  // this tile := its transpose
  __device__ __forceinline__ void transpose() {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      uint4 v[2][2];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          const uint4 s = u[t][ks][mt];
          v[mt][ks] = make_uint4(trans8(s.x), trans8(s.z), trans8(s.y), trans8(s.w));
        }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) u[t][mt][ks] = v[mt][ks];
    }
  }
};

// c += X Y^T, three terms
__device__ __forceinline__ void tile_mma(float (&c)[2][4][4], const Tile16& X, const Tile16& Y) {
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int term = 0; term < 3; ++term)  // lo hi, hi lo, hi hi
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const uint4& y = Y.u[term == 1][nt >> 1][ks];
          mma_f16(c[mt][nt], X.u[term == 0][mt][ks], (nt & 1) ? y.y : y.x, (nt & 1) ? y.w : y.z);
        }
}

// c = -(D B D) tile (i, j) (identity past m), from the high terms of B
__device__ __forceinline__ void tile_from_B(float (&c)[2][4][4], const float2* __restrict__ B,
                                            int m, int ld, const float* dsc, int i, int j,
                                            int lane) {
  const int g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = 32 * i + 16 * mt + g + 8 * (e >> 1);
        const int col = 32 * j + 8 * nt + 2 * q + (e & 1);
        float v = (r == col) ? -1.f : 0.f;
        if (r < m && col < m) v = -B[(int64_t)col * ld + r].x * (dsc[r] * dsc[col]);
        c[mt][nt][e] = v;
      }
}

// accumulators <-> a tile slot, each lane its own values
__device__ __forceinline__ void acc_store(uint4* p, const float (&c)[2][4][4], int lane) {
  float4* f = reinterpret_cast<float4*>(p);
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const float(&v)[4] = c[s >> 2][s & 3];
    f[32 * s + lane] = make_float4(v[0], v[1], v[2], v[3]);
  }
}
__device__ __forceinline__ void acc_load(const uint4* p, float (&c)[2][4][4], int lane) {
  const float4* f = reinterpret_cast<const float4*>(p);
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const float4 v = f[32 * s + lane];
    c[s >> 2][s & 3][0] = v.x;
    c[s >> 2][s & 3][1] = v.y;
    c[s >> 2][s & 3][2] = v.z;
    c[s >> 2][s & 3][3] = v.w;
  }
}

// W = inv(L) of the diagonal tile -c = L L^T, by Gauss elimination of [A | I] with one
// column of both halves per lane: step j publishes row j of A (by symmetry the
// multipliers of every row) in shared memory, and each lane takes its multiple off its
// two columns, two rows per packed FMA.  Rows of the eliminated identity over the square
// roots of the pivots are W, staged and stored as a tile at p.  A chain of 32 steps of
// one shared-memory round trip and one reciprocal (a Cholesky of the tile, then its
// inverse, are two chains of shuffles).  Sets *s_flag on a pivot that is not positive.
__device__ __forceinline__ void diag_inverse(const float (&c)[2][4][4], uint4* p, float* ws,
                                             int lane, int* s_flag) {
  const int g = lane >> 2, q = lane & 3;
  float* s = ws + 32 * WS_LD;  // two rows of 32
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        ws[(16 * mt + g + 8 * (e >> 1)) * WS_LD + 8 * nt + 2 * q + (e & 1)] = -c[mt][nt][e];
  __syncwarp();
  float2 a[16], w[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    a[r] = *reinterpret_cast<const float2*>(ws + lane * WS_LD + 2 * r);
    w[r] = make_float2(2 * r == lane ? 1.f : 0.f, 2 * r + 1 == lane ? 1.f : 0.f);
  }
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    float* sj = s + 32 * (j & 1);
    sj[lane] = (j & 1) ? a[j >> 1].y : a[j >> 1].x;
    __syncwarp();
    const float d = sj[j];
    ok &= d > 0.f;
    const float inv = __fdividef(1.f, d);
    const float fa = -inv * ((j & 1) ? a[j >> 1].y : a[j >> 1].x);
    const float wj = (j & 1) ? w[j >> 1].y : w[j >> 1].x;
    const float fw = -inv * wj;
    if (!(j & 1)) {
      const float l = sj[j + 1];
      a[j >> 1].y = fmaf(l, fa, a[j >> 1].y);
      w[j >> 1].y = fmaf(l, fw, w[j >> 1].y);
      w[j >> 1].x = wj * rsqrtf(d);
    } else {
      w[j >> 1].y = wj * rsqrtf(d);
    }
#pragma unroll
    for (int r = (j >> 1) + 1; r < 16; ++r) {
      const float2 l = *reinterpret_cast<const float2*>(sj + 2 * r);
      a[r] = __ffma2_rn(l, make_float2(fa, fa), a[r]);
      w[r] = __ffma2_rn(l, make_float2(fw, fw), w[r]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    ws[(2 * r) * WS_LD + lane] = w[r].x;
    ws[(2 * r + 1) * WS_LD + lane] = w[r].y;
  }
  if (!__all_sync(0xffffffffu, ok) && lane == 0) *s_flag = 1;
  __syncwarp();
  Tile16 t;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      uint4 &h = t.u[0][mt][ks], &l = t.u[1][mt][ks];
      const float* b = ws + (16 * mt + g) * WS_LD + 16 * ks + 2 * q;
      split_f16(b[0], b[1], h.x, l.x);
      split_f16(b[8 * WS_LD], b[8 * WS_LD + 1], h.y, l.y);
      split_f16(b[8], b[9], h.z, l.z);
      split_f16(b[8 * WS_LD + 8], b[8 * WS_LD + 9], h.w, l.w);
    }
  t.store(p, lane);
  __syncwarp();
}

// The factor of D B D into the tiles LP.  Phase k makes column k: a row's warp takes the
// last term off its accumulator, multiplies by W_kk^T, stores L_ik, takes L_ik L_ik^T off
// its diagonal tile, then accumulates the terms j < k of column k + 1.  Warp 0 has row
// k + 1 and goes on to the inverse of diagonal tile k + 1, the serial chain of the
// factorisation, while the other warps do the bulk; one barrier per phase.  Every
// accumulator stays with the warp that owns its row in that phase.  False on a pivot that
// is not positive.
template <int NT>
__device__ __noinline__ bool chol_factor(const float2* __restrict__ B, int m, int ld, const float* dsc,
                            uint4* LP, float* ws, int* s_flag) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int T = (m + 31) / 32;
  float c[2][4][4];
  if (wid == 0) {
    tile_from_B(c, B, m, ld, dsc, 0, 0, lane);
    diag_inverse(c, LP, ws, lane, s_flag);
  }
  __syncthreads();
  for (int k = 0; k + 1 < T; ++k) {
    for (int i = k + 1 + wid; i < T; i += (wid == 0) ? T : NW - 1) {
      Tile16 X, Y;
      uint4* slot = LP + tile_at(i, k);
      if (k == 0) {
        tile_from_B(c, B, m, ld, dsc, i, 0, lane);
      } else {
        acc_load(slot, c, lane);
        X.load(LP + tile_at(i, k - 1), lane);
        Y.load(LP + tile_at(k, k - 1), lane);
        tile_mma(c, X, Y);
      }
      X.from_acc(c, -1.f);
      Y.load(LP + tile_at(k, k), lane);
#pragma unroll
      for (int e = 0; e < 32; ++e) c[e >> 4][(e >> 2) & 3][e & 3] = 0.f;
      tile_mma(c, X, Y);
      X.from_acc(c, 1.f);
      X.store(slot, lane);
      uint4* dslot = LP + tile_at(i, i);
      if (k == 0)
        tile_from_B(c, B, m, ld, dsc, i, i, lane);
      else
        acc_load(dslot, c, lane);
      tile_mma(c, X, X);
      if (i == k + 1) {
        diag_inverse(c, dslot, ws, lane, s_flag);
      } else {
        acc_store(dslot, c, lane);
        // column k + 1 of this row, terms j < k
        tile_from_B(c, B, m, ld, dsc, i, k + 1, lane);
        for (int j = 0; j < k; ++j) {
          X.load(LP + tile_at(i, j), lane);
          Y.load(LP + tile_at(k + 1, j), lane);
          tile_mma(c, X, Y);
        }
        acc_store(LP + tile_at(i, k + 1), c, lane);
      }
    }
    __syncthreads();
  }
  return *s_flag == 0;
}

// The B operand (K = 32, N = 8) holding the two right-hand sides of block k in its first
// two columns (zeros in the others): b[t][ks] = (b0, b1).
__device__ __forceinline__ void rhs_frags(const float* rx, const float* ry, int lane,
                                          uint2 (&b)[2][2]) {
  const int g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    b[0][ks] = b[1][ks] = make_uint2(0u, 0u);
    if (g < 2) {
      const float* v = (g ? ry : rx) + 16 * ks + 2 * q;
      const float2 v0 = *reinterpret_cast<const float2*>(v);
      const float2 v1 = *reinterpret_cast<const float2*>(v + 8);
      split_f16(v0.x, v0.y, b[0][ks].x, b[1][ks].x);
      split_f16(v1.x, v1.y, b[0][ks].y, b[1][ks].y);
    }
  }
}

// d[mt] = rows 16 mt + g and + 8 of X v (columns 2 q, 2 q + 1: the right-hand sides are
// in the lanes q = 0); the three terms in accumulators of their own (chains of two MMAs)
__device__ __forceinline__ void tile_vec(float (&d)[2][4], const Tile16& X,
                                         const uint2 (&b)[2][2]) {
  float t[3][2][4];
#pragma unroll
  for (int e = 0; e < 24; ++e) t[e >> 3][(e >> 2) & 1][e & 3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int term = 0; term < 3; ++term)
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        const uint2& v = b[term == 1][ks];
        mma_f16(t[term][mt], X.u[term == 0][mt][ks], v.x, v.y);
      }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int e = 0; e < 4; ++e) d[mt][e] = (t[0][mt][e] + t[1][mt][e]) + t[2][mt][e];
}

__device__ __forceinline__ void cp_async16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(smem)),
               "l"(g)
               : "memory");
}

// rows of block n of the right-hand sides: minus d, or d
__device__ __forceinline__ void rhs_put(float* rx, float* ry, const float (&d)[2][4],
                                        bool subtract, int lane) {
  if ((lane & 3) == 0) {
    float* x = rx + (lane >> 2);
    float* y = ry + (lane >> 2);
#pragma unroll
    for (int h = 0; h < 4; ++h) {  // rows g + 8 h
      const float vx = d[h >> 1][2 * (h & 1)], vy = d[h >> 1][2 * (h & 1) + 1];
      x[8 * h] = subtract ? x[8 * h] - vx : vx;
      y[8 * h] = subtract ? y[8 * h] - vy : vy;
    }
  }
  __syncwarp();
}

// Block substitution over the tiles: forward (L y = r) or backward (L^T x = y).  Warp 0
// runs the serial chain: it takes block n - 1's solution off block n and multiplies by
// the inverse of the diagonal tile; its two tiles per step come through a ring of three
// stages in shared memory (asynchronous copies, each lane its own elements).  After the
// barrier that publishes block k's solution the other warps take it off blocks k + 2 and
// on (each block with its warp), their next tile loaded a step ahead.  One barrier per
// step.  ring: null when the tiles are in shared memory themselves.
constexpr int RING_STAGES = 3;
constexpr size_t RING_BYTES = (size_t)RING_STAGES * 2 * TILE16 * sizeof(uint4);
template <int NT, bool BACK>
__device__ __noinline__ void tri_solve(const uint4* LP, int T, float* rx, float* ry,
                                       uint4* ring) {
  constexpr int NO = NT / 32 - 1;  // warps beside the chain's
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // blocks in the order of the substitution: n-th block
  auto blk = [&](int n) { return BACK ? T - 1 - n : n; };
  auto tile_of = [&](int n, int k) {  // the tile coupling block n to block k (k before n)
    return BACK ? tile_at(blk(k), blk(n)) : tile_at(blk(n), blk(k));
  };
  uint2 b[2][2];
  float d[2][4];
  if (wid == 0) {
    auto issue = [&](int n) {
      if (ring != nullptr && n < T) {
        uint4* dst = ring + (n % RING_STAGES) * 2 * TILE16;
        const uint4* w = LP + tile_at(blk(n), blk(n));
#pragma unroll
        for (int e = 0; e < 8; ++e) cp_async16(dst + 32 * e + lane, w + 32 * e + lane);
        if (n > 0) {
          const uint4* x = LP + tile_of(n, n - 1);
#pragma unroll
          for (int e = 0; e < 8; ++e)
            cp_async16(dst + TILE16 + 32 * e + lane, x + 32 * e + lane);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);
    issue(1);
    for (int n = 0; n < T; ++n) {
      issue(n + 2);
      asm volatile("cp.async.wait_group %0;" ::"n"(RING_STAGES - 1) : "memory");
      const uint4* src = ring + (n % RING_STAGES) * 2 * TILE16;
      Tile16 X, W;
      W.load(ring != nullptr ? src : LP + tile_at(blk(n), blk(n)), lane);
      if (BACK) W.transpose();
      float* bx = rx + 32 * blk(n);
      float* by = ry + 32 * blk(n);
      if (n > 0) {
        X.load(ring != nullptr ? src + TILE16 : LP + tile_of(n, n - 1), lane);
        if (BACK) X.transpose();
        __syncthreads();  // block n - 1 is published, the earlier ones are off block n
        tile_vec(d, X, b);
        rhs_put(bx, by, d, true, lane);
      }
      rhs_frags(bx, by, lane, b);
      tile_vec(d, W, b);
      __syncwarp();
      rhs_put(bx, by, d, false, lane);
      rhs_frags(bx, by, lane, b);
    }
    __syncthreads();
  } else {
    // this warp's first block from block n on
    auto first_of = [&](int n) { return n + (wid - 1 - n % NO + NO) % NO; };
    Tile16 X, N;
    int n0 = first_of(2);
    if (n0 < T) X.load(LP + tile_of(n0, 0), lane);
    for (int k = 0; k < T; ++k) {
      const int n1 = first_of(k + 3);
      if (n1 < T) N.load(LP + tile_of(n1, k + 1), lane);
      if (BACK) X.transpose();
      __syncthreads();  // block k is published
      if (n0 < T) {
        rhs_frags(rx + 32 * blk(k), ry + 32 * blk(k), lane, b);
        tile_vec(d, X, b);
        rhs_put(rx + 32 * blk(n0), ry + 32 * blk(n0), d, true, lane);
        for (int n = n0 + NO; n < T; n += NO) {
          X.load(LP + tile_of(n, k), lane);
          if (BACK) X.transpose();
          tile_vec(d, X, b);
          rhs_put(rx + 32 * blk(n), ry + 32 * blk(n), d, true, lane);
        }
      }
      X = N;
      n0 = n1;
    }
  }
}

// rx, ry := D (L L^T)^-1 D of them, two right-hand sides (shared, 16-byte aligned, zero
// from m up to a multiple of 32), each scaled by a power of two to a largest value in
// [1, 2) for the FP16 terms.
template <int NT>
__device__ void chol_solve2(const uint4* LP, int m, const float* dsc, float* rx, float* ry,
                            double* sh, uint4* ring) {
  const int T = (m + 31) / 32;
  float mx = 0.f, my = 0.f;
  for (int i = threadIdx.x; i < m; i += NT) {
    rx[i] *= dsc[i];
    ry[i] *= dsc[i];
    mx = fmaxf(mx, fabsf(rx[i]));
    my = fmaxf(my, fabsf(ry[i]));
  }
  const float2 mxy = block_max2<NT>(mx, my, sh);
  const int ex = mxy.x > 0.f && mxy.x < INFINITY ? ilogbf(mxy.x) : 0;
  const int ey = mxy.y > 0.f && mxy.y < INFINITY ? ilogbf(mxy.y) : 0;
  for (int i = threadIdx.x; i < m; i += NT) {
    rx[i] = ldexpf(rx[i], -ex);
    ry[i] = ldexpf(ry[i], -ey);
  }
  __syncthreads();
  tri_solve<NT, false>(LP, T, rx, ry, ring);
  tri_solve<NT, true>(LP, T, rx, ry, ring);
  for (int i = threadIdx.x; i < m; i += NT) {
    rx[i] = ldexpf(rx[i] * dsc[i], ex);
    ry[i] = ldexpf(ry[i] * dsc[i], ey);
  }
  __syncthreads();
}

// Shared-memory layout of k_tps_solve_mp for subdomains of at most n centres.
struct MpLayout {
  int np;        // n rounded up to 32
  size_t d_off;  // doubles: V 3n, xc n, yc n, Y/C 3n, W 4n
  size_t f2_off; // float2: zx, zy, gx, gy (np each)
  size_t f_off;  // float: vx, vy, rx, ry (np each)
  size_t i2_off; // int2: lattice coordinates (np)
  size_t p_off;  // panel: panel_bytes(warps)
  size_t bytes;
  __host__ __device__ MpLayout(int n, int warps) {
    np = (n + 31) & ~31;
    d_off = 0;
    f2_off = d_off + (size_t)12 * n * sizeof(double);
    f_off = f2_off + (size_t)4 * np * sizeof(float2);
    i2_off = f_off + (size_t)4 * np * sizeof(float);
    p_off = i2_off + (size_t)np * sizeof(int2);
    bytes = p_off + panel_bytes(warps);
  }
};

// One block per subdomain.  Status per subdomain: 0 solved here, 1 needs the FP64
// LU fallback (rank-deficient P, Cholesky breakdown or no convergence).
//
// Buffers per subdomain (offset mat_off, a multiple of 4 elements): matrices holds
// B22 = (Q^T A Q)[3:, 3:] as (hi, lo) float pairs, both triangles, leading
// dimension mp = m rounded up to 4; matrices32 holds the tiles of its Cholesky factor
// (chol_factor; in shared memory for small subdomains).
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT)
    k_tps_solve_mp(const fi_tps_plan* plan_ptr, const double* cx, const double* cy,
                   const float* ux, const float* uy, const int32_t* counts,
                   const int64_t* offsets, const int32_t* indices, const int64_t* mat_off,
                   double* matrices, float* matrices32, const double* phi_table,
                   const float2* phi_table2, int64_t table_size, const int32_t* cxy2,
                   const int32_t* c_on_lattice, double threshold, int use_threshold,
                   const int64_t* w_off, double* weights,
                   double* smoothed_x, double* smoothed_y, int32_t* iters, int32_t* nfixed,
                   int32_t* status, double* max_udiff, int32_t* sweeps,
                   const int32_t* order, int max_refine, int n_layout) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double sh[BLOCK_SUMS];
  __shared__ double s_sum[16];
  __shared__ double s_tau[3], s_T[9];
  __shared__ double s_R[9];
  __shared__ double s_q1[6], s_c[6], s_a[6];
  __shared__ int s_flag, s_bad[2], s_lat;
  const fi_tps_plan p = *plan_ptr;
  // a cluster of csize CTAs per subdomain (1 without cluster launch): all of them
  // factor P and share the FP64 build and projection, rank 0 then solves alone
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks();
  const int crank = (int)cluster.block_rank();
  const int sd = order != nullptr ? order[blockIdx.x / csize] : (int)(blockIdx.x / csize);
  const int N = counts[sd];
  const int m = N - 3;
  const int64_t off = offsets[sd];
  const int32_t* idx = indices + off;
  const double lam = p.smoothing;
  if (threadIdx.x == 0 && crank == 0) {
    status[sd] = 1;
    if (sweeps != nullptr) sweeps[sd] = 0;
  }
  if (m < 1) return;  // fewer than 4 centres: FP64 LU path
  const int mp = (m + 3) & ~3;

  const MpLayout lay(n_layout, NW);
  const int n = n_layout;
  double* V = reinterpret_cast<double*>(smraw + lay.d_off);  // 3 n (rows k: v_k)
  double* xc = V + 3 * n;
  double* yc = xc + n;
  double* YC = yc + n;  // Y = A V (3 n), then C = (Q^T A Q)[0:3, 3:] (3 n)
  double* W = YC + 3 * n;  // 4 n: QR scratch, Z, then t / w
  float2* zx2 = reinterpret_cast<float2*>(smraw + lay.f2_off);
  float2* zy2 = zx2 + lay.np;
  float2* gx2 = zy2 + lay.np;
  float2* gy2 = gx2 + lay.np;
  float* vx = reinterpret_cast<float*>(smraw + lay.f_off);
  float* vy = vx + lay.np;
  float* rx = vy + lay.np;
  float* ry = rx + lay.np;
  int2* cxy = reinterpret_cast<int2*>(smraw + lay.i2_off);
  float* panel = reinterpret_cast<float*>(smraw + lay.p_off);

  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float2* B2 = reinterpret_cast<float2*>(matrices + mat_off[sd]);

  if (threadIdx.x == 0)
    s_lat = (cxy2 != nullptr && c_on_lattice != nullptr && phi_table != nullptr) ? *c_on_lattice : 0;
  for (int i = threadIdx.x; i < N; i += NT) {
    const int a = idx[i];
    xc[i] = cx[a];
    yc[i] = cy[a];
    if (cxy2 != nullptr) cxy[i] = make_int2(cxy2[2 * a], cxy2[2 * a + 1]);
  }
  __syncthreads();
  const bool lat = s_lat != 0;
  // Centres on the lattice: cxy becomes the grid indices ((2x - 2x_0) / gx,
  // (2y - 2y_0) / gy) of the grid of steps (gx, gy) through them, and, when every
  // offset of the grid's extent fits, tab holds the (hi, lo) kernel value of each
  // offset (a, b) at tab[b tw + a] (tw = 0: no table).  The table lives in W's last n
  // doubles, free until the refinement.
  int gx = 1, gy = 1, tw = 0;
  float2* tab = reinterpret_cast<float2*>(W + 3 * n);
  const int tsz32 = (int)(table_size < (int64_t)INT_MAX ? table_size : (int64_t)INT_MAX);
  if (lat) {
    const int2 o = cxy[0];
    int v[6];
    lat_grid_init(v);
    for (int i = threadIdx.x; i < N; i += NT) lat_grid_add(v, cxy[i].x - o.x, cxy[i].y - o.y);
    lat_grid_block(v, reinterpret_cast<int*>(sh));
    const LatTable g = lat_table_of(v, n, tsz32);
    gx = g.gx;
    gy = g.gy;
    for (int i = threadIdx.x; i < N; i += NT)
      cxy[i] = make_int2((cxy[i].x - o.x) / gx, (cxy[i].y - o.y) / gy);
    if (g.ok && phi_table2 != nullptr) {
      tw = g.wx;
      for (int e = threadIdx.x; e < g.wx * g.wy; e += NT) {
        const int b = e / g.wx, a = e - b * g.wx;
        tab[e] = phi_table2[(gy * b) * (gy * b) + (gx * a) * (gx * a)];
      }
    }
    __syncthreads();
  }
  // A = K + lam I, entry (r, c); on the lattice 4 r^2 is an integer table index
  auto a_entry = [&](int r, int c) -> double {
    if (r == c) return lam;
    if (lat) {
      const int2 ca = cxy[r], cb = cxy[c];
      const int64_t dx = (int64_t)gx * (ca.x - cb.x), dy = (int64_t)gy * (ca.y - cb.y);
      const int64_t kq = dy * dy + dx * dx;
      if (kq < table_size) return __ldg(phi_table + kq);
      return phi_pair(xc[r], yc[r], xc[c], yc[c], nullptr, 0);
    }
    return phi_pair(xc[r], yc[r], xc[c], yc[c], phi_table, table_size);
  };
  // the same entry as a (hi, lo) float pair; ci = lattice coordinates of centre i
  const float2 lam2 = df_split(lam);
  auto a_entry_df = [&](int i, int2 ci, int j) -> float2 {
    if (i == j) return lam2;
    if (lat) {
      const int2 cj = cxy[j];
      const int64_t dx = (int64_t)gx * (ci.x - cj.x), dy = (int64_t)gy * (ci.y - cj.y);
      const int64_t kq = dy * dy + dx * dx;
      if (kq < table_size)
        return phi_table2 != nullptr ? phi_table2[kq] : df_split(__ldg(phi_table + kq));
      return df_split(phi_pair(xc[i], yc[i], xc[j], yc[j], nullptr, 0));
    }
    return df_split(phi_pair(xc[i], yc[i], xc[j], yc[j], phi_table, table_size));
  };
  // entries (i, j0 .. j0 + cnt - 1) of A as pairs (0 < cnt <= 8, the rest zero): on the
  // lattice the eight table loads are issued before any is used (the loads, mostly
  // L2 hits, bound these phases), the diagonal and far entries patched afterwards
  auto a_batch_df = [&](int i, int2 ci, int j0, int cnt, float2(&out)[8]) {
    if (lat && tw > 0) {  // every offset in the shared table
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int2 cj = cxy[j0 + min(u, cnt - 1)];
        out[u] = tab[abs(ci.y - cj.y) * tw + abs(ci.x - cj.x)];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (u >= cnt)
          out[u] = make_float2(0.f, 0.f);
        else if (j0 + u == i)
          out[u] = lam2;
      }
    } else if (lat && phi_table2 != nullptr) {
      // 4 r^2 in 32-bit integers: the lattice coordinates are below 2^30 in magnitude,
      // so their differences fit, and |dx|, |dy| <= 32767 keeps dx^2 + dy^2 below
      // 2^31; farther pairs (beyond the table anyway) take the direct kernel value
      int kq[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int2 cj = cxy[j0 + min(u, cnt - 1)];
        const int dx = gx * (ci.x - cj.x), dy = gy * (ci.y - cj.y);
        const bool near = (unsigned)dx + 32767u <= 65534u && (unsigned)dy + 32767u <= 65534u;
        kq[u] = near ? dy * dy + dx * dx : INT_MAX;
        out[u] = phi_table2[kq[u] < tsz32 ? kq[u] : 0];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int j = j0 + u;
        if (u >= cnt)
          out[u] = make_float2(0.f, 0.f);
        else if (j == i)
          out[u] = lam2;
        else if (kq[u] >= tsz32)
          out[u] = df_split(phi_pair(xc[i], yc[i], xc[j], yc[j], nullptr, 0));
      }
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        out[u] = (u < cnt) ? a_entry_df(i, ci, j0 + u) : make_float2(0.f, 0.f);
    }
  };

  // ---- Householder QR of P = [1, y, x] (FP64), V rows k hold v_k (zeros above k).  The
  // first reflector follows from N alone; each of the others needs one block-wide sum
  // (its norm, with its product with the next column); thread 0 does the scalar FP64 work.
  {
    double* Va = V;
    double* Vb = V + n;
    double* Vc = V + 2 * n;
    double s2[2] = {0.0, 0.0};
    for (int i = threadIdx.x; i < N; i += NT) {
      s2[0] += yc[i];
      s2[1] += xc[i];
    }
    block_sums<NT, 2>(s2, sh, s_sum);
    if (threadIdx.x == 0) {
      const double rn = sqrt((double)N), tau = 1.0 / ((double)N + rn);
      s_tau[0] = tau;
      s_R[0] = -rn;
      s_c[0] = tau * (s_sum[0] + rn * yc[0]);
      s_c[1] = tau * (s_sum[1] + rn * xc[0]);
      s_c[2] = 1.0 + rn;
      s_flag = 0;
    }
    __syncthreads();
    s2[0] = s2[1] = 0.0;
    for (int i = threadIdx.x; i < N; i += NT) {
      const double v = (i == 0) ? s_c[2] : 1.0;
      const double y = yc[i] - s_c[0] * v, x = xc[i] - s_c[1] * v;
      Va[i] = v;
      if (i == 0) {
        s_R[1] = y;
        s_R[2] = x;
        Vb[0] = Vc[0] = 0.0;
      } else {
        Vb[i] = y;
        Vc[i] = x;
        s2[0] += y * y;
        s2[1] += y * x;
      }
    }
    block_sums<NT, 2>(s2, sh, s_sum);
    const double tiny = 1e-9 * 1e-9 * (double)N;  // collinear centres: |R_kk|^2 below it
    if (threadIdx.x == 0) {
      const double q = s_sum[0], y1 = Vb[1];
      if (!(q >= tiny)) s_flag = 1;
      const double alpha = (y1 >= 0.0) ? -sqrt(q) : sqrt(q);
      s_tau[1] = 1.0 / (q - alpha * y1);  // 2 / |v|^2, |v|^2 = 2 (q - alpha y1)
      s_R[4] = alpha;
      s_c[0] = s_tau[1] * (s_sum[1] - alpha * Vc[1]);
      Vb[1] = y1 - alpha;
    }
    __syncthreads();
    double s1[1] = {0.0};
    for (int i = 1 + threadIdx.x; i < N; i += NT) {
      const double x = Vc[i] - s_c[0] * Vb[i];
      if (i == 1) {
        s_R[5] = x;
        Vc[1] = 0.0;
      } else {
        Vc[i] = x;
        s1[0] += x * x;
      }
    }
    block_sums<NT, 1>(s1, sh, s_sum);
    if (threadIdx.x == 0) {
      const double q = s_sum[0], x2 = Vc[2];
      if (!(q >= tiny)) s_flag = 1;
      const double alpha = (x2 >= 0.0) ? -sqrt(q) : sqrt(q);
      s_tau[2] = 1.0 / (q - alpha * x2);
      s_R[8] = alpha;
      Vc[2] = x2 - alpha;
    }
    __syncthreads();
    if (s_flag != 0) return;
  }
  const double* V0 = V;
  const double* V1 = V + n;
  const double* V2 = V + 2 * n;
  double* Y0 = YC;
  double* Y1 = YC + n;
  double* Y2 = YC + 2 * n;
  // V and Z as (hi, lo) float pairs, [3][np] each: the f2 and f regions (6 np pairs)
  // are free until the refinement
  float2* Vd = zx2;
  float2* Zd = zx2 + 3 * lay.np;
  const int np = lay.np;
  for (int i = threadIdx.x; i < np; i += NT) {
    const bool in = i < N;
    Vd[i] = in ? df_split(V0[i]) : make_float2(0.f, 0.f);
    Vd[np + i] = in ? df_split(V1[i]) : make_float2(0.f, 0.f);
    Vd[2 * np + i] = in ? df_split(V2[i]) : make_float2(0.f, 0.f);
  }
  __syncthreads();
  // every CTA of the cluster has started (and holds its V) before any CTA writes
  // into a peer's shared memory below
  cluster.sync();
  // ---- Y = A V in double-float on the FP32 pipe.  A is symmetric: lane = column c,
  // the rows r in chunks (jobs = column block x chunk, a multiple of the warp count
  // when the scratch allows); the chunks' partial sums are added in a fixed order.
  // The column blocks are spread over the cluster's CTAs; each Y value is rounded to
  // double and written into every CTA's Y.
  {
    auto write_y = [&](int c, float2 s0, float2 s1, float2 s2) {
      const double y0 = df_to_double(s0), y1 = df_to_double(s1), y2 = df_to_double(s2);
      for (int q = 0; q < csize; ++q) {
        double* Yq = (q == crank) ? YC : cluster.map_shared_rank(YC, q);
        Yq[c] = y0;
        Yq[n + c] = y1;
        Yq[2 * n + c] = y2;
      }
    };
    const int ncb = (N + 31) / 32;
    const int nloc = (crank < ncb) ? (ncb - crank + csize - 1) / csize : 0;
    int rs = 1;
    if (nloc > 0) {
      int a = nloc, b = NW;
      while (b != 0) {
        const int t = a % b;
        a = b;
        b = t;
      }
      rs = NW / a;  // nloc * rs is a multiple of NW
      const int max_jobs = (int)(panel_bytes(NW) / (96 * sizeof(float2)));
      while (rs > 1 && (nloc * rs > max_jobs || 8 * rs > N)) rs >>= 1;
    }
    float2* part = reinterpret_cast<float2*>(panel);  // [job][3][32]
    for (int j = wid; j < nloc * rs; j += NW) {
      const int l = j / rs, ch = j - l * rs;
      const int c = 32 * (crank + csize * l) + lane;
      const int r0 = (int)((int64_t)N * ch / rs), r1 = (int)((int64_t)N * (ch + 1) / rs);
      // sums of V0 and V1 in the lanes of (h01, l01) (packed FP32x2), V2 in (h2, l2)
      float2 h01 = make_float2(0.f, 0.f), l01 = make_float2(0.f, 0.f);
      float h2 = 0.f, l2 = 0.f;
      if (c < N) {
        const int2 cc = cxy[c];
        for (int rb = r0; rb < r1; rb += 8) {
          const int cnt = min(8, r1 - rb);
          float2 a[8];
          a_batch_df(c, cc, rb, cnt, a);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (u < cnt) {
              const int r = rb + u;
              const float2 v0 = Vd[r], v1 = Vd[np + r];
              df_mac_x2(a[u], make_float2(v0.x, v1.x), make_float2(v0.y, v1.y), h01, l01);
              df_mac(a[u], Vd[2 * np + r], h2, l2);
            }
          }
        }
      }
      const float h0 = h01.x, l0 = l01.x, h1 = h01.y, l1 = l01.y;
      if (rs == 1) {
        if (c < N) write_y(c, make_float2(h0, l0), make_float2(h1, l1), make_float2(h2, l2));
      } else {
        part[(3 * j + 0) * 32 + lane] = make_float2(h0, l0);
        part[(3 * j + 1) * 32 + lane] = make_float2(h1, l1);
        part[(3 * j + 2) * 32 + lane] = make_float2(h2, l2);
      }
    }
    if (rs > 1) {
      __syncthreads();
      for (int t = threadIdx.x; t < nloc * 32; t += NT) {
        const int l = t >> 5, ln = t & 31;
        const int c = 32 * (crank + csize * l) + ln;
        if (c >= N) continue;
        const float2* pj = part + (size_t)3 * 32 * (l * rs);
        float2 s0 = pj[ln], s1 = pj[32 + ln], s2 = pj[64 + ln];
        for (int ch = 1; ch < rs; ++ch) {
          pj += 3 * 32;
          s0 = df_add(s0, pj[ln]);
          s1 = df_add(s1, pj[32 + ln]);
          s2 = df_add(s2, pj[64 + ln]);
        }
        write_y(c, s0, s1, s2);
      }
    }
  }
  cluster.sync();
  // ---- Q^T A Q = A - Z V^T - V Z^T (compact WY, Q = H0 H1 H2 = I - V T V^T),
  // Y = A V, M = T^T (V^T Y) T, Z = Y T - V M / 2.  FP64: the projection cancels the
  // large affine part of K.
  double* Z0 = W;
  double* Z1 = W + n;
  double* Z2 = W + 2 * n;
  {
    __shared__ double s_M[9];
    const double* Vk[3] = {V0, V1, V2};
    const double* Yk[3] = {Y0, Y1, Y2};
    double pr[12];  // V^T V above the diagonal, V^T Y
    for (int a = 0; a < 12; ++a) pr[a] = 0.0;
    for (int i = threadIdx.x; i < N; i += NT) {
      pr[0] += V0[i] * V1[i];
      pr[1] += V0[i] * V2[i];
      pr[2] += V1[i] * V2[i];
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) pr[3 + 3 * a + b] += Vk[a][i] * Yk[b][i];
    }
    block_sums<NT, 12>(pr, sh, s_sum);
    const double *vtv = s_sum, *vty = s_sum + 3;
    if (threadIdx.x == 0) {
      double T[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      T[0] = s_tau[0];
      T[4] = s_tau[1];
      T[8] = s_tau[2];
      T[1] = -s_tau[1] * T[0] * vtv[0];                      // T[0][1]
      T[2] = -s_tau[2] * (T[0] * vtv[1] + T[1] * vtv[2]);    // T[0][2]
      T[5] = -s_tau[2] * (T[4] * vtv[2]);                    // T[1][2]
      double G[9];  // (V^T Y) T
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
          double acc = 0.0;
          for (int j = 0; j < 3; ++j) acc += vty[3 * a + j] * T[3 * j + b];
          G[3 * a + b] = acc;
        }
      for (int a = 0; a < 3; ++a)  // M = T^T G
        for (int b = 0; b < 3; ++b) {
          double acc = 0.0;
          for (int j = 0; j < 3; ++j) acc += T[3 * j + a] * G[3 * j + b];
          s_M[3 * a + b] = acc;
        }
      for (int a = 0; a < 9; ++a) s_T[a] = T[a];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += NT) {  // Z = Y T - V M / 2
      const double y[3] = {Y0[i], Y1[i], Y2[i]};
      const double v[3] = {V0[i], V1[i], V2[i]};
      double z[3];
      for (int k = 0; k < 3; ++k) {
        double acc = 0.0;
        for (int j = 0; j < 3; ++j) acc += y[j] * s_T[3 * j + k] - 0.5 * v[j] * s_M[3 * j + k];
        z[k] = acc;
      }
      Z0[i] = z[0];
      Z1[i] = z[1];
      Z2[i] = z[2];
    }
    for (int i = N + threadIdx.x; i < np; i += NT) Zd[i] = Zd[np + i] = Zd[2 * np + i] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += NT) {
      Zd[i] = df_split(Z0[i]);
      Zd[np + i] = df_split(Z1[i]);
      Zd[2 * np + i] = df_split(Z2[i]);
    }
    __syncthreads();
  }
  auto proj = [&](int r, int c) -> double {  // (Q^T A Q)[r][c], global indices
    double v = a_entry(r, c);
    v -= Z0[r] * V0[c] + V0[r] * Z0[c];
    v -= Z1[r] * V1[c] + V1[r] * Z1[c];
    v -= Z2[r] * V2[c] + V2[r] * Z2[c];
    return v;
  };
  // C[k][c] = (Q^T A Q)[k][c + 3], k < 3 (Y is no longer needed)
  double* C = YC;
  if (crank == 0) {
    for (int i = threadIdx.x; i < 3 * m; i += NT) {
      const int k = i / m, c = i - k * m;
      C[k * n + c] = proj(k, c + 3);
    }
  }
  // B22 by 32 x 32 tiles (I >= J), half a tile (16 columns) at a time: the lower
  // entries are written by columns, then mirrored through a per-warp shared tile.
  {
    float2* S = reinterpret_cast<float2*>(panel) + wid * 16 * 33;
    const int T = (m + 31) / 32;
    const int npairs = T * (T + 1) / 2;
    for (int pidx = crank * NW + wid; pidx < npairs; pidx += csize * NW) {
      int I = (int)((sqrtf(8.f * pidx + 1.f) - 1.f) * 0.5f);
      while ((I + 1) * (I + 2) / 2 <= pidx) ++I;
      while (I * (I + 1) / 2 > pidx) --I;
      const int J = pidx - I * (I + 1) / 2;
      const int r = 32 * I + lane;
      // the row's -Z_k and -V_k pairs and lattice coordinates
      const int rg = (r < m) ? r + 3 : 3;
      const int2 cr = cxy[rg];
      float2 nz[3], nv[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float2 zv = Zd[k * np + rg], vv = Vd[k * np + rg];
        nz[k] = make_float2(-zv.x, -zv.y);
        nv[k] = make_float2(-vv.x, -vv.y);
      }
      for (int h = 0; h < 2; ++h) {
        for (int qb = 0; qb < 16; qb += 8) {
          const int c0 = 32 * J + 16 * h + qb;
          if (c0 >= m) break;
          const int cnt = min(8, m - c0);
          float2 a[8];
          a_batch_df(rg, cr, c0 + 3, cnt, a);
          // A - Z V^T - V Z^T in double-float: entries of A up to ~1e5 cancel to B
          // entries ~1e2-1e4; the ~2^-48 |A| rounding leaves B within ~1e-11 of its
          // FP64 value, the interpolated field within ~1e-9 px.  Columns c, c + 1 in
          // the lanes of float2 pairs (packed FP32x2 instructions).
#pragma unroll
          for (int u = 0; u < 8; u += 2) {
            const int c = c0 + u;
            const bool in0 = u < cnt && r < m && r >= c;
            const bool in1 = u + 1 < cnt && r < m && r >= c + 1;
            if (in0 || in1) {
              const int cg0 = c + 3, cg1 = min(c + 4, N - 1);
              float2 sh = make_float2(a[u].x, a[u + 1].x), sl = make_float2(a[u].y, a[u + 1].y);
#pragma unroll
              for (int k = 0; k < 3; ++k) {
                const float2 v0 = Vd[k * np + cg0], v1 = Vd[k * np + cg1];
                const float2 z0 = Zd[k * np + cg0], z1 = Zd[k * np + cg1];
                df_mac_x2(nz[k], make_float2(v0.x, v1.x), make_float2(v0.y, v1.y), sh, sl);
                df_mac_x2(nv[k], make_float2(z0.x, z1.x), make_float2(z0.y, z1.y), sh, sl);
              }
              const float2 hi = __fadd2_rn(sh, sl);
              const float2 lo = __fadd2_rn(sl, df_neg2(__fadd2_rn(hi, df_neg2(sh))));
              if (in0) {
                const float2 sv = make_float2(hi.x, lo.x);
                __stcs(B2 + (int64_t)c * mp + r, sv);  // streaming: keeps L2 for the factor
                S[(qb + u) * 33 + lane] = sv;
              }
              if (in1) {
                const float2 sv = make_float2(hi.y, lo.y);
                __stcs(B2 + (int64_t)(c + 1) * mp + r, sv);
                S[(qb + u + 1) * 33 + lane] = sv;
              }
            }
          }
        }
        __syncwarp();
#pragma unroll 4
        for (int st = 0; st < 16; ++st) {
          const int rr = 2 * st + (lane >> 4), qq = lane & 15;
          const int r2 = 32 * I + rr, c2 = 32 * J + 16 * h + qq;
          if (r2 < m && c2 < m && r2 > c2) __stcs(B2 + (int64_t)r2 * mp + c2, S[qq * 33 + rr]);
        }
        __syncwarp();
      }
    }
  }
  cluster.sync();  // the cluster's B tiles are in global memory, visible to rank 0
  if (crank != 0) return;
  // ---- Cholesky factor of D B22 D (D in xc: the centres are no longer needed)
  float* dsc = reinterpret_cast<float*>(xc);
  if (threadIdx.x == 0) s_flag = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += NT) {
    const float v = B2[(int64_t)i * mp + i].x;
    if (!(v > 0.f)) s_flag = 1;
    dsc[i] = (v > 0.f) ? ldexpf(1.f, -(ilogbf(v) >> 1)) : 1.f;
  }
  __syncthreads();
  uint4* LP = (m <= 32 * SMALL_T)
                  ? reinterpret_cast<uint4*>(smraw + lay.p_off + ((CHOL_SMEM + 15) & ~(size_t)15))
                  : reinterpret_cast<uint4*>(matrices32 + mat_off[sd]);
  if (!chol_factor<NT>(B2, m, mp, dsc, LP, panel, &s_flag)) return;
  uint4* ring = (m <= 32 * SMALL_T) ? nullptr : reinterpret_cast<uint4*>(panel);

  // ---- outlier iterations with refined solves (x and y in lockstep)
  double* wx = W + 2 * n;
  double* wy = W + 3 * n;
  for (int r = threadIdx.x; r < lay.np; r += NT) {
    vx[r] = (r < N) ? ux[idx[r]] : 0.f;
    vy[r] = (r < N) ? uy[idx[r]] : 0.f;
    zx2[r] = zy2[r] = make_float2(0.f, 0.f);
    rx[r] = ry[r] = 0.f;
  }
  __syncthreads();
  int count[2] = {1, 1}, fixed[2] = {0, 0};
  bool done[2] = {false, false};
  bool converged_all = true;
  bool z_zero = true;
  int nsweeps = 0;
  while (true) {
    // g = Q^T u = u - V T^T (V^T u): rows 3.. as double-float for the refinement, rows
    // 0..2 for a
    {
      double pr[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      for (int i = threadIdx.x; i < N; i += NT) {
        const double ux_ = (double)vx[i], uy_ = (double)vy[i];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double v = V[k * n + i];
          pr[k] = fma(v, ux_, pr[k]);
          pr[3 + k] = fma(v, uy_, pr[3 + k]);
        }
      }
      block_sums<NT, 6>(pr, sh, s_sum);
      if (threadIdx.x < 6) {  // T^T (V^T u)
        const int k = threadIdx.x % 3, o = threadIdx.x - k;
        double t = 0.0;
        for (int j = 0; j <= k; ++j) t = fma(s_T[3 * j + k], s_sum[o + j], t);
        s_c[threadIdx.x] = t;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < N; i += NT) {
        double gxv = (double)vx[i], gyv = (double)vy[i];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double v = V[k * n + i];
          gxv = fma(-v, s_c[k], gxv);
          gyv = fma(-v, s_c[3 + k], gyv);
        }
        if (i < 3) {
          s_q1[i] = gxv;
          s_q1[3 + i] = gyv;
        } else {
          gx2[i - 3] = df_split(gxv);
          gy2[i - 3] = df_split(gyv);
        }
      }
      __syncthreads();
    }
    // refine z (B z = g): FP32 Cholesky solves, double-float residuals
    bool conv = false;
    double prev = INFINITY;
    for (int it = 0; it < max_refine; ++it) {
      if (z_zero) {  // z = 0: rho = g
        for (int i = threadIdx.x; i < m; i += NT) {
          rx[i] = __fadd_rn(gx2[i].x, gx2[i].y);
          ry[i] = __fadd_rn(gy2[i].x, gy2[i].y);
        }
        __syncthreads();
        z_zero = false;
      } else {
        residual_df2<NT>(B2, m, mp, zx2, zy2, gx2, gy2, rx, ry);
      }
      chol_solve2<NT>(LP, m, dsc, rx, ry, sh, ring);
      ++nsweeps;
      float dm = 0.f, zm = 0.f;
      for (int i = threadIdx.x; i < m; i += NT) {
        if (!done[0]) zx2[i] = df_add(zx2[i], make_float2(rx[i], 0.f));
        if (!done[1]) zy2[i] = df_add(zy2[i], make_float2(ry[i], 0.f));
        // (beyond the FP16 range of the factor's products the corrections are not finite:
        // their bits compare as the largest)
        const unsigned ax = done[0] ? 0u : __float_as_uint(fabsf(rx[i]));
        const unsigned ay = done[1] ? 0u : __float_as_uint(fabsf(ry[i]));
        dm = __uint_as_float(max(__float_as_uint(dm), max(ax, ay)));
        zm = fmaxf(zm, fmaxf(fabsf(zx2[i].x), fabsf(zy2[i].x)));
      }
      const float2 dz = block_max2<NT>(dm, zm, sh);
      if (!(dz.x < INFINITY)) break;  // the FP64 LU takes over
      const double dmax = (double)dz.x, zmax = (double)dz.y;
      if (dmax == 0.0) {
        conv = true;
        break;
      }
      if (it >= 1) {
        // contraction of the FP32-preconditioned refinement, estimated from the last
        // two corrections; the remaining error is about contraction * dmax (1e-10 of
        // z keeps the interpolated displacements within ~1e-8 px)
        const double rho = dmax / prev;
        if (rho < 0.1 && rho * dmax <= 1e-10 * zmax) {
          conv = true;
          break;
        }
        if (it >= 2 && rho > 0.5) {  // at the residual floor
          conv = dmax <= 1e-9 * zmax;
          break;
        }
      }
      prev = dmax;
    }
    if (!conv) {
      converged_all = false;
      break;
    }
    // a = R^-1 (Q1^T u - C z) (R upper triangular); w = Q [0; z]
    {
      // C z and V^T [0; z] of both components in one block-wide sum
      double pr[12];
      for (int k = 0; k < 12; ++k) pr[k] = 0.0;
      for (int i = threadIdx.x; i < m; i += NT) {
        const double zxv = df_to_double(zx2[i]), zyv = df_to_double(zy2[i]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double cv = C[k * n + i], v = V[k * n + i + 3];
          pr[k] = fma(cv, zxv, pr[k]);
          pr[3 + k] = fma(cv, zyv, pr[3 + k]);
          pr[6 + k] = fma(v, zxv, pr[6 + k]);
          pr[9 + k] = fma(v, zyv, pr[9 + k]);
        }
      }
      block_sums<NT, 12>(pr, sh, s_sum);
      if (threadIdx.x < 2) {  // back substitution with R, one component per thread
        const int o = 3 * threadIdx.x;
        for (int k = 2; k >= 0; --k) {
          double t = s_q1[o + k] - s_sum[o + k];
          for (int j = k + 1; j < 3; ++j) t -= s_R[k * 3 + j] * s_a[o + j];
          s_a[o + k] = t / s_R[k * 3 + k];
        }
      } else if (threadIdx.x >= 32 && threadIdx.x < 38) {  // T (V^T [0; z])
        const int t6 = threadIdx.x - 32, k = t6 % 3, o = t6 - k;
        double t = 0.0;
        for (int j = k; j < 3; ++j) t = fma(s_T[3 * k + j], s_sum[6 + o + j], t);
        s_c[t6] = t;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < N; i += NT) {
        double a = (i < 3) ? 0.0 : df_to_double(zx2[i - 3]);
        double b = (i < 3) ? 0.0 : df_to_double(zy2[i - 3]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double v = V[k * n + i];
          a = fma(-v, s_c[k], a);
          b = fma(-v, s_c[3 + k], b);
        }
        wx[i] = a;
        wy[i] = b;
      }
      __syncthreads();
    }
    // smoothed = u - lam w; outlier test (compute_tps_weights_iter, subdom.py:236-280)
    if (threadIdx.x == 0) s_bad[0] = s_bad[1] = 0;
    __syncthreads();
    double mxx = 0.0, mxy = 0.0;
    int bx = 0, by = 0;
    for (int r = threadIdx.x; r < N; r += NT) {
      const double sxv = __dsub_rn((double)vx[r], __dmul_rn(lam, wx[r]));
      const double syv = __dsub_rn((double)vy[r], __dmul_rn(lam, wy[r]));
      const double dfx = fabs(__dsub_rn(sxv, (double)vx[r]));
      const double dfy = fabs(__dsub_rn(syv, (double)vy[r]));
      if (!done[0]) {
        smoothed_x[off + r] = sxv;
        mxx = fmax(mxx, dfx);
        if (use_threshold && dfx > threshold) bx++;
      }
      if (!done[1]) {
        smoothed_y[off + r] = syv;
        mxy = fmax(mxy, dfy);
        if (use_threshold && dfy > threshold) by++;
      }
    }
    if (count[0] == 1 || count[1] == 1) {  // max_udiff is that of the first solution
      mxx = block_max_pos<NT>(mxx, sh);
      mxy = block_max_pos<NT>(mxy, sh);
    }
    if (bx) atomicAdd(&s_bad[0], bx);
    if (by) atomicAdd(&s_bad[1], by);
    __syncthreads();
    const int nbx = s_bad[0], nby = s_bad[1];
    if (threadIdx.x == 0) {
      if (count[0] == 1 && !done[0]) max_udiff[2 * sd] = mxx;
      if (count[1] == 1 && !done[1]) max_udiff[2 * sd + 1] = mxy;
    }
    // store the weights of the components finishing now
    const int n3 = N + 3;
    double* wxo = weights + w_off[sd];
    double* wyo = wxo + n3;
    bool fin[2];
    fin[0] = !done[0] && (!use_threshold || nbx == 0 || count[0] > 10);
    fin[1] = !done[1] && (!use_threshold || nby == 0 || count[1] > 10);
    for (int r = threadIdx.x; r < N; r += NT) {
      if (fin[0]) wxo[r] = wx[r];
      if (fin[1]) wyo[r] = wy[r];
    }
    if (threadIdx.x == 0) {
      if (fin[0])
        for (int k = 0; k < 3; ++k) wxo[N + k] = s_a[k];
      if (fin[1])
        for (int k = 0; k < 3; ++k) wyo[N + k] = s_a[3 + k];
    }
    // replace the erratic values (rounded to float32 like upstream's array)
    for (int r = threadIdx.x; r < N; r += NT) {
      if (!done[0] && !fin[0]) {
        const double sv = smoothed_x[off + r];
        if (fabs(__dsub_rn(sv, (double)vx[r])) > threshold) vx[r] = (float)sv;
      }
      if (!done[1] && !fin[1]) {
        const double sv = smoothed_y[off + r];
        if (fabs(__dsub_rn(sv, (double)vy[r])) > threshold) vy[r] = (float)sv;
      }
    }
    for (int c = 0; c < 2; ++c) {
      if (done[c]) continue;
      if (fin[c]) {
        done[c] = true;
      } else {
        fixed[c] += (c == 0) ? nbx : nby;
        count[c]++;
      }
    }
    __syncthreads();
    if (done[0] && done[1]) break;
  }
  if (threadIdx.x == 0 && sweeps != nullptr) sweeps[sd] = nsweeps;
  if (!converged_all) return;
  if (threadIdx.x == 0) {
    iters[2 * sd] = count[0];
    iters[2 * sd + 1] = count[1];
    nfixed[2 * sd] = fixed[0];
    nfixed[2 * sd + 1] = fixed[1];
    status[sd] = 0;
  }
}

}  // namespace fi

using namespace fi;

extern "C" int fi_tps_phi_table(double* table, int64_t count, void* stream) {
  FI_REQUIRE(table && count > 0, "fi_tps_phi_table: bad arguments");
  k_phi_table<<<1024, 256, 0, (cudaStream_t)stream>>>(table, count);
  return check_launch("fi_tps_phi_table");
}

extern "C" int fi_tps_phi_table2(float* table2, int64_t count, void* stream) {
  FI_REQUIRE(table2 && count > 0 && ((uintptr_t)table2 & 7) == 0,
             "fi_tps_phi_table2: bad arguments");
  k_phi_table2<<<1024, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<float2*>(table2), count);
  return check_launch("fi_tps_phi_table2");
}

// The tail of a launch of narrow blocks: with slots resident blocks per GPU, a solve
// of slots < nb < 2 slots subdomains (in decreasing size) runs the first wave on the
// caller's stream and the last nb - slots subdomains as clusters of two blocks on a
// side stream (fork and join by events), queued behind the first wave: a cluster
// shares a subdomain's build and projection over two blocks, so the small last
// subdomains, which otherwise run alone after the first wave, finish sooner.  One
// side stream and two events per host thread and device, created on first use.
struct TailStreams {
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};

static cudaError_t tail_streams(int dev, TailStreams** out) {
  static thread_local TailStreams per_dev[FI_SMEM_DEVICES];
  if (dev < 0 || dev >= FI_SMEM_DEVICES) return cudaErrorInvalidDevice;
  TailStreams& t = per_dev[dev];
  if (t.side == nullptr) {
    cudaError_t e = cudaStreamCreateWithFlags(&t.side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&t.fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&t.join, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      t.side = nullptr;
      return e;
    }
  }
  *out = &t;
  return cudaSuccess;
}

extern "C" int fi_tps_solve_mp(const fi_tps_plan* plan, int nb_subdom, int max_members,
                               const double* cx, const double* cy, const float* ux,
                               const float* uy, const int32_t* counts, const int64_t* offsets,
                               const int32_t* indices, const int64_t* mat_offsets,
                               double* matrices, float* matrices32, const double* phi_table,
                               const float* phi_table2, int64_t table_size, const int32_t* cxy2,
                               const int32_t* c_on_lattice, double threshold, int use_threshold,
                               const int64_t* w_offsets, double* weights, double* smoothed_x,
                               double* smoothed_y, int32_t* iters, int32_t* nfixed,
                               int32_t* status, double* max_udiff, int32_t* sweeps,
                               const int32_t* order, void* stream) {
  FI_REQUIRE(plan && cx && cy && ux && uy && counts && offsets && indices && mat_offsets &&
                 matrices && matrices32 && w_offsets && weights && smoothed_x &&
                 smoothed_y &&
                 iters && nfixed && status && max_udiff,
             "fi_tps_solve_mp: null pointer");
  FI_REQUIRE(nb_subdom > 0, "fi_tps_solve_mp: no subdomain");
  FI_REQUIRE(((uintptr_t)matrices & 15) == 0 && ((uintptr_t)matrices32 & 15) == 0,
             "fi_tps_solve_mp: matrices must be 16-byte aligned");
  FI_REQUIRE(((uintptr_t)phi_table2 & 7) == 0, "fi_tps_solve_mp: phi_table2 must be 8-byte aligned");
  const int N = max_members > 4 ? max_members : 4;
  int dev = 0, nsm = 0;
  FI_CUDA_TRY(cudaGetDevice(&dev));
  FI_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // 16 warps per subdomain when the subdomains fit in one wave of blocks (shorter
  // latency per subdomain) or when the shared memory of a subdomain leaves room for
  // only one narrow block per SM (more than ~460 centres: 8 warps per SM would do all
  // the work; 992 subdomains of ~500 centres: 7.2 ms so, 6.5 ms with 16 warps);
  // else two blocks of 8 warps per SM
  static SmemLimit limit_wide, limit_narrow;
  size_t smem = MpLayout(N, 8).bytes;
  int per_sm = 0;  // resident narrow blocks per SM
  bool wide = nb_subdom <= nsm;
  if (!wide && smem <= 220 * 1024) {
    FI_CUDA_TRY(raise_smem_limit(k_tps_solve_mp<256>, smem, limit_narrow));
    // queried once per device and size: the call sits between the host's readback and
    // the launch
    static size_t occ_smem[FI_SMEM_DEVICES] = {};
    static int occ_blocks[FI_SMEM_DEVICES] = {};
    per_sm = -1;
    {
      std::lock_guard<std::mutex> lock(smem_limit_mutex());
      if (dev < FI_SMEM_DEVICES && occ_smem[dev] == smem) per_sm = occ_blocks[dev];
    }
    if (per_sm < 0) {
      FI_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tps_solve_mp<256>,
                                                                256, smem));
      std::lock_guard<std::mutex> lock(smem_limit_mutex());
      if (dev < FI_SMEM_DEVICES) {
        occ_smem[dev] = smem;
        occ_blocks[dev] = per_sm;
      }
    }
    wide = per_sm < 2 && MpLayout(N, 16).bytes <= 220 * 1024;
  }
  if (wide) smem = MpLayout(N, 16).bytes;
  FI_REQUIRE(smem <= 220 * 1024, "fi_tps_solve_mp: subdomain of %d vectors too large",
             max_members);
  if (wide) FI_CUDA_TRY(raise_smem_limit(k_tps_solve_mp<512>, smem, limit_wide));
  if (wide) {
    // clusters of S CTAs per subdomain while the subdomains leave SMs idle
    const int S = (4 * nb_subdom <= nsm) ? 4 : (2 * nb_subdom <= nsm) ? 2 : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nb_subdom * S));
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FI_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_tps_solve_mp<512>, plan, cx, cy, ux, uy, counts,
                                   offsets, indices, mat_offsets, matrices, matrices32,
                                   phi_table, reinterpret_cast<const float2*>(phi_table2),
                                   table_size, cxy2, c_on_lattice, threshold,
                                   use_threshold, w_offsets, weights, smoothed_x, smoothed_y,
                                   iters, nfixed, status, max_udiff, sweeps, order, 60, N));
  } else {
    const int slots = per_sm * nsm;
    const int head = (order != nullptr && slots > 0 && nb_subdom > slots &&
                      nb_subdom < 2 * slots) ? slots : nb_subdom;
    k_tps_solve_mp<256><<<head, 256, smem, (cudaStream_t)stream>>>(
        plan, cx, cy, ux, uy, counts, offsets, indices, mat_offsets, matrices, matrices32,
        phi_table, reinterpret_cast<const float2*>(phi_table2), table_size, cxy2, c_on_lattice,
        threshold, use_threshold, w_offsets, weights,
        smoothed_x, smoothed_y, iters, nfixed, status, max_udiff, sweeps, order, 60, N);
    if (head < nb_subdom) {  // the last subdomains in clusters of two, on the side stream
      FI_CUDA_TRY(cudaGetLastError());
      TailStreams* ts = nullptr;
      FI_CUDA_TRY(tail_streams(dev, &ts));
      FI_CUDA_TRY(cudaEventRecord(ts->fork, (cudaStream_t)stream));
      FI_CUDA_TRY(cudaStreamWaitEvent(ts->side, ts->fork, 0));
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(2 * (nb_subdom - head)));
      cfg.blockDim = dim3(256);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = ts->side;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      FI_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_tps_solve_mp<256>, plan, cx, cy, ux, uy, counts,
                                     offsets, indices, mat_offsets, matrices, matrices32,
                                     phi_table, reinterpret_cast<const float2*>(phi_table2),
                                     table_size, cxy2, c_on_lattice, threshold,
                                     use_threshold, w_offsets, weights, smoothed_x, smoothed_y,
                                     iters, nfixed, status, max_udiff, sweeps, order + head, 60,
                                     N));
      FI_CUDA_TRY(cudaEventRecord(ts->join, ts->side));
      FI_CUDA_TRY(cudaStreamWaitEvent((cudaStream_t)stream, ts->join, 0));
      return check_launch("fi_tps_solve_mp", 2);
    }
  }
  return check_launch("fi_tps_solve_mp");
}
