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
// predicted remaining error is below 4e-11 of z, or when it stagnates (then it must
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

// Bytes of a block's panel: the warps' sums of Y with the table of kernel values behind
// them, then the factorisation's staging with the tiles of small subdomains, then the
// right-hand sides of the substitutions or the tile products of the residual.
__host__ __device__ constexpr size_t panel_bytes(int warps) { return (size_t)(2 + warps) * 4608; }
// entries of the table of kernel values
__host__ __device__ constexpr int panel_table(int warps) {
  return (int)((panel_bytes(warps) - (size_t)warps * 96 * sizeof(float2)) / sizeof(float2));
}

// ---- B = Q2^T (K + lam I) Q2 in memory
// (hi, lo) pairs.  Subdomains of more than 96 unknowns: the 32 x 32 tiles (i, j), i >= j,
// of its lower half, 1024 pairs each at i (i + 1) / 2 + j, by columns (rows and columns
// past m zero, diagonal tiles whole): half the bytes of the whole matrix, which the
// projection writes and every residual reads.  Smaller ones: the whole matrix by columns
// (leading dimension ld), since padded tiles could exceed the slot.
constexpr int SMALL_T = 3;

struct BPairs {
  float2* p;
  int m, ld;
  bool tiles;
  __device__ __forceinline__ float2* tile(int i, int j) const {
    return p + (size_t)1024 * (i * (i + 1) / 2 + j);
  }
  // entry (r, c), r >= c, both below m
  __device__ __forceinline__ float2 at(int r, int c) const {
    if (tiles) return tile(r >> 5, c >> 5)[(c & 31) * 32 + (r & 31)];
    return p[(int64_t)c * ld + r];
  }
};

// Sum over the warp of a pair of double-float values held as (x hi, y hi, x lo, y lo).
__device__ __forceinline__ void df_xor_add(float4& v, int o) {
  float4 w;
  w.x = __shfl_xor_sync(0xffffffffu, v.x, o);
  w.y = __shfl_xor_sync(0xffffffffu, v.y, o);
  w.z = __shfl_xor_sync(0xffffffffu, v.z, o);
  w.w = __shfl_xor_sync(0xffffffffu, v.w, o);
  float2 h = make_float2(v.x, v.y), l = make_float2(v.z, v.w);
  df_acc_x2(make_float2(w.x, w.y), make_float2(w.z, w.w), h, l);
  df_norm_x2(h, l);
  v = make_float4(h.x, h.y, l.x, l.y);
}

// rho = g - B z for both components, in double-float (z, g: (x hi, y hi, x lo, y lo) per
// row, zero past m up to a multiple of 32), rounded to float.  A tile is read once and used
// for its rows and, by symmetry, for its columns: half a tile (16 columns) at a time, one
// row per lane from memory, staged in shared memory for the columns (lanes 0..15 the
// columns with rows 0..15, the others with rows 16..31).  A warp takes whole tile columns
// (J = w, 2 W - 1 - w, ...: a long one with a short one; SPLIT warps share a column's
// tiles), so that the column sums stay in registers; the row sums of each tile go to `part`
// (512 bytes per tile below the diagonal), the column sums behind them, and are added in a
// fixed order at the end.  stage: 16 * 33 pairs per warp.
__host__ __device__ inline size_t residual_part_bytes(int T, int split) {
  return (size_t)512 * (T * (T - 1) / 2 + T * split);
}

template <int NT>
__device__ __noinline__ void residual_tiles(const BPairs B, const float4* z, const float4* g,
                                            float* rx, float* ry, float4* part, float2* stage) {
  constexpr int NW = NT / 32, SPLIT = NW / 8, COLS = NW / SPLIT;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int T = (B.m + 31) / 32;
  float4* colsum = part + 32 * (T * (T - 1) / 2);
  float2* S = stage + wid * 16 * 33;
  const int w = wid / SPLIT, sp = wid % SPLIT;
  const int cq = lane & 15, hf = lane >> 4;
  for (int round = 0; round * COLS < T; ++round) {
    const int J = round * COLS + ((round & 1) ? COLS - 1 - w : w);
    if (J >= T) continue;
    // column sums of the lane's column in each half
    float2 ch[2], cl[2];
    ch[0] = ch[1] = cl[0] = cl[1] = make_float2(0.f, 0.f);
    for (int I = J + sp; I < T; I += SPLIT) {
      const float2* tile = B.tile(I, J);
      float2 rh = make_float2(0.f, 0.f), rl = rh;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2 v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = __ldcs(tile + (16 * h + q) * 32 + lane);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 16; ++q) S[q * 33 + lane] = v[q];
        if (I != J) {
          const float4* zc = z + 32 * J + 16 * h;
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            const float4 f = zc[q];
            df_mac_x2(v[q], make_float2(f.x, f.y), make_float2(f.z, f.w), rh, rl);
          }
        }
        __syncwarp();
        const float4* zr = z + 32 * I + 16 * hf;
        const float2* Sc = S + cq * 33 + 16 * hf;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float4 f = zr[k];
          df_mac_x2(Sc[k], make_float2(f.x, f.y), make_float2(f.z, f.w), ch[h], cl[h]);
        }
      }
      if (I != J) part[32 * (I * (I - 1) / 2 + J) + lane] = make_float4(rh.x, rh.y, rl.x, rl.y);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 v = make_float4(ch[h].x, ch[h].y, cl[h].x, cl[h].y);
      df_xor_add(v, 16);
      if (hf == h) colsum[32 * (SPLIT * J + sp) + lane] = v;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < B.m; i += NT) {
    const int I = i >> 5, l = i & 31;
    const float4 gv = g[i];
    float2 h = make_float2(-gv.x, -gv.y), lo = make_float2(-gv.z, -gv.w);
    for (int q = 0; q < SPLIT; ++q) {
      const float4 f = colsum[32 * (SPLIT * I + q) + l];
      df_acc_x2(make_float2(f.x, f.y), make_float2(f.z, f.w), h, lo);
    }
    for (int J = 0; J < I; ++J) {
      const float4 f = part[32 * (I * (I - 1) / 2 + J) + l];
      df_acc_x2(make_float2(f.x, f.y), make_float2(f.z, f.w), h, lo);
    }
    rx[i] = -__fadd_rn(h.x, lo.x);
    ry[i] = -__fadd_rn(h.y, lo.y);
  }
  __syncthreads();
}

// The same for the whole matrix of a small subdomain: a warp per column, rows over the
// lanes.
template <int NT>
__device__ __noinline__ void residual_small(const BPairs B, const float4* z, const float4* g,
                                            float* rx, float* ry) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c = wid; c < B.m; c += NT / 32) {
    float2 h = make_float2(0.f, 0.f), l = h;
    for (int r = lane; r < B.m; r += 32) {
      const float4 f = z[r];
      df_mac_x2(B.p[(int64_t)c * B.ld + r], make_float2(f.x, f.y), make_float2(f.z, f.w), h, l);
    }
    float4 v = make_float4(h.x, h.y, l.x, l.y);
    for (int o = 16; o > 0; o >>= 1) df_xor_add(v, o);
    if (lane == 0) {
      const float4 gv = g[c];
      float2 sh = make_float2(-gv.x, -gv.y), sl = make_float2(-gv.z, -gv.w);
      df_acc_x2(make_float2(v.x, v.y), make_float2(v.z, v.w), sh, sl);
      rx[c] = -__fadd_rn(sh.x, sl.x);
      ry[c] = -__fadd_rn(sh.y, sl.y);
    }
  }
  __syncthreads();
}

// ---- entries of K
// kernel value of a pair of centres by log(), as a (hi, lo) pair
static __device__ __noinline__ float2 phi_far(double xa, double ya, double xb, double yb,
                                              const double* table, int64_t tsize) {
  return df_split(phi_pair(xa, ya, xb, yb, table, tsize));
}

// How a block finds phi of two centres i, j (K_TABLE: every offset of the centres' grid in
// shared memory, at |code_y| tw + |code_x| of the difference of their codes; K_GATHER: the
// lattice table in memory by 4 r^2 of their lattice coordinates; K_DIRECT: log()).
enum KMode { K_TABLE, K_GATHER, K_DIRECT };

struct KEntries {
  const int2* code;  // grid codes (K_TABLE) or lattice coordinates (K_GATHER)
  const float2* tab;
  int tw;
  const float2* table2;  // (hi, lo) of phi(k / 4), tsz32 entries
  int tsz32;
  const double *xc, *yc;
  const double* table;
  int64_t tsize;
  template <int MODE>
  __device__ __forceinline__ float2 get(int i, int2 ci, int j) const {
    if (MODE == K_DIRECT) return phi_far(xc[i], yc[i], xc[j], yc[j], table, tsize);
    const int2 cj = code[j];
    const int dx = ci.x - cj.x, dy = ci.y - cj.y;
    if (MODE == K_TABLE) return tab[abs(dy) * tw + abs(dx)];
    // 4 r^2 in 32-bit integers: the lattice coordinates are below 2^30 in magnitude, so
    // their differences fit, and |dx|, |dy| <= 32767 keeps dx^2 + dy^2 below 2^31; farther
    // pairs (beyond the table anyway) take the direct kernel value
    const bool near = (unsigned)dx + 32767u <= 65534u && (unsigned)dy + 32767u <= 65534u;
    const int kq = near ? dy * dy + dx * dx : INT_MAX;
    if (kq < tsz32) return table2[kq];
    return phi_far(xc[i], yc[i], xc[j], yc[j], nullptr, 0);
  }
};

// Y = (K + lam I) V in double-float, one column of the symmetric K per lane.  A column
// block at a time, the rows shared by the warps, whose sums are added in a fixed order.
// V's first column is 1 but for its first entry v00, so that sum takes additions only; the
// others' products run as packed pairs (vy: (v1 hi, v2 hi, v1 lo, v2 lo) per row).  Column
// blocks are spread over the cluster's blocks; each value is rounded to double and written
// into every block's Y (3 rows of n).
template <int NT, int MODE>
__device__ __noinline__ void build_y(const KEntries K, const float4* vy, const double* V,
                                     double v00, double lam, int N, int n, double* Y,
                                     float2* part) {
  constexpr int NW = NT / 32;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int r0 = (N * wid / NW) & ~1, r1 = wid == NW - 1 ? N : (N * (wid + 1) / NW) & ~1;
  for (int cb = crank; 32 * cb < N; cb += csize) {
    const int c = min(32 * cb + lane, N - 1);
    const int2 cc = K.code[c];
    // sums of column 0 over even and odd rows in the lanes of (ah, al); of columns 1 and 2
    // in the lanes of (bh, bl)
    float2 ah = make_float2(0.f, 0.f), al = ah, bh = ah, bl = ah;
    int r = r0;
#pragma unroll 4
    for (; r + 1 < r1; r += 2) {
      const float2 k0 = K.get<MODE>(c, cc, r), k1 = K.get<MODE>(c, cc, r + 1);
      const float4 f0 = vy[r], f1 = vy[r + 1];
      df_acc_x2(make_float2(k0.x, k1.x), make_float2(k0.y, k1.y), ah, al);
      df_mac_x2(k0, make_float2(f0.x, f0.y), make_float2(f0.z, f0.w), bh, bl);
      df_mac_x2(k1, make_float2(f1.x, f1.y), make_float2(f1.z, f1.w), bh, bl);
    }
    if (r < r1) {
      const float2 k0 = K.get<MODE>(c, cc, r);
      const float4 f0 = vy[r];
      df_acc_x2(make_float2(k0.x, 0.f), make_float2(k0.y, 0.f), ah, al);
      df_mac_x2(k0, make_float2(f0.x, f0.y), make_float2(f0.z, f0.w), bh, bl);
    }
    float2* pw = part + wid * 96 + lane;
    pw[0] = df_add(make_float2(ah.x, al.x), make_float2(ah.y, al.y));
    pw[32] = make_float2(bh.x, bl.x);
    pw[64] = make_float2(bh.y, bl.y);
    __syncthreads();
    if (wid < 3 && 32 * cb + lane < N) {  // one column of V per warp
      const float2* q = part + 32 * wid + lane;
      float2 sum = q[0];
      for (int w = 1; w < NW; ++w) sum = df_add(sum, q[96 * w]);
      // K has a zero diagonal: lam v; row 0 of column 0 counted as 1
      double y = df_to_double(sum) + lam * V[wid * n + c];
      if (wid == 0) y += (v00 - 1.0) * df_to_double(K.get<MODE>(c, cc, 0));
      for (int b = 0; b < csize; ++b) {
        double* Yb = (b == crank) ? Y : cluster.map_shared_rank(Y, b);
        Yb[wid * n + c] = y;
      }
    }
    __syncthreads();
  }
}

// B = K + lam I - Z V^T - V Z^T below row and column 3, in double-float, by 32 x 32 tiles
// (one row per lane, two columns per packed instruction).  V's first column is 1 there, so
// its two products are additions.  Entries of K up to ~1e5 cancel to B entries ~1e2-1e4;
// the ~2^-48 |K| rounding leaves B within ~1e-11 of its FP64 value, the interpolated field
// within ~1e-9 px.  cols: columns -z0, v1, v2, z1, z2 (np / 2 each) as pairs of
// neighbouring unknowns (hi, hi, lo, lo).
template <int NT, int MODE>
__device__ __noinline__ void build_b(const KEntries K, const float4* cols, int np, float2 lam,
                                     const BPairs B, int crank, int csize) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int m = B.m, N = m + 3;
  const int T = (m + 31) / 32;
  const float4 *nz0 = cols, *v1 = nz0 + np / 2, *v2 = v1 + np / 2, *z1 = v2 + np / 2,
               *z2 = z1 + np / 2;
  for (int pidx = crank * NW + wid; pidx < T * (T + 1) / 2; pidx += csize * NW) {
    int I = (int)((sqrtf(8.f * pidx + 1.f) - 1.f) * 0.5f);
    while ((I + 1) * (I + 2) / 2 <= pidx) ++I;
    while (I * (I + 1) / 2 > pidx) --I;
    const int J = pidx - I * (I + 1) / 2;
    const int r = 32 * I + lane;
    const int rc = min(r, m - 1);
    const int2 cr = K.code[rc + 3];
    auto row_of = [&](const float4* a) {
      const float4 f = a[rc >> 1];
      return (rc & 1) ? make_float2(f.y, f.w) : make_float2(f.x, f.z);
    };
    const float2 rz0 = row_of(nz0);
    float2 rv1 = row_of(v1), rv2 = row_of(v2), rz1 = row_of(z1), rz2 = row_of(z2);
    rv1 = make_float2(-rv1.x, -rv1.y);
    rv2 = make_float2(-rv2.x, -rv2.y);
    rz1 = make_float2(-rz1.x, -rz1.y);
    rz2 = make_float2(-rz2.x, -rz2.y);
    float2* tile = B.tile(I, J) + lane;
#pragma unroll 2
    for (int u = 0; u < 16; ++u) {
      const int c = 32 * J + 2 * u, q = c >> 1;
      float2 h = make_float2(0.f, 0.f), l = h;
      if (c < m) {  // uniform
        float2 k0 = K.get<MODE>(rc + 3, cr, c + 3), k1 = K.get<MODE>(rc + 3, cr, min(c + 4, N - 1));
        if (I == J) {  // K has a zero diagonal
          if (r == c) k0 = lam;
          if (r == c + 1) k1 = lam;
        }
        h = make_float2(k0.x, k1.x);
        l = make_float2(k0.y, k1.y);
        const float4 fz0 = nz0[q], fv1 = v1[q], fz1 = z1[q], fv2 = v2[q], fz2 = z2[q];
        df_acc_x2(make_float2(fz0.x, fz0.y), make_float2(fz0.z, fz0.w), h, l);
        df_acc_x2(make_float2(rz0.x, rz0.x), make_float2(rz0.y, rz0.y), h, l);
        df_mac_x2(rz1, make_float2(fv1.x, fv1.y), make_float2(fv1.z, fv1.w), h, l);
        df_mac_x2(rv1, make_float2(fz1.x, fz1.y), make_float2(fz1.z, fz1.w), h, l);
        df_mac_x2(rz2, make_float2(fv2.x, fv2.y), make_float2(fv2.z, fv2.w), h, l);
        df_mac_x2(rv2, make_float2(fz2.x, fz2.y), make_float2(fz2.z, fz2.w), h, l);
        df_norm_x2(h, l);
      }
      if (B.tiles) {  // padding: zeros
        __stcs(tile + (2 * u) * 32, r < m ? make_float2(h.x, l.x) : make_float2(0.f, 0.f));
        __stcs(tile + (2 * u + 1) * 32,
               r < m && c + 1 < m ? make_float2(h.y, l.y) : make_float2(0.f, 0.f));
      } else if (r < m) {
        if (c < m) B.p[(int64_t)c * B.ld + r] = make_float2(h.x, l.x);
        if (c + 1 < m) B.p[(int64_t)(c + 1) * B.ld + r] = make_float2(h.y, l.y);
        if (I != J) {
          if (c < m) B.p[(int64_t)r * B.ld + c] = make_float2(h.x, l.x);
          if (c + 1 < m) B.p[(int64_t)r * B.ld + c + 1] = make_float2(h.y, l.y);
        }
      }
    }
  }
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
// (the tiles of subdomains of at most 32 SMALL_T unknowns, 24 KB, stay in shared memory:
// with the padding to 32 they could exceed the (m + 6)^2 floats of the slot in memory)

constexpr size_t HV_OFF = 32 * 1024;  // in the panel
static_assert(CHOL_SMEM + 16 + 6 * TILE16 * sizeof(uint4) <= HV_OFF &&
                  HV_OFF + 26 * 128 * sizeof(__half) <= panel_bytes(8), "panel");

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
__device__ __forceinline__ void tile_from_B(float (&c)[2][4][4], const BPairs& B,
                                            const float* dsc, int i, int j, int lane) {
  const int g = lane >> 2, q = lane & 3;
  const int ld = B.tiles ? 32 : B.ld;
  const float2* p = (B.tiles ? B.tile(i, j) : B.p + (int64_t)(32 * j) * ld + 32 * i) + 2 * q * ld + g;
  const int rows = B.m - 32 * i - g, cols = B.m - 32 * j - 2 * q;  // left from this lane's first
  float dr[4], dc[8];
#pragma unroll
  for (int a = 0; a < 4; ++a) dr[a] = 8 * a < rows ? dsc[32 * i + g + 8 * a] : 0.f;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int cl = 8 * (b >> 1) + (b & 1);
    dc[b] = cl < cols ? dsc[32 * j + 2 * q + cl] : 0.f;
  }
#pragma unroll
  for (int b = 0; b < 8; ++b)
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int cl = 8 * (b >> 1) + (b & 1);
      const bool in = 8 * a < rows && cl < cols;
      c[a >> 1][b >> 1][2 * (a & 1) + (b & 1)] = in ? p[cl * ld + 8 * a].x : 0.f;
    }
#pragma unroll
  for (int b = 0; b < 8; ++b)
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      float& v = c[a >> 1][b >> 1][2 * (a & 1) + (b & 1)];
      v *= -dr[a] * dc[b];
      // the identity past m
      if (i == j && 8 * a >= rows && g + 8 * a == 2 * q + 8 * (b >> 1) + (b & 1)) v = -1.f;
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
__device__ __noinline__ bool chol_factor(const BPairs B, const float* dsc, uint4* LP, float* ws,
                                         int* s_flag) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int T = (B.m + 31) / 32;
  float c[2][4][4];
  if (wid == 0) {
    tile_from_B(c, B, dsc, 0, 0, lane);
    diag_inverse(c, LP, ws, lane, s_flag);
  }
  __syncthreads();
  for (int k = 0; k + 1 < T; ++k) {
    for (int i = k + 1 + wid; i < T; i += (wid == 0) ? T : NW - 1) {
      Tile16 X, Y;
      uint4* slot = LP + tile_at(i, k);
      if (k == 0) {
        tile_from_B(c, B, dsc, i, 0, lane);
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
        tile_from_B(c, B, dsc, i, i, lane);
      else
        acc_load(dslot, c, lane);
      tile_mma(c, X, X);
      if (i == k + 1) {
        diag_inverse(c, dslot, ws, lane, s_flag);
      } else {
        acc_store(dslot, c, lane);
        // column k + 1 of this row, terms j < k
        tile_from_B(c, B, dsc, i, k + 1, lane);
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

// The right-hand sides of the products: 32 rows of the two components as FP16 terms, block
// k at 128 k: (x hi, x lo, y hi, y lo), 32 each.
// The B operand (K = 32, N = 8) with the two components in its first two columns (zeros in
// the others): b[t][ks] = (b0, b1).
__device__ __forceinline__ void rhs_frags(const __half* hv, int k, int lane, uint2 (&b)[2][2]) {
  const int g = lane >> 2, q = lane & 3;
  const uint32_t* v = reinterpret_cast<const uint32_t*>(hv + 128 * k + 64 * (g & 1)) + q;
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      const uint2 w = make_uint2(v[16 * t + 8 * ks], v[16 * t + 8 * ks + 4]);
      b[t][ks] = g < 2 ? w : make_uint2(0u, 0u);
    }
}

// d[mt] = rows 16 mt + g and + 8 of X v (columns 2 q, 2 q + 1: the components are in the
// lanes q = 0); the three terms in accumulators of their own (chains of two MMAs)
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

// the rows of d (lanes q = 0) as right-hand side block k
__device__ __forceinline__ void rhs_terms(__half* hv, int k, const float (&d)[2][4], int lane) {
  if ((lane & 3) == 0) {
    __half* v = hv + 128 * k + (lane >> 2);
#pragma unroll
    for (int h = 0; h < 4; ++h)  // rows g + 8 h
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float f = d[h >> 1][2 * (h & 1) + c];
        const __half hi = __float2half_rn(f);
        v[64 * c + 8 * h] = hi;
        v[64 * c + 32 + 8 * h] = __float2half_rn(f - __half2float(hi));
      }
  }
  __syncwarp();
}

// d := rows of block k minus d
__device__ __forceinline__ void rhs_minus(const float* rx, const float* ry, int k,
                                          float (&d)[2][4], int lane) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const int i = 32 * k + (lane >> 2) + 8 * h;
    d[h >> 1][2 * (h & 1)] = rx[i] - d[h >> 1][2 * (h & 1)];
    d[h >> 1][2 * (h & 1) + 1] = ry[i] - d[h >> 1][2 * (h & 1) + 1];
  }
}
__device__ __forceinline__ void rhs_store(float* rx, float* ry, int k, const float (&d)[2][4],
                                          int lane) {
  if ((lane & 3) == 0) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int i = 32 * k + (lane >> 2) + 8 * h;
      rx[i] = d[h >> 1][2 * (h & 1)];
      ry[i] = d[h >> 1][2 * (h & 1) + 1];
    }
  }
}

// tile_vec of a tile in shared memory, its registers loaded as they are needed
__device__ __forceinline__ void tile_vec_at(float (&d)[2][4], const uint4* p, int lane,
                                            const uint2 (&b)[2][2]) {
  float t[3][2][4];
#pragma unroll
  for (int e = 0; e < 24; ++e) t[e >> 3][(e >> 2) & 1][e & 3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      const uint4 hi = p[32 * (2 * mt + ks) + lane], lo = p[32 * (4 + 2 * mt + ks) + lane];
      mma_f16(t[0][mt], lo, b[0][ks].x, b[0][ks].y);
      mma_f16(t[1][mt], hi, b[1][ks].x, b[1][ks].y);
      mma_f16(t[2][mt], hi, b[0][ks].x, b[0][ks].y);
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

// Block substitution over the tiles: forward (L y = r) or backward (L^T x = y).  Warps 0
// and 1 run the serial chain in turns: step k takes block k - 1's solution off block k and
// multiplies by the inverse of the diagonal tile, while the other of the two has its tiles
// for step k + 1 copied to shared memory (buf, 512 elements of 16 bytes each; every lane
// its own elements) and transposes them there.  Meanwhile the other warps take block
// k - 1's solution off blocks k + 1 and on (each block with its warp), the next tile loaded
// behind the products of the one before.  One barrier per step.  Solutions pass between
// the warps as FP16 terms (hv), converted once by the warp that finds them.  (One chain
// warp that also fetched its tiles and converted on every read took 2 300 cycles per step,
// 1 000 of them for this.)  buf: null when the tiles are in shared memory themselves.
template <int NT, bool BACK>
__device__ __noinline__ void tri_solve(const uint4* LP, int T, float* rx, float* ry, __half* hv,
                                       uint4* buf) {
  constexpr int NO = NT / 32 - 2;  // warps beside the chain's
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // blocks in the order of the substitution: n-th block
  auto blk = [&](int n) { return BACK ? T - 1 - n : n; };
  auto tile_of = [&](int n, int k) {  // the tile coupling block n to block k (k before n)
    return BACK ? tile_at(blk(k), blk(n)) : tile_at(blk(n), blk(k));
  };
  uint2 b[2][2];
  float d[2][4];
  if (wid < 2) {
    uint4* W = buf + wid * 2 * TILE16;
    uint4* X = W + TILE16;
    auto fetch = [&](int n) {  // start copying the tiles of step n
      if (buf == nullptr || n >= T) return;
      const uint4* w = LP + tile_at(blk(n), blk(n)) + lane;
      const uint4* x = LP + tile_of(n, n > 0 ? n - 1 : 0) + lane;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        cp_async16(W + 32 * e + lane, w + 32 * e);
        cp_async16(X + 32 * e + lane, x + 32 * e);
      }
    };
    auto ready = [&]() {
      asm volatile("cp.async.wait_all;" ::: "memory");
      if (BACK && buf != nullptr) {
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
          Tile16 t;
          t.load(W + q * TILE16, lane);
          t.transpose();
          t.store(W + q * TILE16, lane);
        }
      }
    };
    auto product = [&](const uint4* at, int tile) {
      if (buf != nullptr) {
        tile_vec_at(d, at, lane, b);
      } else {
        Tile16 t;
        t.load(LP + tile, lane);
        if (BACK) t.transpose();
        tile_vec(d, t, b);
      }
    };
    fetch(wid);
    ready();
    for (int k = 0; k < T; ++k) {
      if ((k & 1) == wid) {
        if (k > 0) {
          rhs_frags(hv, blk(k - 1), lane, b);
          product(X, tile_of(k, k - 1));
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) d[e >> 2][e & 3] = 0.f;
        }
        rhs_minus(rx, ry, blk(k), d, lane);
        rhs_terms(hv, blk(k), d, lane);
        rhs_frags(hv, blk(k), lane, b);
        product(W, tile_at(blk(k), blk(k)));
        __syncwarp();
        rhs_terms(hv, blk(k), d, lane);
        rhs_store(rx, ry, blk(k), d, lane);
        fetch(k + 2);
      } else if (k > 0) {
        ready();
      }
      __syncthreads();  // block k is published, block k - 1 is off the blocks after
    }
  } else {
    // this warp's first block from block n on
    auto first_of = [&](int n) { return n + (wid - 2 - n % NO + NO) % NO; };
    Tile16 N;
    int n0 = first_of(2);
    if (n0 < T) N.load(LP + tile_of(n0, 0), lane);
    __syncthreads();
    for (int k = 1; k < T; ++k) {
      const int n1 = first_of(k + 2);
      if (n0 < T) rhs_frags(hv, blk(k - 1), lane, b);
      for (int n = n0; n < T; n += NO) {
        if (BACK) N.transpose();
        tile_vec(d, N, b);
        if (n + NO < T)
          N.load(LP + tile_of(n + NO, k - 1), lane);
        else if (n1 < T)
          N.load(LP + tile_of(n1, k), lane);
        rhs_minus(rx, ry, blk(n), d, lane);
        __syncwarp();
        rhs_store(rx, ry, blk(n), d, lane);
      }
      n0 = n1;
      __syncthreads();
    }
  }
}

// rx, ry := D (L L^T)^-1 D of them, two right-hand sides (shared, 16-byte aligned, zero
// from m up to a multiple of 32), each scaled by a power of two to a largest value in
// [1, 2) for the FP16 terms.
template <int NT>
__device__ void chol_solve2(const uint4* LP, int m, const float* dsc, float* rx, float* ry,
                            double* sh, __half* hv,
                            uint4* buf) {
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
  tri_solve<NT, false>(LP, T, rx, ry, hv, buf);
  tri_solve<NT, true>(LP, T, rx, ry, hv, buf);
  for (int i = threadIdx.x; i < m; i += NT) {
    rx[i] = ldexpf(rx[i] * dsc[i], ex);
    ry[i] = ldexpf(ry[i] * dsc[i], ey);
  }
  __syncthreads();
}

// Systems of at most this many unknowns are refined three times at least.  The factor's 22
// bits contract the error about 4 times less than FP32's 24: what two sweeps leave is above
// the rounding of B in these.  rms error against FP64, 24 x 26 vectors 8 px apart off the
// lattice, with two sweeps, with three, and with an FP32 factor: subdomains of 40 vectors
// 2.0e-12, 3.8e-13, 7.8e-13; of 60 6.9e-12, 6.6e-13, 2.5e-12.  From 100 vectors on (most
// above 140 unknowns) two sweeps that pass are no worse than with the FP32 factor (0.91 of
// its error over steps of 4 to 32 px, smoothing 0.5 to 5).  The third sweep: 255 x 255
// vectors in subdomains of 40 885 -> 979 us.
constexpr int SETTLE = 128;

// Shared-memory layout of k_tps_solve_mp for subdomains of at most n centres.
struct MpLayout {
  int np;        // n rounded up to 32
  size_t d_off;  // doubles: V 3n, xc n, yc n, Y/C 3n, W 4n
  size_t f2_off; // float4: z, g (np each)
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
// Buffers per subdomain (offset mat_off, a multiple of 4 elements; (m + 6)^2 doubles and as
// many floats): matrices holds B22 = (Q^T A Q)[3:, 3:] as (hi, lo) float pairs, the 32 x 32
// tiles of its lower half (BPairs), and behind them, from 7 tile rows on, the residual's
// partial sums (residual_part_bytes: tiles and sums of T rows are below (32 T - 25)^2 pairs,
// the smallest slot with T rows, for T >= 7); matrices32 holds the tiles of its Cholesky
// factor (chol_factor).  Up to 32 SMALL_T unknowns B22 is whole, both triangles, leading
// dimension mp = m rounded up to 4, and the factor in shared memory.
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
  float4* z4 = reinterpret_cast<float4*>(smraw + lay.f2_off);  // (x hi, y hi, x lo, y lo)
  float4* g4 = z4 + lay.np;
  float* vx = reinterpret_cast<float*>(smraw + lay.f_off);
  float* vy = vx + lay.np;
  float* rx = vy + lay.np;
  float* ry = rx + lay.np;
  int2* cxy = reinterpret_cast<int2*>(smraw + lay.i2_off);
  float* panel = reinterpret_cast<float*>(smraw + lay.p_off);

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
  // Centres on the lattice: when the (hi, lo) kernel values of all their offsets fit the
  // panel, cxy becomes the codes of the centres' grid (lat_codes), whose differences index
  // the table; otherwise it keeps the lattice coordinates.
  KEntries K{cxy,
             reinterpret_cast<const float2*>(panel + NW * 96 * 2),
             0,
             phi_table2,
             (int)(table_size < (int64_t)INT_MAX ? table_size : (int64_t)INT_MAX),
             xc,
             yc,
             phi_table,
             table_size};
  LatCodes lx{1, 0, false}, ly{1, 0, false};
  if (lat) {
    const int2 o = cxy[0];
    int v[6], h[6];  // whole pixels; half-pixel parts
    lat_grid_init(v);
    lat_grid_init(h);
    for (int i = threadIdx.x; i < N; i += NT) {
      lat_grid_add(v, (cxy[i].x >> 1) - (o.x >> 1), (cxy[i].y >> 1) - (o.y >> 1));
      lat_grid_add(h, cxy[i].x & 1, cxy[i].y & 1);
    }
    lat_grid_block(v, reinterpret_cast<int*>(sh));
    lat_grid_block(h, reinterpret_cast<int*>(sh));
    lx = lat_codes(v[0], v[2], v[3], h[2] != h[3]);
    ly = lat_codes(v[1], v[4], v[5], h[4] != h[5]);
    if (phi_table2 != nullptr && (int64_t)lx.width * ly.width <= panel_table(NW) &&
        lat_codes_fit(lx, ly, K.tsz32)) {
      K.tw = lx.width;
      for (int i = threadIdx.x; i < N; i += NT)
        cxy[i] = make_int2(lx.code(cxy[i].x, (o.x >> 1) + v[2]),
                           ly.code(cxy[i].y, (o.y >> 1) + v[4]));
      float2* tab = const_cast<float2*>(K.tab);
      for (int e = threadIdx.x; e < lx.width * ly.width; e += NT) {
        const int b = e / lx.width, a = e - b * lx.width;
        const int dx = lx.offset(a), dy = ly.offset(b);
        tab[e] = phi_table2[dy * dy + dx * dx];
      }
    }
    __syncthreads();
  }
  const int kmode = !lat || phi_table2 == nullptr ? K_DIRECT : K.tw > 0 ? K_TABLE : K_GATHER;
  // A = K + lam I, entry (r, c), FP64; on the lattice 4 r^2 is an integer table index
  auto a_entry = [&](int r, int c) -> double {
    if (r == c) return lam;
    if (lat) {
      const int2 ca = cxy[r], cb = cxy[c];
      const int64_t dx = K.tw > 0 ? lx.coord(ca.x) - lx.coord(cb.x) : (int64_t)ca.x - cb.x;
      const int64_t dy = K.tw > 0 ? ly.coord(ca.y) - ly.coord(cb.y) : (int64_t)ca.y - cb.y;
      const int64_t kq = dy * dy + dx * dx;
      if (kq < table_size) return __ldg(phi_table + kq);
      return phi_pair(xc[r], yc[r], xc[c], yc[c], nullptr, 0);
    }
    return phi_pair(xc[r], yc[r], xc[c], yc[c], phi_table, table_size);
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
  // the pairs of V for Y, then the columns of the projection: the f2 and f regions (48 np
  // bytes) are free until the refinement
  float4* pairs = reinterpret_cast<float4*>(smraw + lay.f2_off);
  const int np = lay.np;
  for (int i = threadIdx.x; i < N; i += NT) {
    const float2 a = df_split(V1[i]), b = df_split(V2[i]);
    pairs[i] = make_float4(a.x, b.x, a.y, b.y);
  }
  __syncthreads();
  // every CTA of the cluster has started (and holds its V) before any CTA writes
  // into a peer's shared memory below
  cluster.sync();
  {
    float2* part = reinterpret_cast<float2*>(panel);
    if (kmode == K_TABLE)
      build_y<NT, K_TABLE>(K, pairs, V, V0[0], lam, N, n, YC, part);
    else if (kmode == K_GATHER)
      build_y<NT, K_GATHER>(K, pairs, V, V0[0], lam, N, n, YC, part);
    else
      build_y<NT, K_DIRECT>(K, pairs, V, V0[0], lam, N, n, YC, part);
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
    __syncthreads();
    float* pf = reinterpret_cast<float*>(pairs);
    for (int c = threadIdx.x; c < np; c += NT) {  // unknown c: row c + 3 (zero past m)
      const bool in = c < m;
      const double src[5] = {in ? -Z0[c + 3] : 0.0, in ? V1[c + 3] : 0.0, in ? V2[c + 3] : 0.0,
                             in ? Z1[c + 3] : 0.0, in ? Z2[c + 3] : 0.0};
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const float2 d = df_split(src[k]);
        float* q = pf + 4 * (k * (np / 2) + (c >> 1)) + (c & 1);
        q[0] = d.x;
        q[2] = d.y;
      }
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
  // ---- B22 in double-float
  const BPairs B{B2, m, mp, m > 32 * SMALL_T};
  {
    const float2 lam2 = df_split(lam);
    if (kmode == K_TABLE)
      build_b<NT, K_TABLE>(K, pairs, np, lam2, B, crank, csize);
    else if (kmode == K_GATHER)
      build_b<NT, K_GATHER>(K, pairs, np, lam2, B, crank, csize);
    else
      build_b<NT, K_DIRECT>(K, pairs, np, lam2, B, crank, csize);
  }
  cluster.sync();  // the cluster's B tiles are in global memory, visible to rank 0
  if (crank != 0) return;
  // ---- Cholesky factor of D B22 D (D in xc: the centres are no longer needed)
  float* dsc = reinterpret_cast<float*>(xc);
  if (threadIdx.x == 0) s_flag = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += NT) {
    const float v = B.at(i, i).x;
    if (!(v > 0.f)) s_flag = 1;
    dsc[i] = (v > 0.f) ? ldexpf(1.f, -(ilogbf(v) >> 1)) : 1.f;
  }
  __syncthreads();
  uint4* LP = (m <= 32 * SMALL_T)
                  ? reinterpret_cast<uint4*>(smraw + lay.p_off + ((CHOL_SMEM + 15) & ~(size_t)15))
                  : reinterpret_cast<uint4*>(matrices32 + mat_off[sd]);
  if (!chol_factor<NT>(B, dsc, LP, panel, &s_flag)) return;
  // the residual: staging of the warps, then the tile products, in the panel when they fit,
  // else behind the tiles of B in its slot (from 7 tile rows on (m + 6)^2 pairs hold both)
  float2* stage = reinterpret_cast<float2*>(panel);
  constexpr size_t STAGE_BYTES = (size_t)NW * 16 * 33 * sizeof(float2);
  const int nT = (m + 31) / 32;
  float4* part = (STAGE_BYTES + residual_part_bytes(nT, NW / 8) <= panel_bytes(NW))
                     ? reinterpret_cast<float4*>(smraw + lay.p_off + STAGE_BYTES)
                     : reinterpret_cast<float4*>(B2 + (size_t)1024 * (nT * (nT + 1) / 2));
  // the substitutions' right-hand sides, behind the tiles of small subdomains
  __half* hv = reinterpret_cast<__half*>(smraw + lay.p_off + HV_OFF);
  uint4* buf = (m <= 32 * SMALL_T) ? nullptr : reinterpret_cast<uint4*>(panel);

  // ---- outlier iterations with refined solves (x and y in lockstep)
  double* wx = W + 2 * n;
  double* wy = W + 3 * n;
  for (int r = threadIdx.x; r < lay.np; r += NT) {
    vx[r] = (r < N) ? ux[idx[r]] : 0.f;
    vy[r] = (r < N) ? uy[idx[r]] : 0.f;
    z4[r] = g4[r] = make_float4(0.f, 0.f, 0.f, 0.f);
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
          const float2 a = df_split(gxv), b = df_split(gyv);
          g4[i - 3] = make_float4(a.x, b.x, a.y, b.y);
        }
      }
      __syncthreads();
    }
    // refine z (B z = g): solves with the factor, double-float residuals
    bool conv = false, near = false;
    double prev = INFINITY;
    for (int it = 0; it < max_refine; ++it) {
      if (z_zero) {  // z = 0: rho = g
        for (int i = threadIdx.x; i < m; i += NT) {
          rx[i] = __fadd_rn(g4[i].x, g4[i].z);
          ry[i] = __fadd_rn(g4[i].y, g4[i].w);
        }
        __syncthreads();
        z_zero = false;
      } else {
        if (B.tiles)
          residual_tiles<NT>(B, z4, g4, rx, ry, part, stage);
        else
          residual_small<NT>(B, z4, g4, rx, ry);
      }
      chol_solve2<NT>(LP, m, dsc, rx, ry, sh, hv, buf);
      ++nsweeps;
      float dm = 0.f, zm = 0.f;
      for (int i = threadIdx.x; i < m; i += NT) {
        const float4 zv = z4[i];
        float2 zh = make_float2(zv.x, zv.y), zl = make_float2(zv.z, zv.w);
        df_acc_x2(make_float2(done[0] ? 0.f : rx[i], done[1] ? 0.f : ry[i]),
                  make_float2(0.f, 0.f), zh, zl);
        df_norm_x2(zh, zl);
        z4[i] = make_float4(zh.x, zh.y, zl.x, zl.y);
        // (beyond the FP16 range of the factor's products the corrections are not finite:
        // their bits compare as the largest)
        const unsigned ax = done[0] ? 0u : __float_as_uint(fabsf(rx[i]));
        const unsigned ay = done[1] ? 0u : __float_as_uint(fabsf(ry[i]));
        dm = __uint_as_float(max(__float_as_uint(dm), max(ax, ay)));
        zm = fmaxf(zm, fmaxf(fabsf(zh.x), fabsf(zh.y)));
      }
      const float2 dz = block_max2<NT>(dm, zm, sh);
      if (!(dz.x < INFINITY)) break;  // the FP64 LU takes over
      const double dmax = (double)dz.x, zmax = (double)dz.y;
      if (dmax == 0.0) {
        conv = true;
        break;
      }
      if (it >= 1) {
        // contraction of the preconditioned refinement, estimated from the last two
        // corrections; the remaining error is about contraction * dmax.  4e-11 of z: the
        // field then carries the rounding of B, not the refinement's (2e-11 to 8e-11
        // relative against FP64 LU; 4e-11 to 1.6e-10 at 1e-10, for 1-2 % less time).  In
        // small systems the rounding of B is below that, so they take three sweeps at
        // least (SETTLE).
        const double rho = dmax / prev;
        near = near || (rho < 0.1 && rho * dmax <= 4e-11 * zmax);
        if (near && it >= (m <= SETTLE ? 2 : 1)) {
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
        const float4 zv = z4[i];
        const double zxv = (double)zv.x + (double)zv.z, zyv = (double)zv.y + (double)zv.w;
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
        const float4 zv = i < 3 ? make_float4(0.f, 0.f, 0.f, 0.f) : z4[i - 3];
        double a = (double)zv.x + (double)zv.z, b = (double)zv.y + (double)zv.w;
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
