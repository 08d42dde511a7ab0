// Grids of the half-integer lattice.  Window centres (and the positions a field is
// interpolated at) are lattice points (2x, 2y integers) on regular grids, so the
// distances between two of them take few values: with g the greatest common divisor
// of the offsets from an origin along an axis, every offset is g times a small
// integer, and the kernel value of a pair depends only on the two integer offsets.
// A block finds g and the extent of its points, per axis, with this reduction, and
// keeps the kernel values of every offset of that extent in shared memory instead of
// gathering them from the lattice table in memory, one sector per pair.
#pragma once

#include <cuda_runtime.h>

#include <climits>

namespace fi {

__device__ __forceinline__ unsigned gcd_u32(unsigned a, unsigned b) {
  while (b != 0u) {
    const unsigned t = a % b;
    a = b;
    b = t;
  }
  return a;
}

// Accumulates the lattice offset (dx, dy) into v = {gcd |dx|, gcd |dy|, min dx,
// max dx, min dy, max dy} (start from lat_grid_init).
__device__ __forceinline__ void lat_grid_init(int (&v)[6]) {
  v[0] = v[1] = 0;
  v[2] = v[4] = INT_MAX;
  v[3] = v[5] = INT_MIN;
}

__device__ __forceinline__ void lat_grid_add(int (&v)[6], int dx, int dy) {
  v[0] = (int)gcd_u32((unsigned)v[0], (unsigned)(dx < 0 ? -dx : dx));
  v[1] = (int)gcd_u32((unsigned)v[1], (unsigned)(dy < 0 ? -dy : dy));
  v[2] = min(v[2], dx);
  v[3] = max(v[3], dx);
  v[4] = min(v[4], dy);
  v[5] = max(v[5], dy);
}

__device__ __forceinline__ void lat_grid_merge(int (&v)[6], const int (&w)[6]) {
  v[0] = (int)gcd_u32((unsigned)v[0], (unsigned)w[0]);
  v[1] = (int)gcd_u32((unsigned)v[1], (unsigned)w[1]);
  v[2] = min(v[2], w[2]);
  v[3] = max(v[3], w[3]);
  v[4] = min(v[4], w[4]);
  v[5] = max(v[5], w[5]);
}

// Block-wide merge of every thread's v; every thread returns with the result.
// scratch: 6 ints per warp of the block (at most 32 warps), not otherwise in use
// between the two barriers of this call.
__device__ __forceinline__ void lat_grid_block(int (&v)[6], int* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  for (int o = 16; o > 0; o >>= 1) {
    int w[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = __shfl_xor_sync(0xffffffffu, v[k], o);
    lat_grid_merge(v, w);
  }
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 6; ++k) scratch[6 * wid + k] = v[k];
  }
  __syncthreads();
  lat_grid_init(v);
  for (int q = 0; q < nw; ++q) {
    int w[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = scratch[6 * q + k];
    lat_grid_merge(v, w);
  }
  __syncthreads();
}

// Codes of lattice coordinates along one axis.  With a coordinate 2 p + e in half pixels
// (e = 0, 1) and whole pixels p = p_min + g a, the offset of two points is 2 g k + s with
// s = -1, 0, 1: points on the grid of step g, or half a pixel off it (the midpoints of odd
// window shifts).  The codes 3 a + e differ by 3 k + s, so a table of one entry per code
// difference holds every offset; when every e is the same (half = false) the codes are a.
struct LatCodes {
  int g, width;  // step in pixels, number of code differences 0 .. width - 1
  bool half;
  __device__ __forceinline__ int code(int c, int p_min) const {
    const int a = ((c >> 1) - p_min) / g;
    return half ? 3 * a + (c & 1) : a;
  }
  // the offset (half pixels, >= 0) of a code difference d >= 0
  __device__ __forceinline__ int offset(int d) const {
    if (!half) return 2 * g * d;
    const int k = (d + 1) / 3;
    return 2 * g * k + (d - 3 * k);
  }
  // a coordinate (half pixels, from the smallest) of a code
  __device__ __forceinline__ int coord(int c) const {
    return half ? 2 * g * (c / 3) + c % 3 : 2 * g * c;
  }
};

// From the reduced whole pixels (their gcd and extremes, lat_grid_*).
__device__ __forceinline__ LatCodes lat_codes(int gcd, int pmin, int pmax, bool half) {
  LatCodes c;
  c.g = gcd > 0 ? gcd : 1;
  c.half = half;
  // (extents beyond 2^15 pixels fail lat_codes_fit: the width saturates)
  const int64_t a = pmin <= pmax ? ((int64_t)pmax - pmin) / c.g : INT_MAX;
  const int64_t w = half ? 3 * a + 2 : a + 1;
  c.width = (int)(w < (1 << 20) ? w : (1 << 20));
  return c;
}

// Whether every offset's 4 r^2 is a 32-bit index below `tsize` (then no pair of the grid
// falls beyond the lattice table).
__device__ __forceinline__ bool lat_codes_fit(const LatCodes& x, const LatCodes& y, int tsize) {
  if (x.width >= (1 << 20) || y.width >= (1 << 20)) return false;
  const int64_t ex = 2 * (int64_t)x.g * ((x.width + 1) / (x.half ? 3 : 1)) + 1;
  const int64_t ey = 2 * (int64_t)y.g * ((y.width + 1) / (y.half ? 3 : 1)) + 1;
  return ex <= 32767 && ey <= 32767 && ex * ex + ey * ey < (int64_t)tsize;
}

}  // namespace fi
