// Rank filters (minimum / maximum / median / percentile) over a box window of a stack of
// images (nt, ny, nx), with the boundary modes of scipy.ndimage ('reflect', 'mirror',
// 'nearest', 'wrap', 'constant'), window [i - s//2, i - s//2 + s - 1] along each axis,
// and img - weight * filtered of the background removal tools
// (works/preproc/_toolbox_py.py:66-155, 189-256) in the same pass.
//
// Values are compared through order-preserving integer keys (key_of): every result is
// exact for every type.  Which kernel runs:
//   minimum and maximum of 2-D windows: k_minmax_tile (separable, tiles in shared memory)
//   any rank of a window along time only: k_time_rank (a pixel's frames in shared memory)
//   other ranks of 2-D windows up to 32 x 32 of 8, 16 and 32 bit types: k_rank_planes where
//   planes_pay
//   other ranks of 2-D windows: k_rank_select_tile while the tile fits
//   the rest (3-D windows, float64 medians): k_minmax_axis, k_rank_select
#include <cstdint>
#include <cstring>

#include "fi_common.cuh"
#include "fi_pre.cuh"

namespace fi {

// What becomes of the filtered key of element e: stored, or img - weight * filtered.
struct RankOut {
  void* out;
  const void* img;  // null: the filtered values themselves
  int dtype;
  Subtract sub;
  __device__ __forceinline__ void put(int64_t e, uint64_t k) const {
    if (img == nullptr)
      store_key(out, dtype, e, k);
    else
      sub.store_keys(out, e, key_of(img, dtype, e), k);
  }
};

// ------------------------------------------------------------------ min / max
// Minimum or maximum over a 2-D window, one output tile per block: the keys of the tile
// and its halo in shared memory (complemented for a maximum, so that both are minima),
// then along each axis the minima of 2, 4, ... p values (p the largest power of two in
// the window) in place of one buffer into the other, and the window as two overlapping
// runs of p.  A 30 x 30 window takes 5 + 5 minima per element instead of 30 + 30 loads of
// 64-bit keys from memory in three passes: 4 frames of 512^2 u8 with the subtraction
// 140 -> 36 us a call.  The kernel takes most of it, by the latency of its steps (a barrier
// between each two of 12): warps 39 % of the most, issue 46 % of the slots, DRAM 0.4 %.
constexpr int MM_TX = 64, MM_TY = 32, MM_NT = 256;
constexpr size_t MM_MAX_SMEM = 160 * 1024;

inline size_t minmax_tile_bytes(int sy, int sx, int key_bytes) {
  return (size_t)2 * (MM_TX + sx - 1) * (MM_TY + sy - 1) * key_bytes;
}

template <typename K>
__global__ void __launch_bounds__(MM_NT)
    k_minmax_tile(const void* in, int dtype, int64_t ny, int64_t nx, int sy, int sx, int mode,
                  uint64_t ckey, int is_max, RankOut ro) {
  extern __shared__ __align__(16) unsigned char mm_smem[];
  const int pw = MM_TX + sx - 1, ph = MM_TY + sy - 1;
  K* a = reinterpret_cast<K*>(mm_smem);
  K* b = a + pw * ph;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.z * ny * nx;
  const int64_t x0 = (int64_t)blockIdx.x * MM_TX, y0 = (int64_t)blockIdx.y * MM_TY;
  const K flip = is_max ? (K)~(K)0 : (K)0;
  for (int r = wid; r < ph; r += MM_NT / 32) {
    const int64_t yc = extend(y0 - sy / 2 + r, ny, mode);
    for (int c = lane; c < pw; c += 32) {
      const int64_t xc = extend(x0 - sx / 2 + c, nx, mode);
      const uint64_t k = (yc < 0 || xc < 0) ? ckey : key_of(in, dtype, base + yc * nx + xc);
      a[r * pw + c] = (K)k ^ flip;
    }
  }
  __syncthreads();
  // along a row, then along a column: values at distance `step` elements
  int p = 1;
  for (; 2 * p <= sx; p *= 2) {
    for (int r = wid; r < ph; r += MM_NT / 32)
      for (int c = lane; c + p < pw; c += 32) {
        const K u = a[r * pw + c], v = a[r * pw + c + p];
        b[r * pw + c] = u < v ? u : v;
      }
    __syncthreads();
    K* t = a;
    a = b;
    b = t;
  }
  for (int r = wid; r < ph; r += MM_NT / 32)
    for (int c = lane; c < MM_TX; c += 32) {
      const K u = a[r * pw + c], v = a[r * pw + c + sx - p];
      b[r * pw + c] = u < v ? u : v;
    }
  __syncthreads();
  K* t0 = a;
  a = b;
  b = t0;
  for (p = 1; 2 * p <= sy; p *= 2) {
    for (int r = wid; r + p < ph; r += MM_NT / 32)
      for (int c = lane; c < MM_TX; c += 32) {
        const K u = a[r * pw + c], v = a[(r + p) * pw + c];
        b[r * pw + c] = u < v ? u : v;
      }
    __syncthreads();
    K* t = a;
    a = b;
    b = t;
  }
  for (int r = wid; r < MM_TY; r += MM_NT / 32)
    for (int c = lane; c < MM_TX; c += 32) {
      const int64_t y = y0 + r, x = x0 + c;
      if (y >= ny || x >= nx) continue;
      const K u = a[r * pw + c], v = a[(r + sy - p) * pw + c];
      ro.put(base + y * nx + x, (uint64_t)(K)((u < v ? u : v) ^ flip));
    }
}

// One axis of a separable minimum or maximum filter over a (nt, ny, nx) stack (the
// windows k_minmax_tile and k_time_rank do not take).  Keys compare like the values; cval
// enters as its key.
__global__ void k_minmax_axis(const void* in, int in_is_key, const uint64_t* kin, int dtype,
                              int64_t nt, int64_t ny, int64_t nx, int axis, int size, int mode,
                              uint64_t ckey, int is_max, uint64_t* kout) {
  const int64_t total = nt * ny * nx;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = e % nx, y = (e / nx) % ny, t = e / (nx * ny);
    const int64_t n = axis == 0 ? nt : axis == 1 ? ny : nx;
    const int64_t pos = axis == 0 ? t : axis == 1 ? y : x;
    const int64_t stride = axis == 0 ? ny * nx : axis == 1 ? nx : 1;
    const int64_t base = e - pos * stride;
    uint64_t best = is_max ? 0ull : ~0ull;
    const int64_t s0 = pos - size / 2;
    for (int k = 0; k < size; ++k) {
      const int64_t j = extend(s0 + k, n, mode);
      const uint64_t v = (j < 0) ? ckey : (in_is_key ? kin[base + j * stride]
                                                      : key_of(in, dtype, base + j * stride));
      best = is_max ? (v > best ? v : best) : (v < best ? v : best);
    }
    kout[e] = best;
  }
}

__global__ void k_keys_out(const uint64_t* k, int64_t count, RankOut ro) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < count;
       e += (int64_t)gridDim.x * blockDim.x)
    ro.put(e, k[e]);
}

// ------------------------------------------------------------------ along time
// Any rank of a window along time only: a thread keeps its pixel's frames in shared
// memory, so that the stack is read once and written once.  8 and 16 bit types take four
// or two pixels per thread (one 32-bit word per frame; V pixels of E bits): minima and
// maxima by packed instructions, other ranks by a radix select over the bits in which the
// pixel's frames differ.  The minimum over 8 frames of 2048^2 u16 with the subtraction
// 1666 -> 80 us (three axis passes over 64-bit keys, a conversion and the subtraction
// before); bound by issue, 84 % of the slots, with DRAM at 43 %.  A thread's output frames are a serial chain, so where the pixels do not fill
// the chip the frames are dealt to blockIdx.y, `span` each (every block reads all frames):
// medians over all frames, whole call, 95 frames of 16^2 u8 5085 -> 71 us, 90 of 48^2 u16
// 5022 -> 127 us, 40 of 64^2 f32 910 -> 144 us (k_rank_select, one thread per value: 342,
// 1447 and 1194 us).
constexpr int TIME_NT = 256;
constexpr size_t TIME_MAX_SMEM = 96 * 1024;

template <typename W>
inline size_t time_bytes(int nt, int st) {
  return (size_t)nt * TIME_NT * sizeof(W) + (size_t)(nt + st) * sizeof(int);
}

// E: bits of a packed element (8, 16), or 0: one key per word; SPLIT: frames dealt to
// blockIdx.y (with the general bounds the unsplit launch is 2 % slower)
template <typename W, int E, bool SPLIT>
__global__ void __launch_bounds__(TIME_NT)
    k_time_rank(const void* in, int dtype, int nt, int64_t npix, int st, int rank, int mode,
                uint64_t ckey, int span, RankOut ro) {
  constexpr int V = E == 8 ? 4 : E == 16 ? 2 : 1;
  const int t_lo = SPLIT ? blockIdx.y * span : 0, t_hi = SPLIT ? min(nt, t_lo + span) : nt;
  extern __shared__ __align__(16) unsigned char tm_smem[];
  W* col = reinterpret_cast<W*>(tm_smem) + threadIdx.x;
  int* at = reinterpret_cast<int*>(reinterpret_cast<W*>(tm_smem) + (size_t)nt * TIME_NT);
  for (int k = threadIdx.x; k < nt + st - 1; k += TIME_NT)
    at[k] = (int)extend((int64_t)k - st / 2, nt, mode);
  __syncthreads();
  const bool is_min = rank == 0, is_max = rank == st - 1;
  W cw = (W)ckey;  // cval in every packed element
  if (E == 8) cw = (W)((uint32_t)ckey * 0x01010101u);
  if (E == 16) cw = (W)((uint32_t)ckey * 0x00010001u);
  const int64_t words = npix / V;
  for (int64_t w0 = (int64_t)blockIdx.x * TIME_NT; w0 < words; w0 += (int64_t)gridDim.x * TIME_NT) {
    const int64_t w = w0 + threadIdx.x;
    if (w >= words) break;
#pragma unroll 8
    for (int t = 0; t < nt; ++t)
      col[t * TIME_NT] = E != 0 ? (W)__ldg(static_cast<const uint32_t*>(in) + t * words + w)
                                : (W)key_of(in, dtype, t * npix + w);
    W differ = 0, all = 0;  // bits in which the frames (and cval) differ
    if (!is_min && !is_max) {
      W lo = ~(W)0, hi = 0;
      for (int t = 0; t < nt; ++t) {
        lo &= col[t * TIME_NT];
        hi |= col[t * TIME_NT];
      }
      if (mode == FI_MODE_CONSTANT) {
        lo &= cw;
        hi |= cw;
      }
      differ = lo ^ hi;
      all = lo;
    }
    for (int t = t_lo; t < t_hi; ++t) {
      W f;
      if (is_min || is_max) {
        f = is_max ? (W)0 : ~(W)0;
        for (int k = 0; k < st; ++k) {
          const int j = at[t + k];
          const W v = j < 0 ? cw : col[j * TIME_NT];
          if (E == 8)
            f = is_max ? __vmaxu4((uint32_t)f, (uint32_t)v) : __vminu4((uint32_t)f, (uint32_t)v);
          else if (E == 16)
            f = is_max ? __vmaxu2((uint32_t)f, (uint32_t)v) : __vminu2((uint32_t)f, (uint32_t)v);
          else
            f = is_max ? (v > f ? v : f) : (v < f ? v : f);
        }
      } else {
        f = 0;
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const int sh = E * q;
          const W em = E == 0 ? ~(W)0 : (W)((((uint32_t)1 << (E == 0 ? 1 : E)) - 1) << sh);
          W prefix = all & em & ~differ, seen = em & ~differ;  // the bits decided so far
          // (bits equal in every frame above the first that differs are decided; below it
          // they enter as the select passes them)
          W left = differ & em;
          int r = rank;
          while (left != 0) {
            const int b = sizeof(W) == 8 ? 63 - __clzll((long long)left)
                                         : 31 - __clz((int)(uint32_t)left);
            const W bit = (W)1 << b;
            int zeros = 0;
            for (int k = 0; k < st; ++k) {
              const int j = at[t + k];
              const W v = j < 0 ? cw : col[j * TIME_NT];
              zeros += ((v & (seen | bit)) == prefix) ? 1 : 0;
            }
            if (r >= zeros) {
              r -= zeros;
              prefix |= bit;
            }
            seen |= bit;
            left &= ~bit;
          }
          f |= prefix;
        }
      }
      const int64_t e = t * npix + w * V;
      if (ro.img == nullptr) {
        if (E != 0)
          static_cast<uint32_t*>(ro.out)[t * words + w] = (uint32_t)f;
        else
          store_key(ro.out, dtype, e, (uint64_t)f);
      } else if (E != 0) {
        const uint32_t a = (uint32_t)col[t * TIME_NT];
        if (ro.sub.exact_int) {
          constexpr uint32_t M = E == 8 ? 0xffu : 0xffffu;
          double2* o = reinterpret_cast<double2*>(static_cast<double*>(ro.out) + e);
#pragma unroll
          for (int q = 0; q < V / 2; ++q)
            o[q] = make_double2(
                ro.sub.of_ints((int)((a >> (2 * q * E)) & M), (int)(((uint32_t)f >> (2 * q * E)) & M)),
                ro.sub.of_ints((int)((a >> ((2 * q + 1) * E)) & M),
                               (int)(((uint32_t)f >> ((2 * q + 1) * E)) & M)));
        } else {
          constexpr uint32_t M = E == 8 ? 0xffu : 0xffffu;
#pragma unroll
          for (int q = 0; q < V; ++q)
            ro.sub.store_keys(ro.out, e + q, (a >> (q * E)) & M, ((uint32_t)f >> (q * E)) & M);
        }
      } else {
        ro.sub.store_keys(ro.out, e, (uint64_t)col[t * TIME_NT], (uint64_t)f);
      }
    }
  }
}

// ------------------------------------------------------------------ rank select
// The rank-th smallest value of 2-D windows up to 32 x 32, a 32 x 32 output tile per warp.
// The tile with its halo (at most 63 x 63 keys) is kept as bit planes: two 32-bit words
// per row and bit.  The count of a window's values in a set given as such a bit image
// takes one funnel shift and one population count per row, so a radix select descends the
// tree of key prefixes for the whole tile at once: at a node (the values with a prefix,
// the pixels whose result has it) the values with a 0 at the next bit are counted for
// every pixel by running sums down the columns, and the pixels go to the two children.
// Pixels of a tile share prefixes (a median varies slowly), and nodes with few pixels are
// finished one pixel at a time, the window's rows over the lanes (one reduction per bit),
// so that even unrelated values cost at most that.  2048^2 u16, 30 x 30: 9160 -> 524 us
// (a thread per pixel counting its 900 values for every bit before).  Bound by the latency
// of a warp's dependent steps: shared memory leaves 12 warps an SM at 16 bits, issue 29 % of
// the slots, L1 23 %.
constexpr int RP_T = 32;            // tile edge
constexpr int RP_ROWS = 64;         // rows of the tile with its halo, at most
constexpr int RP_LD = RP_ROWS + 1;  // row stride of the planes (a row's planes are written
                                    // by different lanes: different banks)
constexpr int RP_MAX_WINDOW = 32;
constexpr int RP_FEW = 40;          // pixels of a node that are finished one by one
constexpr int RP_WARPS = 4;

struct RpSmem {  // offsets of a warp's shared memory for keys of `bits` bits
  size_t planes, sums, res, mask, stack, bytes;
  __host__ __device__ explicit RpSmem(int bits) {
    planes = 0;                                             // uint2 [bits][65]
    sums = planes + (((size_t)bits * RP_LD * 8 + 15) & ~(size_t)15);           // uint16 [64][32]
    res = sums + (size_t)RP_ROWS * RP_T * 2;                // uint32 [32][32]
    mask = res + (size_t)RP_T * RP_T * 4;                   // uint2 [64]
    stack = mask + (size_t)RP_ROWS * 8;                     // uint32 [bits][32]
    bytes = stack + (size_t)bits * RP_T * 4;
  }
};

template <int BITS>
__global__ void __launch_bounds__(32 * RP_WARPS)
    k_rank_planes(const void* in, int dtype, int64_t ny, int64_t nx, int sy, int sx, int rank,
                  int mode, uint32_t ckey, int tiles_x, int tiles, RankOut ro) {
  extern __shared__ __align__(16) unsigned char rp_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int tile = blockIdx.x * RP_WARPS + wid;
  if (tile >= tiles) return;
  const unsigned full = 0xffffffffu;
  const RpSmem lay(BITS);
  unsigned char* sm = rp_smem + wid * lay.bytes;
  uint2* planes = reinterpret_cast<uint2*>(sm + lay.planes);
  uint16_t* sums = reinterpret_cast<uint16_t*>(sm + lay.sums);
  uint32_t* res = reinterpret_cast<uint32_t*>(sm + lay.res);
  uint2* mask = reinterpret_cast<uint2*>(sm + lay.mask);
  uint32_t* stack = reinterpret_cast<uint32_t*>(sm + lay.stack);
  const int64_t base = (int64_t)blockIdx.z * ny * nx;
  const int64_t x0 = (int64_t)(tile % tiles_x) * RP_T, y0 = (int64_t)(tile / tiles_x) * RP_T;
  const int rows = RP_T + sy - 1;
  const unsigned wmask = sx == 32 ? full : (1u << sx) - 1u;
  // ---- bit planes (columns past the halo hold a copy of the last one: never counted)
  uint32_t any = 0u, common = full;
  {
    const int64_t xa = extend(x0 - sx / 2 + lane, nx, mode);
    const int64_t xb = extend(x0 - sx / 2 + min(32 + lane, RP_T + sx - 2), nx, mode);
    for (int r = 0; r < rows; ++r) {
      const int64_t yc = extend(y0 - sy / 2 + r, ny, mode);
      const uint32_t ka = (yc < 0 || xa < 0) ? ckey : (uint32_t)key_of(in, dtype, base + yc * nx + xa);
      const uint32_t kb = (yc < 0 || xb < 0) ? ckey : (uint32_t)key_of(in, dtype, base + yc * nx + xb);
      any |= ka | kb;
      common &= ka & kb;
      uint2 mine = make_uint2(0u, 0u);  // lane b: plane b of this row
#pragma unroll
      for (int b = 0; b < BITS; ++b) {
        const unsigned wa = __ballot_sync(full, (ka >> b) & 1u);
        const unsigned wb = __ballot_sync(full, (kb >> b) & 1u);
        if (lane == b) mine = make_uint2(wa, wb);
      }
      if (lane < BITS) planes[lane * RP_LD + r] = mine;
    }
  }
  any = __reduce_or_sync(full, any);
  common = __reduce_and_sync(full, common);
  const uint32_t differ = any ^ common;  // bits that are not the same in the whole tile
  // pixels of this lane's column: bit y = row y; their remaining rank, later their result
  unsigned members = 0u;
  if (x0 + lane < nx) {
    const int h = (int)min((int64_t)RP_T, ny - y0);
    members = h == 32 ? full : (1u << h) - 1u;
  }
  for (int y = 0; y < RP_T; ++y) res[y * RP_T + lane] = (uint32_t)rank;
  __syncwarp();
  // ---- descent: depth-first over the prefixes, the 1-children's members on the stack
  uint32_t prefix = common;     // the bits decided so far (equal bits included)
  uint32_t left = differ;       // bits not decided at the current node
  unsigned pending = 0u;        // bits whose 1-child waits on the stack
  while (true) {
    bool done = false;
    int few = 0;
    if (left != 0u) {
      few = __reduce_add_sync(full, __popc(members));
      done = few <= RP_FEW;
    }
    if (left == 0u) {  // one value: the members' result
      unsigned m = members;
      while (m) {
        const int y = __ffs((int)m) - 1;
        m &= m - 1u;
        res[y * RP_T + lane] = prefix;
      }
      done = true;
    } else {
      // the node's values: rows `lane` and `lane + 32`, those with the prefix's decided bits
      uint2 e0 = make_uint2(full, full), e1 = e0;
      for (uint32_t d = differ & ~left; d != 0u; d &= d - 1u) {
        const int b = __ffs((int)d) - 1;
        const uint2 p0 = planes[b * RP_LD + lane], p1 = planes[b * RP_LD + 32 + lane];
        const unsigned flip = ((prefix >> b) & 1u) ? 0u : full;
        e0.x &= p0.x ^ flip;
        e0.y &= p0.y ^ flip;
        e1.x &= p1.x ^ flip;
        e1.y &= p1.y ^ flip;
      }
      if (lane >= rows) e0 = make_uint2(0u, 0u);
      if (lane + 32 >= rows) e1 = make_uint2(0u, 0u);
      if (done) {  // few pixels: one by one, the window's rows over the lanes
        unsigned cols = __ballot_sync(full, members != 0u);
        while (cols) {
          const int c = __ffs((int)cols) - 1;
          cols &= cols - 1u;
          unsigned m = __shfl_sync(full, members, c);
          while (m) {
            const int y = __ffs((int)m) - 1;
            m &= m - 1u;
            int r = (int)res[y * RP_T + c];
            unsigned w0 = __funnelshift_r(e0.x, e0.y, c) & wmask;
            unsigned w1 = __funnelshift_r(e1.x, e1.y, c) & wmask;
            if (lane < y || lane >= y + sy) w0 = 0u;
            if (lane + 32 < y || lane + 32 >= y + sy) w1 = 0u;
            uint32_t v = prefix;
            for (uint32_t d = left; d != 0u;) {
              const int b = 31 - __clz((int)d);
              d &= ~(1u << b);
              const uint2 p0 = planes[b * RP_LD + lane], p1 = planes[b * RP_LD + 32 + lane];
              const unsigned q0 = __funnelshift_r(p0.x, p0.y, c);
              const unsigned q1 = __funnelshift_r(p1.x, p1.y, c);
              const int zeros = __reduce_add_sync(full, __popc(w0 & ~q0) + __popc(w1 & ~q1));
              const unsigned flip = r >= zeros ? 0u : full;
              if (r >= zeros) {
                r -= zeros;
                v |= 1u << b;
              }
              w0 &= q0 ^ flip;
              w1 &= q1 ^ flip;
            }
            __syncwarp();
            if (lane == 0) res[y * RP_T + c] = v;
          }
        }
        __syncwarp();
      } else {
        const int b = 31 - __clz((int)left);
        const uint2 p0 = planes[b * RP_LD + lane], p1 = planes[b * RP_LD + 32 + lane];
        const uint2 z0 = make_uint2(e0.x & ~p0.x, e0.y & ~p0.y);
        const uint2 z1 = make_uint2(e1.x & ~p1.x, e1.y & ~p1.y);
        const bool some0 = __any_sync(full, (z0.x | z0.y | z1.x | z1.y) != 0u);
        const bool some1 = __any_sync(full, ((e0.x & p0.x) | (e0.y & p0.y) | (e1.x & p1.x) |
                                             (e1.y & p1.y)) != 0u);
        left &= ~(1u << b);
        unsigned ones = 0u;  // members that go to the 1-child
        if (!some0) {
          ones = members;
        } else if (some1) {
          mask[lane] = z0;
          mask[32 + lane] = z1;
          __syncwarp();
          int s = 0;
#pragma unroll 4
          for (int r = 0; r < rows; ++r) {
            const uint2 w = mask[r];
            s += __popc(__funnelshift_r(w.x, w.y, lane) & wmask);
            sums[r * RP_T + lane] = (uint16_t)s;  // modulo 2^16: differences are exact
          }
#pragma unroll 4
          for (int y = 0; y < RP_T; ++y) {
            const int hi = sums[(y + sy - 1) * RP_T + lane];
            const int lo = y > 0 ? sums[(y - 1) * RP_T + lane] : 0;
            const int zeros = (hi - lo) & 0xffff;
            const int r = (int)res[y * RP_T + lane];
            if (((members >> y) & 1u) && r >= zeros) {
              ones |= 1u << y;
              res[y * RP_T + lane] = (uint32_t)(r - zeros);
            }
          }
          __syncwarp();
        }
        const unsigned zer = members & ~ones;
        const bool go0 = __any_sync(full, zer != 0u), go1 = __any_sync(full, ones != 0u);
        if (go0 && go1) {  // the 0-child first, the 1-child waits
          stack[b * RP_T + lane] = ones;
          pending |= 1u << b;
          members = zer;
        } else if (go1) {
          prefix |= 1u << b;
          members = ones;
        }
      }
    }
    if (done) {
      if (pending == 0u) break;
      // the lowest waiting bit is the deepest node
      const int b = __ffs((int)pending) - 1;
      pending &= pending - 1u;
      members = stack[b * RP_T + lane];
      const uint32_t below = (1u << b) - 1u;
      left = differ & below;
      prefix = (prefix & ~(differ & below)) | (1u << b);
    }
  }
  __syncwarp();
  for (int y = 0; y < RP_T; ++y)
    if (y0 + y < ny && x0 + lane < nx) ro.put(base + (y0 + y) * nx + x0 + lane, res[y * RP_T + lane]);
}

// The rank-th smallest value of each box window, by a radix select over the keys
// (most significant bit first): per bit, count the window values whose key shares
// the prefix found so far and has a 0 at this bit.
__global__ void k_rank_select(const void* in, int dtype, int64_t nt, int64_t ny, int64_t nx,
                              int st, int sy, int sx, int rank, int mode, uint64_t ckey,
                              RankOut ro) {
  const int64_t total = nt * ny * nx;
  const int bits = key_bits(dtype);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = e % nx, y = (e / nx) % ny, t = e / (nx * ny);
    const int64_t t0 = t - st / 2, y0 = y - sy / 2, x0 = x - sx / 2;
    uint64_t prefix = 0;
    int r = rank;
    for (int b = bits - 1; b >= 0; --b) {
      const uint64_t hi_mask = (b == 63) ? 0ull : (~0ull << (b + 1));
      int zeros = 0;
      for (int a = 0; a < st; ++a) {
        const int64_t ta = extend(t0 + a, nt, mode);
        for (int c = 0; c < sy; ++c) {
          const int64_t yc = extend(y0 + c, ny, mode);
          for (int d = 0; d < sx; ++d) {
            const int64_t xd = extend(x0 + d, nx, mode);
            const uint64_t v = (ta < 0 || yc < 0 || xd < 0)
                                   ? ckey
                                   : key_of(in, dtype, (ta * ny + yc) * nx + xd);
            if ((v & hi_mask) == prefix && !((v >> b) & 1ull)) ++zeros;
          }
        }
      }
      if (r >= zeros) {
        r -= zeros;
        prefix |= (1ull << b);
      }
    }
    ro.put(e, prefix);
  }
}

// The same for 2-D windows (st == 1) of integer and float32 images wider or taller than
// k_rank_planes takes, by tiles: a block stages its output tile plus the window halo
// (boundary extension applied once per staged element) as 32-bit keys in shared memory,
// then each thread runs the radix select over its window there; the select starts at the
// highest key bit set in the tile (higher bits are zero for every staged value).  Bound by
// the loads of the loop over the window, which runs slower with the result's conversion and
// subtraction in the same function (put_apart): medians of 1024^2 f32, 7, 10 and 15 px 567,
// 887 and 1938 us so, 479, 842 and 1750 us apart.
// NARROW (windows up to 5 px wide): the values with the prefix and a 0 at bit b as the range
// [prefix, prefix + 2^b), one comparison a value: 1024^2 f32 3 px 148 -> 138 us, 5 px 278 and
// 277; from 7 px on the form of two tests is faster (10 px 888 against 842 us).
constexpr int RS_TX = 32, RS_TY = 16;
constexpr int RS_MAX_SMEM = 96 * 1024;

static __device__ __noinline__ void put_apart(const RankOut& ro, int64_t e, uint32_t key) {
  ro.put(e, key);
}

template <bool NARROW>
__global__ void __launch_bounds__(RS_TX * RS_TY)
    k_rank_select_tile(const void* in, int dtype, int64_t ny, int64_t nx, int sy, int sx,
                       int rank, int mode, uint32_t ckey, RankOut ro) {
  extern __shared__ uint32_t patch[];
  __shared__ uint32_t s_or;
  const int pw = RS_TX + sx - 1, ph = RS_TY + sy - 1;
  const int64_t t = blockIdx.z;
  const int64_t x00 = (int64_t)blockIdx.x * RS_TX - sx / 2;
  const int64_t y00 = (int64_t)blockIdx.y * RS_TY - sy / 2;
  const int tid = threadIdx.y * RS_TX + threadIdx.x;
  if (tid == 0) s_or = 0u;
  __syncthreads();
  uint32_t acc_or = 0u;
  for (int e = tid; e < pw * ph; e += RS_TX * RS_TY) {
    const int py = e / pw, px = e - py * pw;
    const int64_t yc = extend(y00 + py, ny, mode), xd = extend(x00 + px, nx, mode);
    const uint32_t v = (yc < 0 || xd < 0) ? ckey
                                          : (uint32_t)key_of(in, dtype, (t * ny + yc) * nx + xd);
    patch[e] = v;
    acc_or |= v;
  }
  for (int o = 16; o > 0; o >>= 1) acc_or |= __shfl_xor_sync(0xffffffffu, acc_or, o);
  if ((tid & 31) == 0) atomicOr(&s_or, acc_or);
  __syncthreads();
  const int64_t x = (int64_t)blockIdx.x * RS_TX + threadIdx.x;
  const int64_t y = (int64_t)blockIdx.y * RS_TY + threadIdx.y;
  if (x >= nx || y >= ny) return;
  const uint32_t all = s_or;
  int top = 31;
  while (top >= 0 && !((all >> top) & 1u)) --top;
  uint32_t prefix = 0u;
  int r = rank;
  for (int b = top; b >= 0; --b) {
    const uint32_t hi_mask = (b == 31) ? 0u : (~0u << (b + 1));
    int zeros = 0;
    for (int c = 0; c < sy; ++c) {
      const uint32_t* row = patch + (threadIdx.y + c) * pw + threadIdx.x;
      if (NARROW) {
#pragma unroll 4
        for (int d = 0; d < sx; ++d) zeros += row[d] - prefix < (1u << b) ? 1 : 0;
      } else {
        for (int d = 0; d < sx; ++d) {
          const uint32_t v = row[d];
          zeros += ((v & hi_mask) == prefix && !((v >> b) & 1u)) ? 1 : 0;
        }
      }
    }
    if (r >= zeros) {
      r -= zeros;
      prefix |= (1u << b);
    }
  }
  put_apart(ro, (t * ny + y) * nx + x, prefix);
}

__global__ void k_subtract_weighted(const void* img, const void* filt, int64_t count, Subtract sub,
                                    void* out) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < count;
       e += (int64_t)gridDim.x * blockDim.x)
    sub.store_keys(out, e, key_of(img, sub.dtype, e), key_of(filt, sub.dtype, e));
}

// ------------------------------------------------------------------ dispatch
static int key_bytes(int dtype) {
  return dtype == FI_PRE_U8 || dtype == FI_PRE_U16 ? 2 : dtype == FI_PRE_F32 ? 4 : 8;
}

static bool is_extreme(int64_t wsize, int rank) { return rank == 0 || rank == wsize - 1; }

static bool takes_minmax_tile(int dtype, int st, int sy, int sx, int rank) {
  return st == 1 && is_extreme((int64_t)sy * sx, rank) &&
         minmax_tile_bytes(sy, sx, key_bytes(dtype)) <= MM_MAX_SMEM;
}
// k_rank_planes or k_rank_select_tile (both exact).  A thread of the second counts its
// window's values for every bit: 17.5 ns per value and bit, 0.2 ps per pixel, value and bit
// once the chip is full.  A warp of the first takes a 32 x 32 tile in a time that hardly
// depends on the window and not on how many tiles there are while all are resident (16, 12
// or 4 warps an SM by the planes' size): 70 to 390 us for 8 bits, 260 to 1260 for 16, 1440
// to 1900 for 32, less for images than for noise and for large windows.  Which kernel is
// faster near the line depends on the image, which the rule does not see: the values below
// lie between particle images and noise.  Past 16, 8 or 4 tiles an SM the time is taken to
// grow with the tiles; for 16 bits that is before they fill the chip (1216 of 1824 resident
// tiles): at 2048^2, 4096 tiles, particle images take 2.0 times what 1024 tiles take and
// noise 2.9 times, and a line from 1824 on would give 10 to 12 px windows to the planes
// (12 x 12: 1228 against 1695 us, noise 3444 against 2231).
// Median, us, planes and select, particle image / noise:
//   u8  512^2  5 x 5: 160 and 34 / 343 and 33;      30 x 30: 78 and 476 / 160 and 476
//   u16 512^2  5 x 5: 563 and 46 / 1208 and 56;     30 x 30: 344 and 703 / 1029 and 934
//   u16 2048^2 9 x 9: 1355 and 1113 / 3557 and 1458; 30 x 30: 726 and 9212 / 3058 and 12251
//   f32 1024^2 16 x 16: 3483 and 1754 / 3132 and 1753; 30 x 30: 2763 and 6343 / 3013 and 6341
static bool planes_pay(int dtype, int nt, int ny, int nx, int sy, int sx) {
  const int bits = dtype == FI_PRE_U8 ? 8 : dtype == FI_PRE_U16 ? 16 : 32;
  const double tile_us = bits == 8 ? 180.0 : bits == 16 ? 600.0 : 1700.0;
  const double full = (double)num_sms() * 128 / bits;  // 16, 8, 4 tiles an SM
  const double tiles = (double)nt * ((ny + RP_T - 1) / RP_T) * ((nx + RP_T - 1) / RP_T);
  const double counts = (double)sy * sx * bits, pixels = (double)nt * ny * nx;
  const double select_us = counts * (pixels * 2.03e-7 > 0.0175 ? pixels * 2.03e-7 : 0.0175);
  return select_us > tile_us * (tiles > full ? tiles / full : 1.0);
}
static bool takes_time(int dtype, int nt, int st, int sy, int sx) {
  return sy == 1 && sx == 1 && st > 1 &&
         (dtype == FI_PRE_F64 ? time_bytes<uint64_t>(nt, st) : time_bytes<uint32_t>(nt, st)) <=
             TIME_MAX_SMEM;
}

template <typename K>
static int launch_minmax_tile(const void* in, int dtype, int nt, int ny, int nx, int sy, int sx,
                              int mode, uint64_t ckey, int is_max, const RankOut& ro,
                              cudaStream_t s) {
  const size_t smem = minmax_tile_bytes(sy, sx, (int)sizeof(K));
  static SmemLimit limit;
  FI_CUDA_TRY(raise_smem_limit(k_minmax_tile<K>, smem, limit));
  const dim3 grid((unsigned)((nx + MM_TX - 1) / MM_TX), (unsigned)((ny + MM_TY - 1) / MM_TY),
                  (unsigned)nt);
  k_minmax_tile<K><<<grid, MM_NT, smem, s>>>(in, dtype, ny, nx, sy, sx, mode, ckey, is_max, ro);
  return check_launch("fi_rank_filter");
}

template <typename W, int E, bool SPLIT>
static int launch_time_parts(const void* in, int dtype, int nt, int64_t npix, int st, int rank,
                             int mode, uint64_t ckey, int64_t blocks, int span, const RankOut& ro,
                             cudaStream_t s) {
  const size_t smem = time_bytes<W>(nt, st);
  static SmemLimit limit;
  FI_CUDA_TRY(raise_smem_limit(k_time_rank<W, E, SPLIT>, smem, limit));
  const int64_t most = 64 * (int64_t)num_sms();
  const dim3 grid((unsigned)(blocks < most ? blocks : most), (unsigned)((nt + span - 1) / span));
  k_time_rank<W, E, SPLIT><<<grid, TIME_NT, smem, s>>>(in, dtype, nt, npix, st, rank, mode, ckey,
                                                       span, ro);
  return check_launch("fi_rank_filter");
}

template <typename W, int E>
static int launch_time(const void* in, int dtype, int nt, int64_t npix, int st, int rank, int mode,
                       uint64_t ckey, const RankOut& ro, cudaStream_t s) {
  const int V = E == 8 ? 4 : E == 16 ? 2 : 1;
  const int64_t blocks = (npix / V + TIME_NT - 1) / TIME_NT;
  // blocks resident at once, by shared memory (228 KB an SM, 1 KB of it per block) and threads
  const int64_t per_sm = 228 * 1024 / (int64_t)(time_bytes<W>(nt, st) + 1024);
  const int64_t resident = num_sms() * (per_sm < 2048 / TIME_NT ? per_sm : 2048 / TIME_NT);
  const int64_t parts = resident / blocks < nt ? resident / blocks : nt;
  if (parts <= 1)
    return launch_time_parts<W, E, false>(in, dtype, nt, npix, st, rank, mode, ckey, blocks, nt,
                                          ro, s);
  return launch_time_parts<W, E, true>(in, dtype, nt, npix, st, rank, mode, ckey, blocks,
                                       (int)((nt + parts - 1) / parts), ro, s);
}

template <int BITS>
static int launch_planes(const void* in, int dtype, int nt, int ny, int nx, int sy, int sx,
                         int rank, int mode, uint32_t ckey, const RankOut& ro, cudaStream_t s) {
  const size_t smem = RP_WARPS * RpSmem(BITS).bytes;
  static SmemLimit limit;
  FI_CUDA_TRY(raise_smem_limit(k_rank_planes<BITS>, smem, limit));
  const int tx = (nx + RP_T - 1) / RP_T, tiles = tx * ((ny + RP_T - 1) / RP_T);
  const dim3 grid((unsigned)((tiles + RP_WARPS - 1) / RP_WARPS), 1, (unsigned)nt);
  k_rank_planes<BITS><<<grid, 32 * RP_WARPS, smem, s>>>(in, dtype, ny, nx, sy, sx, rank, mode,
                                                        ckey, tx, tiles, ro);
  return check_launch("fi_rank_filter");
}

template <bool NARROW>
static int launch_select(const void* in, int dtype, int nt, int ny, int nx, int sy, int sx,
                         int rank, int mode, uint32_t ckey, const RankOut& ro, size_t smem,
                         cudaStream_t s) {
  static SmemLimit limit;
  FI_CUDA_TRY(raise_smem_limit(k_rank_select_tile<NARROW>, smem, limit));
  const dim3 grid((unsigned)((nx + RS_TX - 1) / RS_TX), (unsigned)((ny + RS_TY - 1) / RS_TY),
                  (unsigned)nt);
  k_rank_select_tile<NARROW><<<grid, dim3(RS_TX, RS_TY), smem, s>>>(in, dtype, ny, nx, sy, sx,
                                                                    rank, mode, ckey, ro);
  return check_launch("fi_rank_filter");
}

static int rank_filter(const void* in, int dtype, int nt, int ny, int nx, int st, int sy, int sx,
                       int rank, int mode, double cval, void* scratch, const RankOut& ro,
                       cudaStream_t s) {
  const int64_t wsize = (int64_t)st * sy * sx;
  FI_REQUIRE(rank >= 0 && rank < wsize, "fi_rank_filter: rank %d not within the window", rank);
  const int64_t count = (int64_t)nt * ny * nx;
  // cval as a key of the image's dtype (scipy casts cval to the input type)
  uint64_t ckey = 0;
  {
    double c = cval;
    switch (dtype) {
      case FI_PRE_U8: ckey = (uint8_t)(int64_t)c; break;
      case FI_PRE_U16: ckey = (uint16_t)(int64_t)c; break;
      case FI_PRE_F32: {
        float f = (float)c;
        uint32_t u;
        memcpy(&u, &f, 4);
        ckey = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        break;
      }
      default: {
        uint64_t u;
        memcpy(&u, &c, 8);
        ckey = (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
      }
    }
  }
  const int g = grid_for(count);
  const int is_max = rank == wsize - 1 && wsize > 1;
  // the frames of a stack are a launch dimension (at most 65535) of the tiled kernels, the
  // tile rows of a frame another
  const bool tiled = nt <= 65535 && ny <= 65535 * RS_TY;
  // minima and maxima whose output overlaps the input: the kernels of one pass would read
  // what other blocks have written; the axis passes write only after all of it is read
  const size_t nbytes = count * element_bytes(dtype);
  const bool in_place = ro.img == nullptr && is_extreme(wsize, rank) &&
                        overlap(in, nbytes, ro.out, nbytes);
  if (!in_place && tiled && takes_minmax_tile(dtype, st, sy, sx, rank)) {
    if (key_bytes(dtype) == 2)
      return launch_minmax_tile<uint16_t>(in, dtype, nt, ny, nx, sy, sx, mode, ckey, is_max, ro, s);
    if (key_bytes(dtype) == 4)
      return launch_minmax_tile<uint32_t>(in, dtype, nt, ny, nx, sy, sx, mode, ckey, is_max, ro, s);
    return launch_minmax_tile<uint64_t>(in, dtype, nt, ny, nx, sy, sx, mode, ckey, is_max, ro, s);
  }
  if (!in_place && takes_time(dtype, nt, st, sy, sx)) {
    const int64_t npix = (int64_t)ny * nx;
    // packed elements: every frame (and output frame) starts on a whole word, the
    // double pairs of the subtraction on 16 bytes
    const bool aligned = (((uintptr_t)in | (uintptr_t)ro.out) & 15) == 0;
    if (dtype == FI_PRE_F64)
      return launch_time<uint64_t, 0>(in, dtype, nt, npix, st, rank, mode, ckey, ro, s);
    if (dtype == FI_PRE_U8 && aligned && npix % 4 == 0)
      return launch_time<uint32_t, 8>(in, dtype, nt, npix, st, rank, mode, ckey, ro, s);
    if (dtype == FI_PRE_U16 && aligned && npix % 2 == 0)
      return launch_time<uint32_t, 16>(in, dtype, nt, npix, st, rank, mode, ckey, ro, s);
    return launch_time<uint32_t, 0>(in, dtype, nt, npix, st, rank, mode, ckey, ro, s);
  }
  if (is_extreme(wsize, rank)) {
    FI_REQUIRE(scratch, "fi_rank_filter: this min/max filter needs scratch[2 * count] (uint64)");
    uint64_t* k0 = static_cast<uint64_t*>(scratch);
    uint64_t* k1 = k0 + count;
    k_minmax_axis<<<g, 256, 0, s>>>(in, 0, nullptr, dtype, nt, ny, nx, 2, sx, mode, ckey, is_max, k0);
    k_minmax_axis<<<g, 256, 0, s>>>(nullptr, 1, k0, dtype, nt, ny, nx, 1, sy, mode, ckey, is_max, k1);
    k_minmax_axis<<<g, 256, 0, s>>>(nullptr, 1, k1, dtype, nt, ny, nx, 0, st, mode, ckey, is_max, k0);
    k_keys_out<<<g, 256, 0, s>>>(k0, count, ro);
    return check_launch("fi_rank_filter", 4);
  }
  if (tiled && st == 1 && dtype != FI_PRE_F64 && sy <= RP_MAX_WINDOW && sx <= RP_MAX_WINDOW &&
      planes_pay(dtype, nt, ny, nx, sy, sx)) {
    if (dtype == FI_PRE_U8)
      return launch_planes<8>(in, dtype, nt, ny, nx, sy, sx, rank, mode, (uint32_t)ckey, ro, s);
    if (dtype == FI_PRE_U16)
      return launch_planes<16>(in, dtype, nt, ny, nx, sy, sx, rank, mode, (uint32_t)ckey, ro, s);
    return launch_planes<32>(in, dtype, nt, ny, nx, sy, sx, rank, mode, (uint32_t)ckey, ro, s);
  }
  const size_t tile_smem = (size_t)(RS_TX + sx - 1) * (RS_TY + sy - 1) * sizeof(uint32_t);
  if (tiled && st == 1 && dtype != FI_PRE_F64 && tile_smem <= RS_MAX_SMEM)
    return sx <= 5 ? launch_select<true>(in, dtype, nt, ny, nx, sy, sx, rank, mode, (uint32_t)ckey,
                                         ro, tile_smem, s)
                   : launch_select<false>(in, dtype, nt, ny, nx, sy, sx, rank, mode,
                                          (uint32_t)ckey, ro, tile_smem, s);
  k_rank_select<<<g, 256, 0, s>>>(in, dtype, nt, ny, nx, st, sy, sx, rank, mode, ckey, ro);
  return check_launch("fi_rank_filter");
}

static int check_rank_args(const void* in, const void* out, int dtype, int nt, int ny, int nx,
                           int st, int sy, int sx, int mode) {
  FI_REQUIRE(in && out, "fi_rank_filter: null pointer");
  FI_REQUIRE(dtype >= FI_PRE_U8 && dtype <= FI_PRE_F64, "fi_rank_filter: bad dtype %d", dtype);
  FI_REQUIRE(mode >= FI_MODE_REFLECT && mode <= FI_MODE_WRAP, "fi_rank_filter: bad mode %d",
             mode);
  FI_REQUIRE(nt >= 1 && ny >= 1 && nx >= 1 && st >= 1 && sy >= 1 && sx >= 1,
             "fi_rank_filter: bad sizes");
  return FI_OK;
}

}  // namespace fi

using namespace fi;

extern "C" int fi_rank_needs_scratch(int dtype, int nt, int ny, int st, int sy, int sx, int rank) {
  const int64_t wsize = (int64_t)st * sy * sx;
  if (!is_extreme(wsize, rank)) return 0;
  const bool tiled = nt <= 65535 && ny <= 65535 * RS_TY;
  return !(tiled && takes_minmax_tile(dtype, st, sy, sx, rank)) && !takes_time(dtype, nt, st, sy, sx);
}

extern "C" int fi_rank_filter(const void* in, void* out, int dtype, int nt, int ny, int nx,
                              int st, int sy, int sx, int rank, int mode, double cval,
                              void* scratch, void* stream) {
  if (check_rank_args(in, out, dtype, nt, ny, nx, st, sy, sx, mode) != FI_OK) return FI_ERR_INVALID;
  const RankOut ro{out, nullptr, dtype, Subtract::make(dtype, 0.0, dtype, 0)};
  return rank_filter(in, dtype, nt, ny, nx, st, sy, sx, rank, mode, cval, scratch, ro,
                     (cudaStream_t)stream);
}

static int check_subtract(const char* who, int dtype, int out_dtype) {
  FI_REQUIRE(out_dtype == FI_PRE_F64 || out_dtype == FI_PRE_F32 ||
                 (out_dtype == dtype && (dtype == FI_PRE_U8 || dtype == FI_PRE_U16)),
             "%s: bad output dtype %d", who, out_dtype);
  return FI_OK;
}

extern "C" int fi_rank_subtract(const void* in, void* out, int dtype, int nt, int ny, int nx,
                                int st, int sy, int sx, int rank, int mode, double cval,
                                double weight, int out_dtype, int clamp, void* scratch,
                                void* stream) {
  if (check_rank_args(in, out, dtype, nt, ny, nx, st, sy, sx, mode) != FI_OK ||
      check_subtract("fi_rank_subtract", dtype, out_dtype) != FI_OK)
    return FI_ERR_INVALID;
  const size_t count = (size_t)nt * ny * nx;
  FI_REQUIRE(!overlap(in, count * element_bytes(dtype), out, count * element_bytes(out_dtype)),
             "fi_rank_subtract: the output overlaps the input");
  const RankOut ro{out, in, dtype, Subtract::make(dtype, weight, out_dtype, clamp)};
  return rank_filter(in, dtype, nt, ny, nx, st, sy, sx, rank, mode, cval, scratch, ro,
                     (cudaStream_t)stream);
}

extern "C" int fi_subtract_weighted(const void* img, const void* filtered, int dtype,
                                    int64_t count, double weight, int out_dtype, int clamp,
                                    void* out, void* stream) {
  FI_REQUIRE(img && filtered && out && count > 0, "fi_subtract_weighted: bad arguments");
  if (check_subtract("fi_subtract_weighted", dtype, out_dtype) != FI_OK) return FI_ERR_INVALID;
  k_subtract_weighted<<<grid_for(count), 256, 0, (cudaStream_t)stream>>>(
      img, filtered, count, Subtract::make(dtype, weight, out_dtype, clamp), out);
  return check_launch("fi_subtract_weighted");
}
