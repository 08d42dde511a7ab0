// Linear interpolation on the Delaunay triangulation of the PIV vectors, with the
// nearest vector outside their convex hull: the griddata path of apply_interp
// (calcul/interpolate/griddata.py:11-27, works/piv/singlepass.py:498-556), which
// upstream runs through scipy (Qhull Delaunay + barycentric interpolation, then a
// k-d tree for the points outside the hull).
//
// The centres are the valid vectors of a pass: each sits at its window-grid node
// (or half a pixel off it, the midpoint of an odd integer shift), so a node map of
// the grid replaces a spatial index.  For a query point q the Delaunay triangle
// containing q is found among the centres of the grid nodes around q: of the
// triangles of those centres that contain q, the Delaunay one minimises the linear
// interpolant of the lifted heights |p - q|^2 at q (the lower convex hull of the
// lifted points); its circumcircle must then hold no other gathered centre and lie
// inside the gathered window (else the window grows).  All predicates are exact
// integer arithmetic on doubled coordinates (PIV positions are half-integers).
// Where four or more centres are cocircular (a regular grid's cells) several
// triangulations are Delaunay; upstream takes Qhull's, here the triangle with the
// smallest vertex indices, and the query is flagged.
#include "fi_common.cuh"

namespace fi {

namespace {

constexpr int GD_RMAX = 8;                        // window half-width in grid steps
                                                  // (then the whole grid)
constexpr int GD_MAXC = 64;                       // nearest centres of the window kept

struct GdArgs {
  const double* cx;
  const double* cy;
  const float* ux;
  const float* uy;
  int nc;
  const int32_t* ixvecs;
  int nx;
  const int32_t* iyvecs;
  int ny;
  const int32_t* nodemap;   // [ny][nx] centre index or -1
  const int2* cxy;          // doubled centre coordinates (exact: half-integers)
  const int2* hull_left;    // left chain of the hull, increasing Y (doubled coords)
  const int2* hull_right;   // right chain
  const int32_t* hull_n;    // [2]: lengths
  const double* px;
  const double* py;
  int npts;
  double* out_x;
  double* out_y;
  int32_t* rx;
  int32_t* ry;
  uint8_t* flags;
  int32_t* status;
};

__device__ __forceinline__ long long orient2(long long ax, long long ay, long long bx,
                                             long long by, long long cx, long long cy) {
  return (bx - ax) * (cy - ay) - (by - ay) * (cx - ax);
}

// largest k with 2 * v[k] <= X2 (-1 if none); v increasing
__device__ __forceinline__ int floor_index(const int32_t* v, int n, long long X2) {
  int lo = 0, hi = n;  // first index with 2 v > X2
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (2LL * v[mid] > X2) hi = mid; else lo = mid + 1;
  }
  return lo - 1;
}

// Position of q against the convex hull (chains of the hull, increasing Y): 1
// strictly outside, 2 on a hull edge (*e0, *e1: the chain vertices around q on it),
// 0 inside.
__device__ int hull_position(const GdArgs& a, long long X, long long Y, int2* e0, int2* e1) {
  const int nl = a.hull_n[0], nr = a.hull_n[1];
  const int2* L = a.hull_left;
  const int2* R = a.hull_right;
  if (nl == 0) return 1;  // no valid centre (*status tells)
  if (Y < L[0].y || Y > L[nl - 1].y) return 1;
  // going up, the inside is to the right of the left chain (o <= 0) and to the left
  // of the right chain (o >= 0)
  int res = 0;
  for (int side = 0; side < 2; ++side) {
    const int2* C = side == 0 ? L : R;
    const int n = side == 0 ? nl : nr;
    if (n == 1) {
      if (side == 0 ? (X < C[0].x) : (X > C[0].x)) return 1;
      continue;
    }
    // the segment arriving at the first vertex with y >= Y (its lower end below Y,
    // or the first segment)
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (C[mid].y >= Y) hi = mid; else lo = mid + 1;
    }
    lo = min(max(lo - 1, 0), n - 2);
    if (C[lo].y == C[lo + 1].y) {  // horizontal (bottom or top) edge at Y
      const int xmin = min(C[lo].x, C[lo + 1].x), xmax = max(C[lo].x, C[lo + 1].x);
      if (side == 0 ? (X < xmin) : (X > xmax)) return 1;
      if (Y == C[lo].y && X >= xmin && X <= xmax) {
        *e0 = C[lo];
        *e1 = C[lo + 1];
        res = 2;
      }
      continue;
    }
    const long long o = orient2(C[lo].x, C[lo].y, C[lo + 1].x, C[lo + 1].y, X, Y);
    if (side == 0 ? (o > 0) : (o < 0)) return 1;
    if (o == 0) {
      *e0 = C[lo];
      *e1 = C[lo + 1];
      res = 2;
    }
  }
  return res;
}

constexpr long long GD_NONE = 0x7fffffffffffffffLL;

// Keys whose integer order is the lexicographic order of (hi, lo), |lo| < 2^30.
__device__ __forceinline__ long long gd_key(int hi, int lo) {
  return ((long long)hi << 32) | (long long)(unsigned)(lo + 0x40000000);
}
__device__ __forceinline__ int gd_key_hi(long long k) { return (int)(k >> 32); }
__device__ __forceinline__ int gd_key_lo(long long k) {
  return (int)(k & 0xffffffffLL) - 0x40000000;
}

__global__ void k_gd_reset(int32_t* nodemap, int nnodes, long long* ext, int next,
                           int32_t* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nnodes) nodemap[i] = -1;
  if (i < next) ext[i] = (i & 1) ? ~GD_NONE : GD_NONE;
  if (i == 0) *status = 0;
}

// Node map, doubled coordinates, and the extremes of each grid row (ext[2 r], the
// smallest (x, y); ext[2 r + 1], the largest) and column (after the rows, (y, x)): four
// 64-bit atomics a centre instead of one thread walking each row in the hull kernel.
__global__ void k_gd_nodemap(const int32_t* sel, const double* cx, const double* cy, int nc,
                             int32_t* nodemap, int2* cxy, long long* ext, int nx, int ny,
                             int32_t* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const int w = sel[i];
  const int nnodes = nx * ny;
  const double X = 2.0 * cx[i], Y = 2.0 * cy[i];
  if (w < 0 || w >= nnodes || X != rint(X) || Y != rint(Y) || fabs(X) > 1e9 || fabs(Y) > 1e9) {
    atomicExch(status, w < 0 || w >= nnodes ? 3 : 1);
    cxy[i] = make_int2(0, 0);
    return;
  }
  const int x = (int)X, y = (int)Y;
  cxy[i] = make_int2(x, y);
  nodemap[w] = i;
  const int row = w / nx, col = w - row * nx;
  const long long kr = gd_key(x, y), kc = gd_key(y, x);
  atomicMin(ext + 2 * row, kr);
  atomicMax(ext + 2 * row + 1, kr);
  atomicMin(ext + 2 * (ny + col), kc);
  atomicMax(ext + 2 * (ny + col) + 1, kc);
}

// Convex hull of the centres.  Every hull vertex is extreme in its grid row or in
// its grid column (a centre with grid neighbours on both sides in both directions is
// inside them: the half-pixel offsets are below half a grid step), so the two chains
// (increasing Y, then X) are built from those extremes, sorted in shared memory
// (bitonic).  One block; a warp a chain: a point that does not turn strictly outwards
// between its two neighbours is no vertex, and a vertex turns outwards between any two
// points, so all such points go at once, and what is left when none goes is the chain
// (a few rounds; one point at a time is a serial chain of ~250 cycles a point).  Bound
// by the latency of the sort's 45 to 78 stages and of the rounds: 9 us for a 53 x 42
// grid and 12 us for 106 x 84 (86 and 191 us with a thread a row and one thread's
// chains).
constexpr int GD_HULL_MAX = 4096;  // row and column extremes (2 (nx + ny))

__global__ void __launch_bounds__(1024) k_gd_hull(int nx, int ny, int m2, int2* left,
                                                  int2* right, int32_t* hull_n) {
  __shared__ long long key[GD_HULL_MAX];
  __shared__ uint16_t chain[2][GD_HULL_MAX];
  const int m = 2 * (nx + ny);
  const int tid = threadIdx.x;
  // the extremes lie where the left chain goes (k_gd_reset, k_gd_nodemap)
  const long long* ext = reinterpret_cast<const long long*>(left);
  for (int t = tid; t < m2; t += blockDim.x) {
    long long k = GD_NONE;
    if (t < m) {
      k = ext[t];
      if (k == ~GD_NONE) k = GD_NONE;  // a row or column without centres
      if (t < 2 * ny && k != GD_NONE) k = gd_key(gd_key_lo(k), gd_key_hi(k));
    }
    key[t] = k;
  }
  __syncthreads();
  // bitonic sort of the keys (Y, then X); m2 / 2 pairs, the pairs of 64 keys always
  // with one warp, so the strides up to 32 need no block barrier
  for (int size = 2; size <= m2; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int j = tid; j < m2 / 2; j += blockDim.x) {
        const int t = ((j & ~(stride - 1)) << 1) | (j & (stride - 1));
        const bool up = (t & size) == 0;
        const long long x = key[t], y = key[t + stride];
        if ((x > y) == up) {
          key[t] = y;
          key[t + stride] = x;
        }
      }
      const int next = stride > 1 ? stride >> 1 : size;
      if (stride > 32 || next > 32) __syncthreads();
      else __syncwarp();
    }
  __syncthreads();
  // going up, the left chain turns clockwise (orient < 0) at each vertex and the
  // right chain counter-clockwise; the lists start as the distinct points
  const int side = tid >> 5, lane = tid & 31;
  if (side < 2) {
    uint16_t* st = chain[side];
    const unsigned below = (1u << lane) - 1;
    int n = 0;
    for (int t0 = 0; t0 < m2; t0 += 32) {
      const long long k = key[t0 + lane];
      const bool keep = k != GD_NONE && (t0 + lane == 0 || k != key[t0 + lane - 1]);
      const unsigned kept = __ballot_sync(0xffffffffu, keep);
      if (keep) st[n + __popc(kept & below)] = (uint16_t)(t0 + lane);
      n += __popc(kept);
    }
    __syncwarp();
    auto vertex = [&](int k) { return make_int2(gd_key_lo(key[k]), gd_key_hi(key[k])); };
    for (int before = n + 1; n < before;) {
      before = n;
      n = 0;
      int last = 0;  // the rank before this 32, which may have been overwritten
      for (int t0 = 0; t0 < before; t0 += 32) {
        const int t = t0 + lane;
        const int rank = t < before ? st[t] : 0;
        const int after = t + 1 < before ? st[t + 1] : 0;
        int prev = __shfl_up_sync(0xffffffffu, rank, 1);
        if (lane == 0) prev = last;
        last = __shfl_sync(0xffffffffu, rank, 31);
        bool keep = t < before;
        if (t > 0 && t + 1 < before) {
          const int2 p0 = vertex(prev), p1 = vertex(rank), p2 = vertex(after);
          const long long o = orient2(p0.x, p0.y, p1.x, p1.y, p2.x, p2.y);
          keep = side == 0 ? o < 0 : o > 0;
        }
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        __syncwarp();  // all lanes have read
        if (keep) st[n + __popc(kept & below)] = (uint16_t)rank;
        n += __popc(kept);
        __syncwarp();
      }
    }
    if (lane == 0) hull_n[side] = n;
  }
  __syncthreads();
  for (int c = 0; c < 2; ++c) {
    const int n = hull_n[c];
    int2* out = c == 0 ? left : right;
    for (int t = tid; t < n; t += blockDim.x) {
      const long long k = key[chain[c][t]];
      out[t] = make_int2(gd_key_lo(k), gd_key_hi(k));
    }
  }
}

struct Cand {
  int dx, dy;   // doubled coordinates relative to q
  int idx;      // centre index (-1: none)
  __device__ __forceinline__ long long d2() const {
    return (long long)dx * dx + (long long)dy * dy;
  }
};

__device__ __forceinline__ Cand make_cand(const GdArgs& a, int i, long long X, long long Y) {
  const int2 p = a.cxy[i];
  return Cand{(int)(p.x - X), (int)(p.y - Y), i};
}

// The predicates below in the integers I that hold them: int where every coordinate is
// below 2^13 (all windows of steps up to 256 px), where differences stay below 2^14,
// areas below 2^29 and the in-circle determinant below 2^60; long long otherwise.
constexpr int GD_SMALL = 1 << 13;

__device__ __forceinline__ bool is_small(const Cand& c) {
  return (unsigned)(c.dx + GD_SMALL) < 2u * GD_SMALL && (unsigned)(c.dy + GD_SMALL) < 2u * GD_SMALL;
}

template <typename I>
__device__ __forceinline__ I area2(const Cand& A, const Cand& B, const Cand& C) {
  return ((I)B.dx - A.dx) * ((I)C.dy - A.dy) - ((I)B.dy - A.dy) * ((I)C.dx - A.dx);
}
template <typename I>
__device__ __forceinline__ I cross(const Cand& A, const Cand& B) {
  return (I)A.dx * B.dy - (I)A.dy * B.dx;
}

// makes (A, B, C) counter-clockwise
template <typename I>
__device__ __forceinline__ void orient_ccw(Cand& A, Cand& B, Cand& C) {
  if (area2<I>(A, B, C) < 0) {
    const Cand t = B;
    B = C;
    C = t;
  }
}

// q (the origin) in the closed triangle: barycentric numerators o (of A, B, C) and
// their sum *D > 0
template <typename I>
__device__ __forceinline__ bool contains_q(const Cand& A, const Cand& B, const Cand& C,
                                           I (&o)[3], I* D) {
  I oa = cross<I>(B, C), ob = cross<I>(C, A), oc = cross<I>(A, B);
  I d = oa + ob + oc;
  if (d < 0) {  // clockwise
    d = -d;
    oa = -oa;
    ob = -ob;
    oc = -oc;
  }
  o[0] = oa;
  o[1] = ob;
  o[2] = oc;
  *D = d;
  return d != 0 && oa >= 0 && ob >= 0 && oc >= 0;
}

// squared distance (doubled units), at most 2^30 - 1: beyond any window of GD_RMAX steps
__device__ __forceinline__ long long capped_d2(const Cand& c) {
  return min(c.d2(), 0x3fffffffLL);
}

// lifted interpolant numerator at q: sum o_i |p_i - q|^2
__device__ __forceinline__ long long lifted(const Cand& A, const Cand& B, const Cand& C,
                                            const int (&o)[3]) {
  return o[0] * capped_d2(A) + o[1] * capped_d2(B) + o[2] * capped_d2(C);
}
__device__ __forceinline__ __int128 lifted(const Cand& A, const Cand& B, const Cand& C,
                                           const long long (&o)[3]) {
  return (__int128)o[0] * capped_d2(A) + (__int128)o[1] * capped_d2(B) +
         (__int128)o[2] * capped_d2(C);
}

// incircle(A, B, C, P) > 0 <=> P strictly inside the circle of (A, B, C)
// (counter-clockwise).  Window coordinates stay below 2^13, so the terms stay below
// 2^58: exact in 64-bit integers.
template <typename I>
__device__ __forceinline__ long long incircle(const Cand& A, const Cand& B, const Cand& C,
                                              const Cand& P) {
  const I adx = (I)A.dx - P.dx, ady = (I)A.dy - P.dy;
  const I bdx = (I)B.dx - P.dx, bdy = (I)B.dy - P.dy;
  const I cdx = (I)C.dx - P.dx, cdy = (I)C.dy - P.dy;
  return (long long)(adx * adx + ady * ady) * (bdx * cdy - cdx * bdy) -
         (long long)(bdx * bdx + bdy * bdy) * (adx * cdy - cdx * ady) +
         (long long)(cdx * cdx + cdy * cdy) * (adx * bdy - bdx * ady);
}

__device__ __forceinline__ void sort3(int (&s)[3]) {
  const int lo = min(s[0], min(s[1], s[2])), hi = max(s[0], max(s[1], s[2]));
  s[1] = s[0] ^ s[1] ^ s[2] ^ lo ^ hi;
  s[0] = lo;
  s[2] = hi;
}

// two triangles weight the centres alike (zero weights for the others)
template <typename I>
__device__ __forceinline__ bool same_weights(const int (&ti)[3], const I (&to)[3], I tD,
                                             const int (&bi)[3], const I (&bo)[3], I bD) {
  bool same = true;
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    I w = 0;
#pragma unroll
    for (int v = 0; v < 3; ++v)
      if (bi[v] == ti[u]) w = bo[v];
    if (sizeof(I) == 4)
      same &= (long long)to[u] * bD == (long long)w * tD;
    else
      same &= (__int128)to[u] * bD == (__int128)w * tD;
  }
#pragma unroll
  for (int v = 0; v < 3; ++v) {  // centres of b that t does not have weigh nothing
    bool shared = false;
#pragma unroll
    for (int u = 0; u < 3; ++u) shared |= ti[u] == bi[v];
    same &= shared || bo[v] == 0;
  }
  return same;
}

// ---- a group of lanes a query ----
constexpr int GD_THREADS = 128;  // a block
constexpr int GD_LANES = 8;      // lanes a query, while its window is small
constexpr int GD_QUICK = 2;      // steps of those windows (then a warp takes the query)
// Up to this many queries an SM a block has four of them, one warp's groups: all blocks are
// resident at once (four an SM, by registers), and each query that is left has a warp of its
// own.  With 16 a block four follow each other on a warp while most SMs are idle: 414
// queries around 5 vectors of a 2 x 23 grid 99 us so, 47 with four (a thread a query: 65),
// 464 of a full 4 x 29 grid 74 and 44; equal where no query is left, and from 2432 on.
constexpr int GD_FEW = 16;

// The groups of a warp go in step: every collective is the warp's (a group's own mask
// would have its groups run one after the other), so what a group decides for itself is
// a predicate, and loops run until the last group is done.
constexpr unsigned GD_ALL = 0xffffffffu;

template <int G>
struct Group {
  int lane;  // in the group
  int base;  // its first lane in the warp
  __device__ __forceinline__ explicit Group(int thread)
      : lane(thread % G), base(thread % 32 - lane) {}
};

// the candidates of a window of grid nodes, row-major: the first (the 16 of a window
// of two steps at least) in registers, dealt to the lanes in turn
template <int G>
struct Window {
  static constexpr int HELD = G < 16 ? 16 / G : 1;
  int c0, r0, w, n;  // first column and row, columns, nodes (0: the group is done)
  int most;          // nodes of the warp's largest window
  Cand held[HELD];
};

template <int G>
__device__ __forceinline__ Cand window_cand(const GdArgs& a, const Window<G>& win, int t, long long X,
                                            long long Y) {
  Cand c{0, 0, -1};
  if (t >= win.n) return c;
  const int r = t / win.w;
  const int i = a.nodemap[(win.r0 + r) * a.nx + win.c0 + (t - r * win.w)];
  if (i >= 0) c = make_cand(a, i, X, Y);
  return c;
}

// calls f(candidate) on the lanes for each node of the window, in their order: f runs on
// all lanes of the warp together (idx -1: no centre)
template <int G, typename F>
__device__ __forceinline__ void for_centres(const GdArgs& a, const Window<G>& win, const Group<G>& g,
                                            long long X, long long Y, F f) {
#pragma unroll
  for (int u = 0; u < Window<G>::HELD; ++u)
    if (u * G < win.most) f(win.held[u]);
  for (int t = Window<G>::HELD * G; t < win.most; t += G) {
    const Cand c = window_cand(a, win, t + g.lane, X, Y);
    f(c);
  }
}

// the group's lanes where p holds, from bit 0
template <int G>
__device__ __forceinline__ unsigned group_ballot(const Group<G>& g, bool p) {
  return (__ballot_sync(GD_ALL, p) >> g.base) & (GD_ALL >> (32 - G));
}

// the smallest key of the group
template <int G>
__device__ __forceinline__ unsigned long long group_min(const Group<G>& g, unsigned long long k) {
#pragma unroll
  for (int d = G / 2; d > 0; d >>= 1) {
    const unsigned long long o = __shfl_xor_sync(GD_ALL, k, d);
    if (o < k) k = o;
  }
  return k;
}

// the entry of the group with the largest v (ties: the smallest i; i < 0: none)
template <int G>
__device__ __forceinline__ void group_best(const Group<G>& g, long long& v, int& i) {
#pragma unroll
  for (int d = G / 2; d > 0; d >>= 1) {
    const long long ov = __shfl_xor_sync(GD_ALL, v, d);
    const int oi = __shfl_xor_sync(GD_ALL, i, d);
    if (oi >= 0 && (i < 0 || ov > v || (ov == v && oi < i))) {
      v = ov;
      i = oi;
    }
  }
}

// a candidate's place among the nearest: d2, then its index (all ones: none, or beyond
// any window of GD_RMAX steps)
constexpr unsigned long long GD_FAR = ~0ULL;
__device__ __forceinline__ unsigned long long near_key(const Cand& c) {
  const long long d2 = c.d2();
  if (c.idx < 0 || d2 > 0x3fffffffLL) return GD_FAR;
  return ((unsigned long long)d2 << 32) | (unsigned)c.idx;
}

// Adds the lanes' candidates to the nearest GD_MAXC, kept in order of their keys: each
// entry's new place is its rank among the old and the new keys.
template <int G>
__device__ __forceinline__ int merge_nearest(const Group<G>& g, unsigned long long* near, int n,
                                             unsigned long long k) {
  if (n == GD_MAXC && k > near[GD_MAXC - 1]) k = GD_FAR;
  const unsigned fresh = group_ballot(g, k != GD_FAR);
  if (!__any_sync(GD_ALL, fresh != 0)) return n;
  constexpr int EACH = GD_MAXC / G;
  unsigned long long old[EACH];
  int at[EACH];
#pragma unroll
  for (int u = 0; u < EACH; ++u) {
    const int p = g.lane + G * u;
    old[u] = p < n ? near[p] : GD_FAR;
    at[u] = p;
  }
  int mine = 0;
#pragma unroll
  for (int l = 0; l < G; ++l) {
    const unsigned long long o = __shfl_sync(GD_ALL, k, g.base + l);
    mine += o < k;
#pragma unroll
    for (int u = 0; u < EACH; ++u) at[u] += o < old[u];
  }
  for (int p = 0; p < n; ++p) mine += near[p] < k;
  __syncwarp();
#pragma unroll
  for (int u = 0; u < EACH; ++u)
    if (old[u] != GD_FAR && at[u] < GD_MAXC) near[at[u]] = old[u];
  if (k != GD_FAR && mine < GD_MAXC) near[mine] = k;
  __syncwarp();
  return min(n + __popc(fresh), GD_MAXC);
}

// Of the triangles of the nearest k centres that contain q, the one with the smallest
// lifted interpolant (ties: the first in the order of their ranks); T its centres,
// unchanged if there is none (or k is 0).  The lanes take the triples in turn.
template <typename I, int G>
__device__ __forceinline__ void nearest_triangle(const GdArgs& a, const Group<G>& g,
                                                 const unsigned long long* near, int k,
                                                 long long X, long long Y, int (&T)[3]) {
  const int total = k * (k - 1) * (k - 2) / 6;
  int ia = 0, ib = 1, ic = 2 + g.lane;
  long long bN = 0, bD = 0;  // bD 0: none (numerators below 2^62: d2 below 2^30)
  int bt = 0x7fffffff, bi[3] = {-1, -1, -1};
  for (int t = g.lane; t < total; t += G, ic += G) {
    while (ic >= k) {  // past the end of this pair's thirds
      const int over = ic - k;
      if (++ib >= k - 1) {
        ++ia;
        ib = ia + 1;
      }
      ic = ib + 1 + over;
    }
    const Cand A = make_cand(a, (int)(unsigned)near[ia], X, Y);
    const Cand B = make_cand(a, (int)(unsigned)near[ib], X, Y);
    const Cand C = make_cand(a, (int)(unsigned)near[ic], X, Y);
    I o[3], D;
    if (!contains_q<I>(A, B, C, o, &D)) continue;
    const long long N = (long long)lifted(A, B, C, o);
    if (bD == 0 || (__int128)N * bD < (__int128)bN * D) {
      bN = N;
      bD = D;
      bt = t;
      bi[0] = A.idx;
      bi[1] = B.idx;
      bi[2] = C.idx;
    }
  }
  __syncwarp();
#pragma unroll
  for (int d = G / 2; d > 0; d >>= 1) {
    const long long oN = __shfl_xor_sync(GD_ALL, bN, d), oD = __shfl_xor_sync(GD_ALL, bD, d);
    const int ot = __shfl_xor_sync(GD_ALL, bt, d);
    const int o0 = __shfl_xor_sync(GD_ALL, bi[0], d), o1 = __shfl_xor_sync(GD_ALL, bi[1], d),
              o2 = __shfl_xor_sync(GD_ALL, bi[2], d);
    const __int128 l = (__int128)oN * bD, r = (__int128)bN * oD;
    if (oD != 0 && (bD == 0 || l < r || (l == r && ot < bt))) {
      bN = oN;
      bD = oD;
      bt = ot;
      bi[0] = o0;
      bi[1] = o1;
      bi[2] = o2;
    }
  }
  if (bD != 0) {
    T[0] = bi[0];
    T[1] = bi[1];
    T[2] = bi[2];
  }
}

// the open box that a window covers, relative to q
struct Covered {
  float xlo, xhi, ylo, yhi;
};

// The triangle of the window's centres at q, for the groups with `run`: T (kept between
// windows) is found among the nearest, improved and certified.  True: the result is the
// weights wo / wD of the centres wi, on all lanes of the group, with *tie; false: the
// window has to grow.
template <typename I, int G>
__device__ __forceinline__ bool window_triangle(const GdArgs& a, const Group<G>& g,
                                                const Window<G>& win, bool run,
                                                long long X, long long Y, const Covered& box,
                                                unsigned long long* near, int (&T)[3],
                                                I (&wo)[3], I* wD, int (&wi)[3], bool* tie) {
  // a triangle of centres containing q: among the nearest k, the one with the
  // smallest lifted interpolant at q (kept from the previous window when found)
  if (__any_sync(GD_ALL, run && T[0] < 0)) {
    const bool search = run && T[0] < 0;
    int n = 0;
    for_centres(a, win, g, X, Y, [&](const Cand& c) {
      n = merge_nearest(g, near, n, search ? near_key(c) : GD_FAR);
    });
    for (int kk = 0; kk < 3; ++kk) {
      int k = min(n, kk == 0 ? 12 : (kk == 1 ? 24 : GD_MAXC));
      if (T[0] >= 0 || !search || (kk > 0 && k <= (kk == 1 ? 12 : 24))) k = 0;
      if (!__any_sync(GD_ALL, k > 0)) break;
      nearest_triangle<I>(a, g, near, k, X, Y, T);
    }
    __syncwarp();
    run = run && T[0] >= 0;
  }
  // Lawson descent: while a centre of the window lies strictly inside the
  // circumcircle of T (its lifted point is below T's plane), replace T by the
  // triangle of that centre and an edge of T that contains q (its plane at q is
  // lower); ends on a triangle whose circumcircle holds no centre of the window.  The
  // last look at the window also tells which centres are on that circle.
  Cand A{0, 0, -1}, B = A, C = A;
  int S[8], ns = 0;
  bool certified = false;
  for (int it = 0; it < 256; ++it) {
    const bool go = run && !certified;
    if (!__any_sync(GD_ALL, go)) break;
    if (go) {
      A = make_cand(a, T[0], X, Y);
      B = make_cand(a, T[1], X, Y);
      C = make_cand(a, T[2], X, Y);
      orient_ccw<I>(A, B, C);
      S[0] = A.idx;
      S[1] = B.idx;
      S[2] = C.idx;
      ns = 3;
    }
    int inside = -1;
    long long best_det = 0;
    for_centres(a, win, g, X, Y, [&](const Cand& P) {
      const bool other =
          go && P.idx >= 0 && P.idx != A.idx && P.idx != B.idx && P.idx != C.idx;
      const long long det = other ? incircle<I>(A, B, C, P) : -1;
      if (det > best_det || (det > 0 && det == best_det && P.idx < inside)) {
        best_det = det;
        inside = P.idx;
      }
      unsigned hits = group_ballot(g, det == 0);
      while (__any_sync(GD_ALL, hits != 0 && ns < 8)) {  // in the order of the nodes
        const int i = __shfl_sync(GD_ALL, P.idx, g.base + (hits ? __ffs(hits) - 1 : 0));
        if (hits != 0 && ns < 8) {
#pragma unroll
          for (int z = 3; z < 8; ++z)
            if (z == ns) S[z] = i;
          ++ns;
          hits &= hits - 1;
        }
      }
    });
    const bool found = group_ballot(g, inside >= 0) != 0;
    certified = certified || (go && !found);
    if (!__any_sync(GD_ALL, found)) break;
    group_best(g, best_det, inside);
    if (found) {
      const Cand P = make_cand(a, inside, X, Y);
      // of the sub-triangles (P, B, C), (A, P, C), (A, B, P) containing q, the one
      // with the smallest lifted interpolant at q (the lower hull of A, B, C, P over q)
      bool any = false;
      __int128 bN = 0;
      I bD = 1;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const Cand U = (e == 0) ? P : A;
        const Cand V = (e == 1) ? P : B;
        const Cand W = (e == 2) ? P : C;
        I o[3], D;
        if (!contains_q<I>(U, V, W, o, &D)) continue;
        const __int128 N = lifted(U, V, W, o);
        if (!any || N * bD < bN * D) {
          any = true;
          bN = N;
          bD = D;
          T[0] = U.idx;
          T[1] = V.idx;
          T[2] = W.idx;
        }
      }
      run = any;  // (none: cannot happen for a triangle containing q)
    }
  }
  run = run && certified;
  // the circumcircle must lie in the covered region (else centres outside the
  // window could be inside it)
  if (run) {
    // circumcentre numerators in exact integers, the test in float with a margin
    // far above its rounding (conservative: a rejected circle only grows the window)
    const long long ax = A.dx, ay = A.dy, bx = B.dx, by = B.dy, cx = C.dx, cy = C.dy;
    const long long dd = 2 * (ax * (by - cy) + bx * (cy - ay) + cx * (ay - by));
    const long long a2 = ax * ax + ay * ay, b2 = bx * bx + by * by, c2 = cx * cx + cy * cy;
    const float ux = (float)(a2 * (by - cy) + b2 * (cy - ay) + c2 * (ay - by)) / (float)dd;
    const float uy = (float)(a2 * (cx - bx) + b2 * (ax - cx) + c2 * (bx - ax)) / (float)dd;
    const float ex = (float)ax - ux, ey = (float)ay - uy;
    const float rad = sqrtf(ex * ex + ey * ey);
    const float mg = 1e-4f * (fabsf(ux) + fabsf(uy) + rad + 1.f);
    run = ux - rad - mg > box.xlo && ux + rad + mg < box.xhi && uy - rad - mg > box.ylo &&
          uy + rad + mg < box.yhi;
  }
  if (!__any_sync(GD_ALL, run)) return false;
  // cocircular centres (on the circumcircle): the triangles of that set containing
  // q are all Delaunay; take the smallest sorted index triple, flag the query when
  // their weights differ
  int ref[3] = {T[0], T[1], T[2]};
  I o0[3] = {0, 0, 0}, D0 = 1;
  sort3(ref);
  if (run)
    contains_q<I>(make_cand(a, ref[0], X, Y), make_cand(a, ref[1], X, Y),
                  make_cand(a, ref[2], X, Y), o0, &D0);
#pragma unroll
  for (int z = 0; z < 3; ++z) {
    wi[z] = ref[z];
    wo[z] = o0[z];
  }
  *wD = D0;
  *tie = false;
  const int nt = run && ns > 3 ? ns : 0;
  if (__any_sync(GD_ALL, nt > 0)) {
    // (indices are below 2^20: at most GD_HULL_MAX / 2 rows and columns together)
    auto order = [](const int (&s)[3]) {
      return ((unsigned long long)s[0] << 40) | ((unsigned long long)s[1] << 20) |
             (unsigned long long)s[2];
    };
    unsigned long long best = nt > 0 ? order(ref) : 0;
    bool differs = false;
    int t = 0;
    for (int u = 0; u < nt; ++u)
      for (int v = u + 1; v < nt; ++v)
        for (int w = v + 1; w < nt; ++w, ++t) {
          if (t % G != g.lane) continue;
          const int ti[3] = {S[u], S[v], S[w]};
          I o[3], D;
          if (!contains_q<I>(make_cand(a, ti[0], X, Y), make_cand(a, ti[1], X, Y),
                             make_cand(a, ti[2], X, Y), o, &D))
            continue;
          if (!same_weights<I>(ti, o, D, ref, o0, D0)) differs = true;
          int st[3] = {ti[0], ti[1], ti[2]};
          sort3(st);
          const unsigned long long k = order(st);
          if (k < best) {
            best = k;
#pragma unroll
            for (int z = 0; z < 3; ++z) {
              wo[z] = o[z];
              wi[z] = ti[z];
            }
            *wD = D;
          }
        }
    __syncwarp();
    *tie = group_ballot(g, differs) != 0;
    // the lanes that hold the smallest hold the same triangle
    const unsigned long long all = group_min(g, best);
    const int from = g.base + __ffs(group_ballot(g, best == all)) - 1;
#pragma unroll
    for (int z = 0; z < 3; ++z) {
      wi[z] = __shfl_sync(GD_ALL, wi[z], from);
      wo[z] = __shfl_sync(GD_ALL, wo[z], from);
    }
    *wD = __shfl_sync(GD_ALL, *wD, from);
  }
  return run;
}

// the same in 64-bit integers (wider grids, and the whole grid)
__device__ __noinline__ bool wide_triangle(const GdArgs& a, const Group<32>& g,
                                           const Window<32>& win, long long X, long long Y,
                                           const Covered& box, unsigned long long* near,
                                           int (&T)[3], long long (&wo)[3], long long* wD,
                                           int (&wi)[3], bool* tie) {
  return window_triangle<long long>(a, g, win, true, X, Y, box, near, T, wo, wD, wi, tie);
}

struct Query {
  int q, r;  // index; steps of the next window (1 .. GD_RMAX, then the whole grid)
  int T[3];  // a triangle (centre indices) containing q (-1: none yet)
};

// Takes the groups' queries (q < 0: none) on, up to windows of `stop` steps.  True: the
// query is done; false: it goes on from qs (a wider window, or 64-bit integers, which
// the warp has).  The groups of a warp start at the same window.
template <int G>
__device__ __forceinline__ bool take_query(const GdArgs& a, const Group<G>& g, Query& qs, int stop,
                                           unsigned long long* near) {
  const int q = qs.q;
  bool run = q >= 0, done = !run;
  long long X = 0, Y = 0;
  int hpos = 0, i0 = 0, j0 = 0;
  int2 e0 = make_int2(0, 0), e1 = make_int2(0, 0);
  if (run) {
    const double qx2 = 2.0 * a.px[q], qy2 = 2.0 * a.py[q];
    if (qx2 != rint(qx2) || qy2 != rint(qy2) || fabs(qx2) > 1e9 || fabs(qy2) > 1e9) {
      if (g.lane == 0) atomicExch(a.status, 1);  // off the half-integer lattice
      run = false;
      done = true;
    } else {
      X = (long long)qx2;
      Y = (long long)qy2;
      hpos = hull_position(a, X, Y, &e0, &e1);
      i0 = floor_index(a.ixvecs, a.nx, X);
      j0 = floor_index(a.iyvecs, a.ny, Y);
    }
  }
  __syncwarp();
  const bool outside = hpos == 1;
  uint8_t flag = 0;
  // sum of weight * value over nw centres, in their order: the first lane takes x, the
  // second y (doubles are slow: no lane takes both)
  auto store = [&](const int (&i)[3], const double (&w)[3], int nw) {
    if (g.lane >= 2) return;
    const float* u = g.lane == 0 ? a.ux : a.uy;
    double v;
    if (nw == 1) {
      v = (double)u[i[0]];
    } else if (nw == 2) {
      v = w[0] * (double)u[i[0]] + w[1] * (double)u[i[1]];
    } else {
      v = 0.0;
#pragma unroll
      for (int z = 0; z < 3; ++z) v += w[z] * (double)u[i[z]];
    }
    (g.lane == 0 ? a.out_x : a.out_y)[q] = v;
    int32_t* r = g.lane == 0 ? a.rx : a.ry;
    if (r) r[q] = (int32_t)rint(v);
    if (g.lane == 0 && a.flags) a.flags[q] = flag;
  };
  int wi[3] = {0, 0, 0};
  double w[3] = {1.0, 0.0, 0.0};
  for (int r = qs.r; r <= stop && __any_sync(GD_ALL, run); ++r) {
    if (run) qs.r = r;
    // nodes of columns [i0 - r + 1, i0 + r] and rows [j0 - r + 1, j0 + r]; past
    // GD_RMAX steps (a large region without vectors) the whole grid
    const bool all = r > GD_RMAX;
    const int c0 = all ? 0 : max(i0 - r + 1, 0), c1 = all ? a.nx - 1 : min(i0 + r, a.nx - 1);
    const int r0 = all ? 0 : max(j0 - r + 1, 0), r1 = all ? a.ny - 1 : min(j0 + r, a.ny - 1);
    Window<G> win;
    win.c0 = c0;
    win.r0 = r0;
    win.w = max(c1 - c0 + 1, 0);
    win.n = run ? win.w * max(r1 - r0 + 1, 0) : 0;
    win.most = G == 32 ? win.n : __reduce_max_sync(GD_ALL, win.n);
#pragma unroll
    for (int u = 0; u < Window<G>::HELD; ++u)
      win.held[u] = window_cand(a, win, g.lane + G * u, X, Y);
    // the nearest centre (ties: smallest index) and whether others are as near
    unsigned long long nearest = GD_FAR;
    bool tied = false, big = false;
    for_centres(a, win, g, X, Y, [&](const Cand& c) {
      big |= !is_small(c);
      const unsigned long long k = near_key(c);
      if (k == GD_FAR) return;
      if ((k >> 32) <= (nearest >> 32)) tied = (k >> 32) == (nearest >> 32);
      if (k < nearest) nearest = k;
    });
    __syncwarp();
    {
      const unsigned long long best = group_min(g, nearest);
      const bool as_near = (nearest >> 32) == (best >> 32);
      const unsigned holders = group_ballot(g, as_near);
      const unsigned ties = group_ballot(g, as_near && tied);
      tied = __popc(holders) > 1 || ties != 0;
      big = group_ballot(g, big) != 0;
      nearest = best;
    }
    // exclusive bounds of the region the window covers: a centre of column c has
    // 2 ixvecs[c] <= X2 <= 2 ixvecs[c] + 1
    const bool bxlo = !all && i0 - r >= 0, bxhi = !all && i0 + r + 1 < a.nx;
    const bool bylo = !all && j0 - r >= 0, byhi = !all && j0 + r + 1 < a.ny;
    constexpr long long OPEN = 1LL << 60;
    const long long xlo = bxlo ? 2LL * a.ixvecs[i0 - r] + 1 - X : -OPEN;
    const long long xhi = bxhi ? 2LL * a.ixvecs[i0 + r + 1] - X : OPEN;
    const long long ylo = bylo ? 2LL * a.iyvecs[j0 - r] + 1 - Y : -OPEN;
    const long long yhi = byhi ? 2LL * a.iyvecs[j0 + r + 1] - Y : OPEN;
    bool at_one = false;  // the nearest centre's value
    if (run && nearest != GD_FAR) {
      if (outside) {
        // nearest centre (ties: smallest index), certified when the nearest distance
        // is below the distance to the uncovered region
        const double d = sqrt((double)(int)(nearest >> 32));
        const double margin = (double)min(min(-xlo, xhi), min(-ylo, yhi));
        at_one = d < margin * (1.0 - 1e-12);
        if (at_one && tied) flag |= 2;
      } else {
        // q on a centre: its value (the weights of every triangle at that vertex)
        at_one = (nearest >> 32) == 0;
      }
    }
    if (at_one) {
      wi[0] = (int)(unsigned)nearest;
      store(wi, w, 1);
      run = false;
      done = true;
    }
    if (__any_sync(GD_ALL, run && hpos == 2)) {
      // q on a hull edge: the Delaunay edge containing q joins the nearest centres on
      // that line on either side (the chain vertices e0, e1 unless collinear centres
      // lie between); certified when both lie in the covered region
      const bool edge = run && hpos == 2;
      const long long ux_ = e1.x - e0.x, uy_ = e1.y - e0.y;
      // positions along the line, relative to q (scaled by |e1 - e0|^2)
      const long long t_e0 = (e0.x - X) * ux_ + (e0.y - Y) * uy_;  // < 0
      const long long t_e1 = (e1.x - X) * ux_ + (e1.y - Y) * uy_;  // > 0
      long long v_lo = 0, v_hi = 0;  // largest t below 0, largest -t above 0
      int i_lo = -1, i_hi = -1;
      for_centres(a, win, g, X, Y, [&](const Cand& c) {
        if (!edge || c.idx < 0) return;
        const long long px_ = c.dx, py_ = c.dy;  // relative to q
        if ((px_ + X - e0.x) * uy_ - (py_ + Y - e0.y) * ux_ != 0) return;  // off the line
        const long long t = px_ * ux_ + py_ * uy_;
        if (t < 0 && t >= t_e0) {
          if (i_lo < 0 || t > v_lo || (t == v_lo && c.idx < i_lo)) {
            v_lo = t;
            i_lo = c.idx;
          }
        } else if (t > 0 && t <= t_e1) {
          if (i_hi < 0 || -t > v_hi || (-t == v_hi && c.idx < i_hi)) {
            v_hi = -t;
            i_hi = c.idx;
          }
        }
      });
      __syncwarp();
      group_best(g, v_lo, i_lo);
      group_best(g, v_hi, i_hi);
      auto covered = [&](int i) {
        const Cand c = make_cand(a, i, X, Y);
        return c.dx > xlo && c.dx < xhi && c.dy > ylo && c.dy < yhi;
      };
      if (edge && i_lo >= 0 && i_hi >= 0 && covered(i_lo) && covered(i_hi)) {
        w[1] = (double)(-v_lo) / (double)(-v_hi - v_lo);  // weight of the high end
        w[0] = 1.0 - w[1];
        wi[0] = i_lo;
        wi[1] = i_hi;
        store(wi, w, 2);
        run = false;
        done = true;
      }
    }
    if (G < 32 && run && big) run = false;  // left to the warp
    const bool inner = run && hpos == 0;
    if (!__any_sync(GD_ALL, inner)) continue;
    Covered box;
    box.xlo = bxlo ? (float)xlo : -INFINITY;
    box.xhi = bxhi ? (float)xhi : INFINITY;
    box.ylo = bylo ? (float)ylo : -INFINITY;
    box.yhi = byhi ? (float)yhi : INFINITY;
    double wo, D;  // this lane's weight
    bool tie, found;
    if (G == 32 && big) {
      if constexpr (G == 32) {
        long long o[3], d;
        found = wide_triangle(a, g, win, X, Y, box, near, qs.T, o, &d, wi, &tie);
        wo = (double)(g.lane == 0 ? o[0] : g.lane == 1 ? o[1] : o[2]);
        D = (double)d;
      }
    } else {
      int o[3], d;
      found = window_triangle<int>(a, g, win, inner, X, Y, box, near, qs.T, o, &d, wi, &tie);
      wo = (double)(g.lane == 0 ? o[0] : g.lane == 1 ? o[1] : o[2]);
      D = (double)d;
    }
    if (!__any_sync(GD_ALL, found)) continue;
    // each lane divides one weight (a quotient is ~10 instructions in doubles)
    const double mine = found ? wo / D : 0.0;
#pragma unroll
    for (int z = 0; z < 3; ++z) w[z] = __shfl_sync(GD_ALL, mine, g.base + z);
    if (found) {
      if (tie) flag |= 1;
      store(wi, w, 3);
      run = false;
      done = true;
    }
  }
  if (run) qs.r = stop + 1;
  return done;
}

// Bound by the dependent instructions of a query's exact predicates at 16 warps an SM
// (registers; issue 22 and 39 % of the slots for 8 900 and 36 000 queries) and, at the
// borders and around holes, by the few queries whose window grows (up to C(64, 3) triples
// each).
// Eight lanes take a query: they share the nodes of a window (each loaded once, in
// registers up to two steps) and the triples, and every decision is the group's.  The
// block's queries that need more than GD_QUICK steps are then taken by whole warps (the
// border and the holes: C(24, 3) triples on eight lanes set the block's time).
// Measured, whole call: 79 x 63 grid with 10 % holes, 20 193 queries: 3.1 ms with a
// thread a query, 0.51 ms with eight lanes throughout, 0.30 ms with a warp throughout,
// 0.22 ms as here; the same grid with 2 % holes 260, 79, 193 and 81 us; 255 x 255 with
// 3 % holes, 261 121 queries: 27, 7.8, 2.9 and 2.4 ms.
__global__ void __launch_bounds__(GD_THREADS) k_gd_interp(GdArgs a, int per_block) {
  __shared__ unsigned long long s_near[GD_THREADS / GD_LANES][GD_MAXC];
  __shared__ Query s_left[GD_THREADS / GD_LANES];
  __shared__ int s_nleft;
  if (threadIdx.x == 0) s_nleft = 0;
  __syncthreads();
  const int slot = threadIdx.x / GD_LANES;
  const int q = blockIdx.x * per_block + slot;
  if (slot < per_block) {  // whole warps
    const Group<GD_LANES> g(threadIdx.x);
    Query qs{q < a.npts ? q : -1, 1, {-1, -1, -1}};
    if (!take_query(a, g, qs, GD_QUICK, s_near[slot]) && g.lane == 0)
      s_left[atomicAdd(&s_nleft, 1)] = qs;
  }
  __syncthreads();
  const Group<32> g(threadIdx.x);
  const int warp = threadIdx.x / 32;
  for (int k = warp; k < s_nleft; k += GD_THREADS / 32) {
    Query qs = s_left[k];
    __syncwarp();
    if (take_query(a, g, qs, GD_RMAX + 1, s_near[warp]) || g.lane != 0) continue;
    atomicExch(a.status, 2);  // no certified triangle (cannot happen with the whole grid)
    a.out_x[qs.q] = a.out_y[qs.q] = NAN;
    if (a.rx) a.rx[qs.q] = 0;
    if (a.ry) a.ry[qs.q] = 0;
  }
}

}  // namespace

}  // namespace fi

using namespace fi;

extern "C" int fi_griddata(const double* cx, const double* cy, const float* ux, const float* uy,
                           const int32_t* selection, int num_centers, const int32_t* ixvecs,
                           int nx, const int32_t* iyvecs, int ny, const double* px,
                           const double* py, int npts, int32_t* scratch, double* out_x,
                           double* out_y, int32_t* rx, int32_t* ry, uint8_t* flags,
                           int32_t* status, void* stream) {
  FI_REQUIRE(cx && cy && ux && uy && selection && ixvecs && iyvecs && px && py && scratch &&
                 out_x && out_y && status,
             "fi_griddata: null pointer");
  FI_REQUIRE(num_centers > 0 && nx > 0 && ny > 0 && npts > 0, "fi_griddata: bad sizes");
  FI_REQUIRE(((uintptr_t)scratch & 7) == 0, "fi_griddata: scratch must be 8-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const int nnodes = nx * ny;
  FI_REQUIRE(2 * (nx + ny) <= GD_HULL_MAX, "fi_griddata: window grid of %d x %d too large",
             nx, ny);
  FI_REQUIRE(num_centers <= nnodes, "fi_griddata: more centres than grid nodes");
  int32_t* nodemap = scratch;
  int2* cxy = reinterpret_cast<int2*>(scratch + ((nnodes + 1) & ~1));
  int2* left = cxy + nnodes;
  int2* right = left + 2 * (nx + ny);
  int32_t* hull_n = reinterpret_cast<int32_t*>(right + 2 * (nx + ny));
  long long* ext = reinterpret_cast<long long*>(left);  // 2 (nx + ny), until the hull
  GdArgs a{cx, cy, ux, uy, num_centers, ixvecs, nx, iyvecs, ny, nodemap, cxy, left, right,
           hull_n, px, py, npts, out_x, out_y, rx, ry, flags, status};
  const int next = 2 * (nx + ny);
  const int nreset = max(nnodes, next);
  k_gd_reset<<<(nreset + 255) / 256, 256, 0, s>>>(nodemap, nnodes, ext, next, status);
  k_gd_nodemap<<<(num_centers + 255) / 256, 256, 0, s>>>(selection, cx, cy, num_centers,
                                                         nodemap, cxy, ext, nx, ny, status);
  int m2 = 64;
  while (m2 < next) m2 <<= 1;
  k_gd_hull<<<1, min(1024, max(64, m2 / 2)), 0, s>>>(nx, ny, m2, left, right, hull_n);
  const int per_block = npts <= GD_FEW * num_sms() ? 32 / GD_LANES : GD_THREADS / GD_LANES;
  k_gd_interp<<<(npts + per_block - 1) / per_block, GD_THREADS, 0, s>>>(a, per_block);
  return check_launch("fi_griddata", 4);
}

extern "C" int64_t fi_griddata_scratch_ints(int nx, int ny) {
  return (int64_t)((nx * ny + 1) & ~1) + 2LL * nx * ny + 8LL * (nx + ny) + 2;
}
