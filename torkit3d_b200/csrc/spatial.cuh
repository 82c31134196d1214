// Spatially ordered copy of a batch of point clouds: the index that the pruned neighbour searches
// walk (spatial.cu: build and up to four nearest neighbours, spatial_knn.cu: up to 64,
// spatial_ball.cu: ball query).
//
// The points of a cloud are ordered along a Hilbert curve: by one of 4096 cells (16 per axis), and
// within WINDOWS of 256 points by one of 256 cells per axis.  Eight consecutive points form a LEAF, a
// window is 32 leaves; leaves and windows have bounding boxes.  A warp takes 32 consecutive points as
// queries (one lane each, close together in space), finds the windows and leaves whose boxes can hold
// a neighbour of one of its queries, and scans those.
//
// Why eight: all lanes of a warp read the same key, and a 16-byte load hands 512 bytes to the lanes
// whatever it reads, four cycles of the SM's L1; that, not arithmetic, bounds a scan.  Two clouds of
// 16384 points, one neighbour, keys scanned per warp (counted on the CPU): leaves of 32 / 16 / 8 points
// 433 / 272 / 156 in a volume, 262 / 177 / 112 on a surface, 573 / 369 / 236 in blobs.  Along a Morton
// curve it would be about 1.6 times as many.
//
// Exactness.  Neighbour decisions are taken on d = ((dx*dx + dy*dy) + dz*dz) with individually
// rounded operations.  The distance from a point to a box, and from a box to a box, is evaluated
// with the same operations on componentwise differences max(lo - q, q - hi, 0).  Rounding is
// monotonic: for a key r inside the box |fl(r - q)| is at least that difference, and squares and sums
// keep the order, so a box distance is never above the d of any point inside, in float32 as computed,
// without any slack.  A leaf also carries the lowest original index among its points, so a leaf
// whose box is exactly at the current distance is visited only if it can win the tie.
//
// What the index cannot serve is flagged per cloud (SpGrid::irregular): non-finite coordinates (their ordering
// rules belong to the sweeping kernels), and clouds of which more than half sit in cells of more than SP_CROWD
// points (duplicates, or an outlier that stretches the grid), where boxes prune little.  A sample finds more of
// them out before anything is sorted (spatial.cu): a grid too coarse for the cloud, pairs of clouds so placed
// that most leaves are within reach of every query, balls too dense.  The searches skip flagged clouds, and the
// sweeping kernels, launched behind them, skip all others (a ball query sweeps where it is).
#pragma once

#include "tk3d_common.cuh"

namespace tk3d {

constexpr int SP_GROUP = 32;    // queries of a warp
constexpr int SP_LEAF = 8;
constexpr int SP_WINDOW = 256;  // 32 leaves
constexpr int SP_CELLS = 4096;  // 16 per axis
constexpr int SP_CROWD = 4096;
constexpr int64_t SP_MAX_POINTS = 1 << 20;

struct SpGrid {
  float lox, loy, loz, inv;  // fine cell (256 per axis) = clamp((x - lo) * inv)
  int irregular;
  int pad[3];
};

// One side of a search: B clouds of N points and the arrays built from them.
struct SpCloud {
  const float *xyz;
  XyzLayout l;
  int N, groups, windows;
  float *pts;     // [B][windows * 32][4][8]: x, y, z and original index of a leaf's points; padding is NaN
  float4 *boxes;  // [B][windows * 32][2]: (lo x, y, z, hi x), (hi y, hi z, lowest original index, -)
  float4 *wbox;   // [B][windows][2]
  int *table;     // [B][SP_CELLS]: first position of every cell
  SpGrid *grid;   // [B]
};

inline size_t sp_align(size_t n) { return (n + 255) / 256 * 256; }

inline size_t sp_cloud_bytes(int64_t B, int64_t N) {
  const int64_t windows = (N + SP_WINDOW - 1) / SP_WINDOW;
  return sp_align((size_t)B * windows * SP_WINDOW * 16) + sp_align((size_t)B * windows * 32 * 32) +
         sp_align((size_t)B * windows * 32) + sp_align((size_t)B * SP_CELLS * 4) + sp_align((size_t)B * sizeof(SpGrid));
}

// Lays the arrays of one side out at `at` (256-byte aligned).
inline SpCloud sp_cloud(const float *xyz, int channel_first, int64_t B, int64_t N, char *at) {
  SpCloud c;
  c.xyz = xyz;
  c.l = xyz_layout(channel_first, N);
  c.N = (int)N;
  c.groups = (int)((N + SP_GROUP - 1) / SP_GROUP);
  c.windows = (int)((N + SP_WINDOW - 1) / SP_WINDOW);
  c.pts = reinterpret_cast<float *>(at);
  at += sp_align((size_t)B * c.windows * SP_WINDOW * 16);
  c.boxes = reinterpret_cast<float4 *>(at);
  at += sp_align((size_t)B * c.windows * 32 * 32);
  c.wbox = reinterpret_cast<float4 *>(at);
  at += sp_align((size_t)B * c.windows * 32);
  c.table = reinterpret_cast<int *>(at);
  at += sp_align((size_t)B * SP_CELLS * 4);
  c.grid = reinterpret_cast<SpGrid *>(at);
  return c;
}

// Shapes that the index takes.
inline bool sp_supported(int64_t B, int64_t N1, int64_t N2) {
  return B > 0 && N1 >= 1 && N1 <= SP_MAX_POINTS && N2 >= 512 && N2 <= SP_MAX_POINTS;
}

// The index is built for as many clouds at a time as fit into about 512 MB.
inline int64_t sp_batch(int64_t B, int64_t N1, int64_t N2) {
  const int64_t fit = (int64_t)((512u << 20) / (sp_cloud_bytes(1, N1) + sp_cloud_bytes(1, N2)));
  return fit < 1 ? 1 : (fit < B ? fit : B);
}
inline size_t sp_search_bytes(int64_t B, int64_t N1, int64_t N2) {
  const int64_t n = sp_batch(B, N1, N2);
  return sp_cloud_bytes(n, N1) + sp_cloud_bytes(n, N2) + 256;
}
inline char *sp_align_ptr(void *p) {
  return reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) + 255) & ~(uintptr_t)255);
}

// What the index is built for: a search of a's points in b, `both`: and the other way round.  Pairs of clouds that the
// order would not serve are flagged irregular (spatial.cu):
struct SpUse {
  bool both;
  bool prunes;    // where nothing would be pruned
  bool resolves;  // where the grid is too coarse
  int row;        // of a ball query: its row length and squared radius; where balls are dense
  float r2;
};

// Builds the index of both sides (two launches); `b` may be null: both sides are a.  SP_DECLINED where the device
// refuses the cluster launch (a partition without room for it): nothing was built, the caller sweeps.
constexpr int SP_DECLINED = -1;
int sp_build(const SpCloud &a, const SpCloud *b, int64_t B, const SpUse &use, cudaStream_t st);

// Searches over built indexes; rows of clouds that are irregular on either side are left alone.
int sp_chamfer(const SpCloud &a, const SpCloud &b, int64_t B, float *dist1, int64_t *idx1, float *dist2, int64_t *idx2,
               double *sums, cudaStream_t st);
int sp_knn_small(const SpCloud &q, const SpCloud &k, int64_t B, int K, bool weights, float eps, float *dist,
                 IndexOut index, cudaStream_t st);
int sp_knn_select(const SpCloud &q, const SpCloud &k, int64_t B, int K, float *dist, IndexOut index, cudaStream_t st);
int sp_ball_query(const float *query, const float *key, int64_t B, int64_t N1, int64_t N2, int channel_first, float r2,
                  int k, void *index, int index32, void *scratch, cudaStream_t st);
constexpr int64_t SP_SELECT_POINTS = 1 << 19;  // keys at most: leaf numbers are kept in 16 bits

// What a sweeping kernel is to do: all pairs of clouds, or (launched behind a search) those that the search left, by
// the grids of the two sides.  A type of its own for all pairs: a null pointer to test cost the sweeps 1 to 12 %.
struct SpAll {
#ifdef __CUDACC__
  __device__ __forceinline__ bool skip(int64_t) const { return false; }
  __device__ __forceinline__ bool idle(int64_t) const { return false; }
#endif
};
struct SpOnly {
  const SpGrid *q, *k;
#ifdef __CUDACC__
  __device__ __forceinline__ bool skip(int64_t b) const { return !(q[b].irregular | k[b].irregular); }
  // Nothing to do at all (called by the whole block).
  __device__ __forceinline__ bool idle(int64_t B) const {
    int any = 0;
    for (int64_t b = threadIdx.x; b < B; b += blockDim.x) any |= q[b].irregular | k[b].irregular;
    return !__syncthreads_or(any);
  }
#endif
};

#ifdef __CUDACC__
// Position along a Hilbert curve with BITS bits per axis (J. Skilling, "Programming the Hilbert
// curve", 2004: undo the reflections and axis swaps from the top bit down, then decode the Gray code).
// The leading bits depend on the leading bits of the coordinates alone.
template <int BITS>
__device__ __forceinline__ unsigned sp_hilbert(unsigned x, unsigned y, unsigned z) {
#pragma unroll
  for (int s = BITS - 1; s > 0; --s) {
    const unsigned P = (1u << s) - 1;
    x ^= (0u - ((x >> s) & 1u)) & P;
    const unsigned my = 0u - ((y >> s) & 1u), ty = (x ^ y) & P & ~my;
    x ^= (my & P) | ty;
    y ^= ty;
    const unsigned mz = 0u - ((z >> s) & 1u), tz = (x ^ z) & P & ~mz;
    x ^= (mz & P) | tz;
    z ^= tz;
  }
  y ^= x;
  z ^= y;
  unsigned t = z >> 1;  // t: parity of the bits of z above each bit
  t ^= t >> 1;
  t ^= t >> 2;
  t ^= t >> 4;
  x ^= t, y ^= t, z ^= t;
  unsigned code = 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    unsigned v = c == 0 ? x : c == 1 ? y : z;
    v = (v | (v << 8)) & 0x00F00F;
    v = (v | (v << 4)) & 0x0C30C3;
    v = (v | (v << 2)) & 0x249249;
    code |= v << (2 - c);
  }
  return code;
}

__device__ __forceinline__ unsigned sp_axis(float x, float lo, float inv) {
  return (unsigned)fminf(fmaxf((x - lo) * inv, 0.f), 255.f);  // a NaN product (0 * inf) counts as 0
}
// Cell of the position table.
__device__ __forceinline__ unsigned sp_cell(float x, float y, float z, const SpGrid &g) {
  return sp_hilbert<4>(sp_axis(x, g.lox, g.inv) >> 4, sp_axis(y, g.loy, g.inv) >> 4, sp_axis(z, g.loz, g.inv) >> 4);
}
__device__ __forceinline__ unsigned sp_fine(float x, float y, float z, const SpGrid &g) {
  return sp_hilbert<8>(sp_axis(x, g.lox, g.inv), sp_axis(y, g.loy, g.inv), sp_axis(z, g.loz, g.inv));
}

__device__ __forceinline__ float sp_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float sp_min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float sp_warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float sp_warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float sp_inf() { return __int_as_float(0x7f800000); }
__device__ __forceinline__ float sp_nan() { return __int_as_float(0x7fc00000); }

__device__ __forceinline__ float sp_sq3(float dx, float dy, float dz) {
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

struct SpBox {
  float lx, ly, lz, hx, hy, hz;
};
__device__ __forceinline__ SpBox sp_box(const float4 *__restrict__ at) {
  const float4 a = __ldg(at);
  const float2 c = __ldg(reinterpret_cast<const float2 *>(at + 1));
  return {a.x, a.y, a.z, a.w, c.x, c.y};
}

// Lower bound of d between any point of one box and any point of another.
__device__ __forceinline__ float sp_box_box(const SpBox &a, const SpBox &c) {
  return sp_sq3(sp_max3(__fsub_rn(a.lx, c.hx), __fsub_rn(c.lx, a.hx), 0.f),
                sp_max3(__fsub_rn(a.ly, c.hy), __fsub_rn(c.ly, a.hy), 0.f),
                sp_max3(__fsub_rn(a.lz, c.hz), __fsub_rn(c.lz, a.hz), 0.f));
}
__device__ __forceinline__ float sp_point_box(float x, float y, float z, const SpBox &c) {
  return sp_sq3(sp_max3(__fsub_rn(c.lx, x), __fsub_rn(x, c.hx), 0.f), sp_max3(__fsub_rn(c.ly, y), __fsub_rn(y, c.hy), 0.f),
                sp_max3(__fsub_rn(c.lz, z), __fsub_rn(z, c.hz), 0.f));
}

// Exact squared distances of a leaf's eight keys, two at a time, from the query (-q, -q).  `one` must
// be 1.0f and unknown to the compiler: fma(a, 1, b) rounds once, like the addition it stands for, and
// is not fused with the product before it.  Padding keys give NaN.
__device__ __forceinline__ void sp_leaf_dist(const float *__restrict__ leaf, float2 nx, float2 ny, float2 nz, float2 one,
                                             float2 (&d)[4]) {
  const float4 *v = reinterpret_cast<const float4 *>(leaf);
  float4 c[6];
#pragma unroll
  for (int u = 0; u < 6; ++u) c[u] = __ldg(v + u);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float4 X = c[u >> 1], Y = c[2 + (u >> 1)], Z = c[4 + (u >> 1)];
    const float2 dx = __fadd2_rn((u & 1) ? make_float2(X.z, X.w) : make_float2(X.x, X.y), nx);
    const float2 dy = __fadd2_rn((u & 1) ? make_float2(Y.z, Y.w) : make_float2(Y.x, Y.y), ny);
    const float2 dz = __fadd2_rn((u & 1) ? make_float2(Z.z, Z.w) : make_float2(Z.x, Z.y), nz);
    d[u] = __ffma2_rn(__ffma2_rn(__fmul2_rn(dx, dx), one, __fmul2_rn(dy, dy)), one, __fmul2_rn(dz, dz));
  }
}
__device__ __forceinline__ void sp_leaf_index(const float *__restrict__ leaf, int (&i)[8]) {
  const int4 a = __ldg(reinterpret_cast<const int4 *>(leaf) + 6), c = __ldg(reinterpret_cast<const int4 *>(leaf) + 7);
  i[0] = a.x, i[1] = a.y, i[2] = a.z, i[3] = a.w, i[4] = c.x, i[5] = c.y, i[6] = c.z, i[7] = c.w;
}
__device__ __forceinline__ float sp_min8(const float2 (&d)[4]) {
  float m = sp_min3(d[0].x, d[0].y, d[1].x);
  m = sp_min3(m, d[1].y, d[2].x);
  m = sp_min3(m, d[2].y, d[3].x);
  return fminf(m, d[3].y);
}

// Positions and leaves of an ordered cloud of `windows` windows; the range-checked build counts those outside.
#ifdef TK3D_BOUNDS
__device__ __forceinline__ int sp_checked(int i, int n) { return (int)tk3d_checked(i, n); }
#else
__device__ __forceinline__ int sp_checked(int i, int) { return i; }
#endif
__device__ __forceinline__ const float *sp_leaf(const float *__restrict__ pts, int leaf, int windows) {
  return pts + sp_checked(leaf, windows * 32) * 32;
}

// Point `pos` of an ordered cloud: coordinates and original index.
__device__ __forceinline__ float4 sp_point(const float *__restrict__ pts, int pos, int windows) {
  pos = sp_checked(pos, windows * SP_WINDOW);
  const float *f = pts + (int64_t)(pos >> 3) * 32 + (pos & 7);
  return make_float4(__ldg(f), __ldg(f + 8), __ldg(f + 16), __ldg(f + 24));
}
#endif

}  // namespace tk3d
