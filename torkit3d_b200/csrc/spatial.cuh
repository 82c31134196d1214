// Spatially ordered copy of a batch of point clouds: the index that the pruned neighbour searches
// walk (spatial.cu: build and up to four nearest neighbours).
//
// The points of a cloud are ordered along a Hilbert curve (16 cells per axis, refined to 256 within
// windows of 256 points) and cut into LEAVES of 32 consecutive points; every leaf has a bounding box,
// and so has every SUPER leaf of 32 leaves.  A leaf is what a warp handles at a time: as queries (one
// lane each, close together in space) and as keys (scanned only when its box can hold a neighbour of
// one of the warp's queries).  Of 512 leaves of a 16384-point cloud a warp has to scan 8 (points on a
// surface) to 14 (in a volume) for nearest neighbours; along a Morton curve it would be 10 to 22.
//
// Exactness.  Neighbour decisions are taken on d = ((dx*dx + dy*dy) + dz*dz) with individually
// rounded operations.  The distance from a point to a box, and from a box to a box, is evaluated
// with the same operations on componentwise differences max(lo - q, q - hi, 0).  Rounding is
// monotonic: for a key r inside the box |fl(r - q)| is at least that difference, and squares and sums
// keep the order, so a box distance is never above the d of any point inside, in float32 as computed,
// without any slack.  A leaf also carries the lowest original index among its points, so a leaf
// whose box is exactly at the current distance is visited only if it can win the tie.
//
// What the index cannot serve is flagged per cloud (SpGrid::irregular): non-finite coordinates
// (their ordering rules belong to the sweeping kernels), and clouds of which more than half sit in
// cells of more than SP_CROWD points (duplicates, or an outlier that stretches the grid), where boxes
// prune little.  The searches skip flagged clouds and the sweeping kernels, launched behind them,
// skip all others.
#pragma once

#include "tk3d_common.cuh"

namespace tk3d {

constexpr int SP_LEAF = 32;
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
  int N, leaves, supers;
  float4 *pts;    // [B][leaves * 32]: two points are two float4, (x0,x1,y0,y1) (z0,z1,i0,i1); i = original index
  float4 *boxes;  // [B][leaves][2]: (lo, lowest original index), (hi, -)
  float4 *sup;    // [B][supers][2]
  int *table;     // [B][SP_CELLS]: first position of every cell
  SpGrid *grid;   // [B]
};

inline size_t sp_align(size_t n) { return (n + 255) / 256 * 256; }

inline size_t sp_cloud_bytes(int64_t B, int64_t N) {
  const int64_t leaves = (N + SP_LEAF - 1) / SP_LEAF, supers = (leaves + 31) / 32;
  return sp_align((size_t)B * leaves * SP_LEAF * 16) + sp_align((size_t)B * leaves * 32) +
         sp_align((size_t)B * supers * 32) + sp_align((size_t)B * SP_CELLS * 4) + sp_align((size_t)B * sizeof(SpGrid));
}

// Lays the arrays of one side out at `at` (256-byte aligned).
inline SpCloud sp_cloud(const float *xyz, int channel_first, int64_t B, int64_t N, char *at) {
  SpCloud c;
  c.xyz = xyz;
  c.l = xyz_layout(channel_first, N);
  c.N = (int)N;
  c.leaves = (int)((N + SP_LEAF - 1) / SP_LEAF);
  c.supers = (c.leaves + 31) / 32;
  c.pts = reinterpret_cast<float4 *>(at);
  at += sp_align((size_t)B * c.leaves * SP_LEAF * 16);
  c.boxes = reinterpret_cast<float4 *>(at);
  at += sp_align((size_t)B * c.leaves * 32);
  c.sup = reinterpret_cast<float4 *>(at);
  at += sp_align((size_t)B * c.supers * 32);
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

// Builds the index of both sides (one launch); `b` may be null.
int sp_build(const SpCloud &a, const SpCloud *b, int64_t B, cudaStream_t st);

// Searches over built indexes; rows of clouds that are irregular on either side are left alone.
int sp_chamfer(const SpCloud &a, const SpCloud &b, int64_t B, float *dist1, int64_t *idx1, float *dist2, int64_t *idx2,
               double *sums, cudaStream_t st);
int sp_knn_small(const SpCloud &q, const SpCloud &k, int64_t B, int K, bool weights, float eps, float *dist,
                 IndexOut index, cudaStream_t st);

// For the sweeping kernels launched behind a search: the grids of the two sides, null for a launch on its own.
struct SpOnly {
  const SpGrid *q, *k;
#ifdef __CUDACC__
  __device__ __forceinline__ bool skip(int64_t b) const { return q && !(q[b].irregular | k[b].irregular); }
  // Nothing to do at all (called by the whole block).
  __device__ __forceinline__ bool idle(int64_t B) const {
    if (!q) return false;
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

// Lower bound of d between any point of box [alo, ahi] and any point of box [blo, bhi].
__device__ __forceinline__ float sp_box_box(const float4 &alo, const float4 &ahi, const float4 &blo,
                                            const float4 &bhi) {
  return sp_sq3(sp_max3(__fsub_rn(alo.x, bhi.x), __fsub_rn(blo.x, ahi.x), 0.f),
                sp_max3(__fsub_rn(alo.y, bhi.y), __fsub_rn(blo.y, ahi.y), 0.f),
                sp_max3(__fsub_rn(alo.z, bhi.z), __fsub_rn(blo.z, ahi.z), 0.f));
}

__device__ __forceinline__ float sp_point_box(float x, float y, float z, const float4 &lo, const float4 &hi) {
  return sp_sq3(sp_max3(__fsub_rn(lo.x, x), __fsub_rn(x, hi.x), 0.f),
                sp_max3(__fsub_rn(lo.y, y), __fsub_rn(y, hi.y), 0.f),
                sp_max3(__fsub_rn(lo.z, z), __fsub_rn(z, hi.z), 0.f));
}

// Two exact squared distances at once: keys (x0,x1) .. against the query (-q, -q).  `one` must be
// 1.0f and unknown to the compiler: fma(a, 1, b) rounds once, like the addition it stands for, and is
// not fused with the product before it.
__device__ __forceinline__ float2 sp_dist2(const float4 &A, const float4 &Bv, float2 nx, float2 ny, float2 nz,
                                           float2 one) {
  const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nx), dy = __fadd2_rn(make_float2(A.z, A.w), ny),
               dz = __fadd2_rn(make_float2(Bv.x, Bv.y), nz);
  return __ffma2_rn(__ffma2_rn(__fmul2_rn(dx, dx), one, __fmul2_rn(dy, dy)), one, __fmul2_rn(dz, dz));
}

// Point `pos` of an ordered cloud (pair layout).
__device__ __forceinline__ float4 sp_point(const float4 *__restrict__ pts, int pos) {
  const float *f = reinterpret_cast<const float *>(pts) + (pos >> 1) * 8 + (pos & 1);
  return make_float4(__ldg(f), __ldg(f + 2), __ldg(f + 4), __ldg(f + 6));
}
#endif

}  // namespace tk3d
