// Spatially ordered clouds (see spatial.cuh): the build, and the nearest-neighbour search over it.
#include <cooperative_groups.h>

#include "spatial.cuh"

namespace cg = cooperative_groups;

namespace tk3d {

namespace {

// ---------------------------------------------------------------------------------------------
// Build: one thread-block cluster of CL blocks per cloud.  A counting sort by coarse cell: every block
// counts its slice of the points into a histogram in its own shared memory; the exclusive prefix over
// (cell, block) is formed across the cluster through distributed shared memory, each block for its
// share of the cells; then every block writes its points to their places.  The order inside a cell is
// whatever the atomics give.  Then every warp takes windows of 256 consecutive points, sorts them by
// their fine position along the curve (a bitonic network on registers) and forms the leaf boxes.
// Searches decide by original index, so no result depends on the order.
constexpr int SB_THREADS = 512;
constexpr int SB_WARPS = SB_THREADS / 32;
constexpr int SB_WINDOW = 256;

struct SpPair {
  SpCloud c[2];
};

template <int CL>
__global__ void __launch_bounds__(SB_THREADS)
spatial_build_kernel(const __grid_constant__ SpPair pair, int B) {
  constexpr int SHARE = SP_CELLS / CL;      // cells of one block
  constexpr int MINE = SHARE / SB_THREADS;  // cells of one thread
  static_assert(MINE >= 1 && MINE * CL * SB_THREADS == SP_CELLS, "whole cells per thread");
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CL > 1 ? (int)cluster.block_rank() : 0;
  const int id = blockIdx.x / CL;
  const SpCloud &c = pair.c[id >= B];
  const int64_t b = id >= B ? id - B : id;
  const int N = c.N;
  __shared__ __align__(16) int hist[SP_CELLS];
  __shared__ float red[SB_WARPS][8];
  __shared__ float part[8];  // this block's (lo, hi, non-finite)
  __shared__ int warp_total[SB_WARPS];
  __shared__ int block_total, crowd;
  auto sync = [&]() {
    if constexpr (CL > 1) cluster.sync();
    else __syncthreads();
  };
  auto remote = [&](auto *p, int o) {
    if constexpr (CL > 1) return cluster.map_shared_rank(p, o);
    else return p;
  };
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float *xyz = c.xyz + b * 3 * (int64_t)N;
  float4 *pts = c.pts + b * (int64_t)c.leaves * SP_LEAF;
  const int NL = (N + CL - 1) / CL;
  const int beg = min(N, rank * NL), end = min(N, beg + NL);

#pragma unroll
  for (int e = 0; e < SP_CELLS / SB_THREADS; ++e) hist[tid + e * SB_THREADS] = 0;
  if (tid == 0) crowd = 0;
  float v[7] = {sp_inf(), sp_inf(), sp_inf(), -sp_inf(), -sp_inf(), -sp_inf(), 0.f};
#pragma unroll 4
  for (int j = beg + tid; j < end; j += SB_THREADS) {
    float x, y, z;
    load_xyz(xyz, j, c.l, x, y, z);
    v[0] = fminf(v[0], x), v[1] = fminf(v[1], y), v[2] = fminf(v[2], z);
    v[3] = fmaxf(v[3], x), v[4] = fmaxf(v[4], y), v[5] = fmaxf(v[5], z);
    if (!(fabsf(x) < sp_inf() && fabsf(y) < sp_inf() && fabsf(z) < sp_inf())) v[6] = 1.f;
  }
#pragma unroll
  for (int i = 0; i < 7; ++i) v[i] = i < 3 ? sp_warp_min(v[i]) : sp_warp_max(v[i]);
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < 7; ++i) red[warp][i] = v[i];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < 7; ++i) {
      const float w = red[lane & (SB_WARPS - 1)][i];
      const float r = i < 3 ? sp_warp_min(w) : sp_warp_max(w);
      if (lane == 0) part[i] = r;
    }
  }
  sync();
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    float r = part[i];
#pragma unroll
    for (int o = 0; o < CL; ++o) {
      const float w = *remote(&part[i], o);
      r = i < 3 ? fminf(r, w) : fmaxf(r, w);
    }
    v[i] = r;
  }
  SpGrid g;
  g.lox = v[0], g.loy = v[1], g.loz = v[2];
  const float ext = fmaxf(fmaxf(v[3] - v[0], v[4] - v[1]), v[5] - v[2]);
  g.inv = (ext > 0.f && ext < sp_inf()) ? 256.f / ext : 0.f;
  g.irregular = v[6] != 0.f;

#pragma unroll 4
  for (int j = beg + tid; j < end; j += SB_THREADS) {
    float x, y, z;
    load_xyz(xyz, j, c.l, x, y, z);
    atomicAdd(&hist[sp_cell(x, y, z, g)], 1);
  }
  sync();

  // exclusive prefix over (cell, block): this thread's cells are c0 .. c0 + MINE - 1
  const int c0 = rank * SHARE + tid * MINE;
  int n[CL][MINE], sum = 0;
#pragma unroll
  for (int o = 0; o < CL; ++o)
#pragma unroll
    for (int i = 0; i < MINE; ++i) n[o][i] = remote(hist, o)[c0 + i];
#pragma unroll
  for (int i = 0; i < MINE; ++i) {
    int t = 0;
#pragma unroll
    for (int o = 0; o < CL; ++o) t += n[o][i];
    if (t > SP_CROWD) atomicAdd(remote(&crowd, 0), t);
    sum += t;
  }
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int p = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += p;
  }
  if (lane == 31) warp_total[warp] = inc;
  __syncthreads();
  int at = inc - sum;
#pragma unroll
  for (int w = 0; w < SB_WARPS; ++w) at += w < warp ? warp_total[w] : 0;
  if (CL > 1) {
    if (tid == SB_THREADS - 1) block_total = at + sum;
    sync();
    for (int o = 0; o < rank; ++o) at += *remote(&block_total, o);
  }
#pragma unroll
  for (int i = 0; i < MINE; ++i) {
    c.table[b * SP_CELLS + c0 + i] = at;
#pragma unroll
    for (int o = 0; o < CL; ++o) {
      remote(hist, o)[c0 + i] = at;
      at += n[o][i];
    }
  }
  sync();

#pragma unroll 4
  for (int j = beg + tid; j < end; j += SB_THREADS) {
    float x, y, z;
    load_xyz(xyz, j, c.l, x, y, z);
    const int to = atomicAdd(&hist[sp_cell(x, y, z, g)], 1);
    pts[to] = make_float4(x, y, z, __int_as_float(j));
  }
  if (rank == 0) {
    // padding of the last leaf: NaN distances are never below or at a bound
    for (int j = N + tid; j < c.leaves * SP_LEAF; j += SB_THREADS)
      pts[j] = make_float4(sp_nan(), sp_nan(), sp_nan(), __int_as_float(0x7fffffff));
    if (tid == 0) {
      if (2 * (int64_t)crowd > N) g.irregular = 1;
      g.pad[0] = g.pad[1] = g.pad[2] = 0;
      c.grid[b] = g;
    }
  }
  sync();

  // windows: element e = 32 r + lane of a window is register r
  float4 *boxes = c.boxes + b * (int64_t)c.leaves * 2;
  const int windows = (c.leaves + 7) / 8;
  for (int w = rank * SB_WARPS + warp; w < windows; w += CL * SB_WARPS) {
    float4 *p = pts + (int64_t)w * SB_WINDOW;
    const int live = min(8, c.leaves - 8 * w);  // leaves of this window
    unsigned key[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const unsigned e = 32 * r + lane;
      key[r] = 0xffffff00u | e;  // padding sorts last
      if (r < live) {
        const float4 q = __ldcg(p + e);
        if (__float_as_int(q.w) != 0x7fffffff) key[r] = (sp_fine(q.x, q.y, q.z, g) << 8) | e;
      }
    }
#pragma unroll
    for (int k = 2; k <= SB_WINDOW; k <<= 1) {
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        if (j >= 32) {
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const int o = r ^ (j >> 5);
            if (o > r) {
              const bool up = ((32 * r) & k) == 0;
              const unsigned lo = min(key[r], key[o]), hi = max(key[r], key[o]);
              key[r] = up ? lo : hi;
              key[o] = up ? hi : lo;
            }
          }
        } else {
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const unsigned other = __shfl_xor_sync(0xffffffffu, key[r], j);
            const bool up = ((32 * r + lane) & k) == 0, low = (lane & j) == 0;
            key[r] = up == low ? min(key[r], other) : max(key[r], other);
          }
        }
      }
    }
    float4 q[8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < live) q[r] = __ldcg(p + (key[r] & 255u));
    __syncwarp();  // every point is in registers before its place is written
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < live) {
        const int leaf = 8 * w + r;
        const float4 lo = make_float4(sp_warp_min(q[r].x), sp_warp_min(q[r].y), sp_warp_min(q[r].z),
                                      __int_as_float(__reduce_min_sync(0xffffffffu, __float_as_int(q[r].w))));
        const float4 hi = make_float4(sp_warp_max(q[r].x), sp_warp_max(q[r].y), sp_warp_max(q[r].z), 0.f);
        if (lane == 0) {
          boxes[2 * leaf] = lo;
          boxes[2 * leaf + 1] = hi;
        }
        // pair p becomes (x0,x1,y0,y1) (z0,z1,i0,i1): lane l writes float4 number l
        const int o = lane & 1;
        const float s0 = o ? q[r].x : q[r].z, s1 = o ? q[r].y : q[r].w;  // what the pair's other lane stores
        const float t0 = __shfl_xor_sync(0xffffffffu, s0, 1), t1 = __shfl_xor_sync(0xffffffffu, s1, 1);
        p[32 * r + lane] = o ? make_float4(t0, q[r].z, t1, q[r].w) : make_float4(q[r].x, t0, q[r].y, t1);
      }
    }
  }
  sync();
  for (int s = rank * SB_WARPS + warp; s < c.supers; s += CL * SB_WARPS) {
    const int leaf = s * 32 + lane;
    float4 lo = make_float4(sp_inf(), sp_inf(), sp_inf(), __int_as_float(0x7fffffff));
    float4 hi = make_float4(-sp_inf(), -sp_inf(), -sp_inf(), 0.f);
    if (leaf < c.leaves) {
      lo = __ldcg(boxes + 2 * leaf);
      hi = __ldcg(boxes + 2 * leaf + 1);
    }
    lo = make_float4(sp_warp_min(lo.x), sp_warp_min(lo.y), sp_warp_min(lo.z),
                     __int_as_float(__reduce_min_sync(0xffffffffu, __float_as_int(lo.w))));
    hi = make_float4(sp_warp_max(hi.x), sp_warp_max(hi.y), sp_warp_max(hi.z), 0.f);
    if (lane == 0) {
      c.sup[(b * c.supers + s) * 2] = lo;
      c.sup[(b * c.supers + s) * 2 + 1] = hi;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// K <= 4 nearest keys of every query: one warp per query leaf, lane = query.
//   1. SEEDS keys around the position of the query's cell in the key cloud bound its K-th distance.
//   2. The warp scans the leaf it is closest to, then walks super leaves and leaves whose boxes come
//      within the largest bound of its 32 queries; a leaf is scanned when at least one lane's own
//      bound reaches its box.
//   3. A scan evaluates exact distances two keys at a time (every lane reads the same 32 bytes) and
//      branches once per eight keys.
// The list starts as K entries (bound, INT_MAX): the K keys behind the bound all order before or at
// it, so they fill the list whatever order the leaves come in, and (distance, index) decides as in a
// sweep in index order.  For the chamfer distance it starts as (+inf, -1) instead: there a distance of
// +inf is no neighbour.
template <int K>
struct SpList {
  float d[K];
  int i[K];
  __device__ __forceinline__ void offer(float dn, int in) {
    if (dn < d[K - 1] || (dn == d[K - 1] && in < i[K - 1])) {
      d[K - 1] = dn;
      i[K - 1] = in;
#pragma unroll
      for (int c = K - 1; c > 0; --c) {
        if (d[c] < d[c - 1] || (d[c] == d[c - 1] && i[c] < i[c - 1])) {
          const float td = d[c];
          d[c] = d[c - 1];
          d[c - 1] = td;
          const int ti = i[c];
          i[c] = i[c - 1];
          i[c - 1] = ti;
        }
      }
    }
  }
};

constexpr int SN_THREADS = 128;
constexpr int SN_WARPS = SN_THREADS / 32;

template <int K>
__device__ __forceinline__ void sp_scan(const float4 *__restrict__ leaf, float2 nx, float2 ny, float2 nz, float2 one,
                                        SpList<K> &list) {
  float4 A[8];  // four key pairs, loaded one step ahead
#pragma unroll
  for (int u = 0; u < 8; ++u) A[u] = __ldg(leaf + u);
#pragma unroll
  for (int p = 0; p < SP_LEAF; p += 8) {
    float2 d[4], id[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      d[u] = sp_dist2(A[2 * u], A[2 * u + 1], nx, ny, nz, one);
      id[u] = make_float2(A[2 * u + 1].z, A[2 * u + 1].w);
    }
    if (p + 8 < SP_LEAF) {
#pragma unroll
      for (int u = 0; u < 8; ++u) A[u] = __ldg(leaf + p + 8 + u);
    }
    float m = sp_min3(d[0].x, d[0].y, d[1].x);
    m = sp_min3(m, d[1].y, d[2].x);
    m = sp_min3(m, d[2].y, d[3].x);
    m = fminf(m, d[3].y);
    if (m <= list.d[K - 1]) {
      if constexpr (K == 1) {  // only the smallest of the eight can enter: its lowest index
        int i = 0x7fffffff;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          i = min(i, d[u].x == m ? __float_as_int(id[u].x) : 0x7fffffff);
          i = min(i, d[u].y == m ? __float_as_int(id[u].y) : 0x7fffffff);
        }
        list.offer(m, i);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (d[u].x <= list.d[K - 1]) list.offer(d[u].x, __float_as_int(id[u].x));
          if (d[u].y <= list.d[K - 1]) list.offer(d[u].y, __float_as_int(id[u].y));
        }
      }
    }
  }
}

enum { SN_CHAMFER = 0, SN_KNN = 1, SN_WEIGHTS = 2 };

// The two directions of a launch: side s searches the other side's keys for its own points.
struct SpSearch {
  SpCloud c[2];
  float *dist[2];
  IndexOut index[2];
  int64_t tasks[2];  // query leaves of all clouds
  int64_t blocks0;   // blocks of direction 0
};

template <int K, int MODE>
__global__ void __launch_bounds__(SN_THREADS)
spatial_nn_kernel(const __grid_constant__ SpSearch job, double *__restrict__ sums, float eps, float one_) {
  constexpr int SEEDS = 8;
  static_assert(K <= SEEDS / 2, "the seeds bound the K-th distance");
  __shared__ double ssum[SN_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rev = blockIdx.x >= job.blocks0;
  const SpCloud &qc = job.c[rev], &kc = job.c[1 - rev];
  const int64_t task = (blockIdx.x - (rev ? job.blocks0 : 0)) * SN_WARPS + warp;
  double total = 0.0;
  if (task < job.tasks[rev]) {
    const int64_t b = task / qc.leaves;
    const int ql = (int)(task - b * qc.leaves);
    const SpGrid g = kc.grid[b];
    if (!(g.irregular | qc.grid[b].irregular)) {
      const float4 q = sp_point(qc.pts + b * (int64_t)qc.leaves * SP_LEAF, ql * SP_LEAF + lane);
      const float4 *qbox = qc.boxes + (b * qc.leaves + ql) * 2;
      const float4 qlo = __ldg(qbox), qhi = __ldg(qbox + 1);
      const bool valid = ql * SP_LEAF + lane < qc.N;
      const float2 one = make_float2(one_, one_);
      const float2 nx = make_float2(-q.x, -q.x), ny = make_float2(-q.y, -q.y), nz = make_float2(-q.z, -q.z);
      const float4 *kpts = kc.pts + b * (int64_t)kc.leaves * SP_LEAF;
      const float4 *kbox = kc.boxes + b * (int64_t)kc.leaves * 2;
      const float4 *ksup = kc.sup + b * (int64_t)kc.supers * 2;

      // 1. seeds
      const int *tab = kc.table + b * SP_CELLS;
      const int e = sp_cell(q.x, q.y, q.z, g);
      const int p0 = __ldg(tab + e), p1 = e + 1 < SP_CELLS ? __ldg(tab + e + 1) : kc.N;
      const int seed = min(max(((p0 + p1) >> 1) - SEEDS / 2, 0), kc.N - SEEDS - 1) & ~1;
      SpList<K> list;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        list.d[c] = sp_inf();
        list.i[c] = MODE == SN_CHAMFER ? -1 : 0x7fffffff;
      }
#pragma unroll
      for (int u = 0; u < SEEDS / 2; ++u) {
        const float4 A = __ldg(kpts + seed + 2 * u), Bv = __ldg(kpts + seed + 2 * u + 1);
        const float2 d = sp_dist2(A, Bv, nx, ny, nz, one);
        list.offer(d.x, __float_as_int(Bv.z));
        list.offer(d.y, __float_as_int(Bv.w));
      }
      if constexpr (K > 1) {
        // the seeds come again with their leaves: keep their bound only
        const float bound = list.d[K - 1];
#pragma unroll
        for (int c = 0; c < K; ++c) {
          list.d[c] = bound;
          list.i[c] = 0x7fffffff;
        }
      }
      if (!valid) list.d[K - 1] = -1.f;  // never reached by a distance

      // 2. the closest leaf, then the rest
      const int home = __shfl_sync(0xffffffffu, seed + SEEDS / 2, min(16, qc.N - ql * SP_LEAF - 1)) >> 5;
      sp_scan<K>(kpts + (int64_t)home * SP_LEAF, nx, ny, nz, one, list);
      float gb = sp_warp_max(list.d[K - 1]);
      const int chunks = (kc.supers + 31) >> 5;
      int ch = home >> 10;
      for (int cc = 0; cc < chunks; ++cc) {
        const int s = ch * 32 + lane;
        bool hit = false;
        if (s < kc.supers) hit = sp_box_box(qlo, qhi, __ldg(ksup + 2 * s), __ldg(ksup + 2 * s + 1)) <= gb;
        unsigned smask = __ballot_sync(0xffffffffu, hit);
        unsigned first = cc == 0 ? smask & (1u << ((home >> 5) & 31)) : 0u;
        while (smask) {
          const int sl = __ffs(first ? first : smask) - 1;
          first = 0u;
          smask &= ~(1u << sl);
          const int l0 = (ch * 32 + sl) * 32;
          hit = false;
          if (l0 + lane < kc.leaves && l0 + lane != home)
            hit = sp_box_box(qlo, qhi, __ldg(kbox + 2 * (l0 + lane)), __ldg(kbox + 2 * (l0 + lane) + 1)) <= gb;
          unsigned lmask = __ballot_sync(0xffffffffu, hit);
          while (lmask) {
            const int l = l0 + __ffs(lmask) - 1;
            lmask &= lmask - 1;
            const float4 lo = __ldg(kbox + 2 * l), hi = __ldg(kbox + 2 * l + 1);
            const float bd = sp_point_box(q.x, q.y, q.z, lo, hi);
            const bool need =
                bd < list.d[K - 1] || (bd == list.d[K - 1] && __float_as_int(lo.w) < list.i[K - 1]);
            if (__any_sync(0xffffffffu, need)) sp_scan<K>(kpts + (int64_t)l * SP_LEAF, nx, ny, nz, one, list);
          }
          gb = sp_warp_max(list.d[K - 1]);
        }
        ch = ch + 1 < chunks ? ch + 1 : 0;
      }

      // 3. results go to the query's own row
      if (valid) {
        const int64_t row = (b * qc.N + __float_as_int(q.w)) * K;
        float *out = job.dist[rev] + row;
        const IndexOut &io = job.index[rev];
        float w[K];
#pragma unroll
        for (int c = 0; c < K; ++c) w[c] = list.d[c];
        if constexpr (MODE == SN_WEIGHTS) {
          float sum = 0.f;
#pragma unroll
          for (int c = 0; c < K; ++c) {
            w[c] = __fdiv_rn(1.0f, fmaxf(w[c], eps));
            sum = c == 0 ? w[c] : __fadd_rn(sum, w[c]);
          }
#pragma unroll
          for (int c = 0; c < K; ++c) w[c] = __fdiv_rn(w[c], sum);
        }
#pragma unroll
        for (int c = 0; c < K; ++c) {
          out[c] = w[c];
          io.put(row + c, list.i[c]);
        }
        total = (double)list.d[0];
      }
    }
  }
  if (MODE == SN_CHAMFER && sums != nullptr) {
    total = warp_sum(total);
    if (lane == 0) ssum[warp] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
#pragma unroll
      for (int w = 0; w < SN_WARPS; ++w) t += ssum[w];
      atomicAdd(sums + rev, t);
    }
  }
}

}  // namespace

int sp_build(const SpCloud &a, const SpCloud *b, int64_t B, cudaStream_t st) {
  const int64_t clouds = b ? 2 * B : B;
  const int big = b && b->N > a.N ? b->N : a.N;
  // Blocks per cloud: as many as the SMs hold at once (two each), at least 512 points per block.
  int CL = 1;
  while (CL < 8 && clouds * CL <= sm_count() && big >= CL * 2 * SB_THREADS) CL *= 2;
  SpPair pair;
  pair.c[0] = a;
  pair.c[1] = b ? *b : a;
  const void *kern = CL == 8   ? (const void *)spatial_build_kernel<8>
                     : CL == 4 ? (const void *)spatial_build_kernel<4>
                     : CL == 2 ? (const void *)spatial_build_kernel<2>
                               : (const void *)spatial_build_kernel<1>;
  int B_ = (int)B;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clouds * CL));
  cfg.blockDim = dim3(SB_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *args[] = {&pair, &B_};
  TK3D_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
  return check_launch("spatial_build_kernel");
}

int sp_chamfer(const SpCloud &a, const SpCloud &b, int64_t B, float *dist1, int64_t *idx1, float *dist2, int64_t *idx2,
               double *sums, cudaStream_t st) {
  SpSearch job;
  job.c[0] = a, job.c[1] = b;
  job.dist[0] = dist1, job.dist[1] = dist2;
  job.index[0] = index_out(idx1, 0, B * a.N), job.index[1] = index_out(idx2, 0, B * b.N);
  job.tasks[0] = B * a.leaves, job.tasks[1] = B * b.leaves;
  job.blocks0 = (job.tasks[0] + SN_WARPS - 1) / SN_WARPS;
  const int64_t blocks = job.blocks0 + (job.tasks[1] + SN_WARPS - 1) / SN_WARPS;
  spatial_nn_kernel<1, SN_CHAMFER><<<(unsigned)blocks, SN_THREADS, 0, st>>>(job, sums, 0.f, 1.0f);
  return check_launch("spatial_nn_kernel");
}

int sp_knn_small(const SpCloud &q, const SpCloud &k, int64_t B, int K, bool weights, float eps, float *dist,
                 IndexOut index, cudaStream_t st) {
  SpSearch job;
  job.c[0] = q, job.c[1] = k;
  job.dist[0] = job.dist[1] = dist;
  job.index[0] = job.index[1] = index;
  job.tasks[0] = B * q.leaves, job.tasks[1] = 0;
  job.blocks0 = (job.tasks[0] + SN_WARPS - 1) / SN_WARPS;
  const unsigned grid = (unsigned)job.blocks0;
#define SN_LAUNCH(KK, MODE) spatial_nn_kernel<KK, MODE><<<grid, SN_THREADS, 0, st>>>(job, nullptr, eps, 1.0f)
  if (weights) SN_LAUNCH(3, SN_WEIGHTS);
  else if (K == 1) SN_LAUNCH(1, SN_KNN);
  else if (K == 2) SN_LAUNCH(2, SN_KNN);
  else if (K == 3) SN_LAUNCH(3, SN_KNN);
  else SN_LAUNCH(4, SN_KNN);
#undef SN_LAUNCH
  return check_launch("spatial_nn_kernel");
}

}  // namespace tk3d

TK3D_BOUNDS_TU(spatial)
