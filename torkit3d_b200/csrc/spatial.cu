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
// whatever the atomics give.  A second launch then sorts every window of 256 points by fine cell (a warp
// each, a bitonic network on registers) and forms the boxes.  Searches decide by original index, so no
// result depends on the order.
constexpr int SB_THREADS = 512;
constexpr int SB_WARPS = SB_THREADS / 32;

struct SpPair {
  SpCloud c[2];
};

// Inputs that the order would not serve are found out from a sample before anything is sorted, and flagged as
// irregular.
//
// Dense balls (16 queries and 512 keys).  Where balls hold more than about twice the wanted hits, sweeping the keys
// in index order stops early and ordering them is wasted.  32 x 1024 queries of 8192 keys, k = 32, 20 / 100 /
// 1000 hits, us: sweep 137, 95, 29; ordered 72, 171, 145.
//
// Nothing to prune.  Where most sampled keys are no farther from a query than its nearest sampled key and the
// spacing of the sample together, most leaves come within reach of every group of queries: a cloud that has
// collapsed, or lies in the middle of the other one.  The share of such keys was at most 0.1 for volumes, surfaces,
// blobs, lattices and clouds away from one another, and 0.9 and more for a cloud of radius 0.01 in the middle
// of a sphere (sweep / ordered, us: chamfer 32 x 4096^2 208 / 384, 2 x 8192^2 102 / 309, k = 3 16 x 4096^2
// 133 / 246, k = 16 168 / 342, k = 32 340 / 450, k = 64 709 / 700: flagged above a half, up to 32 neighbours).
// The look costs 2 to 3 us; a flagged pair pays 10 to 20 us over its sweep.
//
// A grid too coarse.  Where a fine cell around a point holds a good part of the cloud, the windows cannot be sorted:
// an outlier that squeezes all other points into a few cells, heavy tails.  Share of the cloud in such a cell and
// sweep / ordered, us, chamfer 32 x 4096^2: a sphere with an outlier at 10 radii 0.0001, 229 / 83; at 100 radii
// 0.012, 229 / 255; at 1000 all of it, 229 / 616; points on a line 0.004, 245 / 93: flagged above 1 / PK_COARSE.
// More than four neighbours are found twice to ten times as fast in order even then (16 x 4096^2, k = 16, 1000
// radii: 1950 / 460), because the sweep's lists overflow.
constexpr int PK_SAMPLE = 8;  // queries, and keys whose surroundings are looked at
constexpr int PK_KEYS = 128;  // keys they are held against
constexpr int PK_COARSE = 32;
static_assert(PK_KEYS == 128 && SB_WARPS == 16, "two directions, four slices of the keys, two halves of the queries");

// Sampled key i of N: one of each PK_KEYS-th of the cloud, at varying places (a cloud that repeats itself must not
// give the same points over and over).
__device__ __forceinline__ int64_t pk_key(int i, int N) {
  return ((int64_t)(i * PK_KEYS + ((i * 73) & (PK_KEYS - 1))) * N) / (PK_KEYS * PK_KEYS);
}

template <int CL>
__global__ void __launch_bounds__(SB_THREADS, 2)
spatial_sort_kernel(const __grid_constant__ SpPair pair, int B, SpUse use) {
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
  __shared__ int block_total, crowd, close;
  __shared__ __align__(16) float least[2][2][PK_SAMPLE / CL][PK_KEYS / 32];
  __shared__ int near[2];  // sampled keys that would come within reach
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
  float4 *pts = reinterpret_cast<float4 *>(c.pts) + b * (int64_t)c.windows * SP_WINDOW;
  const int NL = (N + CL - 1) / CL;
  const int beg = min(N, rank * NL), end = min(N, beg + NL);

  if (use.row > 0) {
    const SpCloud &qc = pair.c[0], &kc = pair.c[1];
    float kx, ky, kz;
    load_xyz(kc.xyz + b * 3 * (int64_t)kc.N, (int64_t)tid * kc.N / SB_THREADS, kc.l, kx, ky, kz);
    int hits = 0;
#pragma unroll 4
    for (int i = 0; i < 16; ++i) {
      float x, y, z;
      load_xyz(qc.xyz + b * 3 * (int64_t)qc.N, (int64_t)i * qc.N / 16, qc.l, x, y, z);
      hits += sqdist<float>(kx, ky, kz, x, y, z) < use.r2 ? 1 : 0;
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    if (lane == 0) warp_total[warp] = hits;
    __syncthreads();
    hits = 0;
#pragma unroll
    for (int w = 0; w < SB_WARPS; ++w) hits += warp_total[w];
    // hits per query = hits * N2 / (16 * 512)
    if ((double)hits * kc.N > 2.0 * 16 * SB_THREADS * use.row) {  // the same in all blocks of the cluster
      if (rank == 0 && tid == 0) c.grid[b].irregular = 1;
      return;
    }
    __syncthreads();
  }

#pragma unroll
  for (int e = 0; e < SP_CELLS / SB_THREADS; ++e) hist[tid + e * SB_THREADS] = 0;
  if (tid == 0) crowd = close = 0;

  // This block's share of the sample, PER queries in each direction: 0 searches a's points in b, 1 the other way round.
  // A warp takes one direction, 32 of the keys and half of the queries.
  constexpr int PER = PK_SAMPLE / CL, HALF = (PER + 1) / 2;
  const int dir = warp & 1, slice = (warp >> 1) & (PK_KEYS / 32 - 1), i0 = (warp >> 3) * HALF;
  const bool looks = use.prunes && (dir == 0 || use.both) && i0 < PER;
  float kx, ky, kz, qx[HALF], qy[HALF], qz[HALF], nx[HALF], ny[HALF], nz[HALF];
  if (looks) {  // loaded ahead, looked at behind the first pass
    const SpCloud &qc = pair.c[dir], &kc = pair.c[1 - dir];
    const float *kp = kc.xyz + b * 3 * (int64_t)kc.N, *qp = qc.xyz + b * 3 * (int64_t)qc.N;
    load_xyz(kp, pk_key(slice * 32 + lane, kc.N), kc.l, kx, ky, kz);
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const int s = rank * PER + i0 + i;
      load_xyz(qp, (int64_t)s * qc.N / PK_SAMPLE, qc.l, qx[i], qy[i], qz[i]);
      load_xyz(kp, pk_key(s * (PK_KEYS / PK_SAMPLE), kc.N), kc.l, nx[i], ny[i], nz[i]);
    }
  }
  if (tid < 2) near[tid] = 0;
  float v[7] = {sp_inf(), sp_inf(), sp_inf(), -sp_inf(), -sp_inf(), -sp_inf(), 0.f};
#pragma unroll 4
  for (int j = beg + tid; j < end; j += SB_THREADS) {
    float x, y, z;
    load_xyz(xyz, j, c.l, x, y, z);
    v[0] = fminf(v[0], x), v[1] = fminf(v[1], y), v[2] = fminf(v[2], z);
    v[3] = fmaxf(v[3], x), v[4] = fmaxf(v[4], y), v[5] = fmaxf(v[5], z);
    if (!(fabsf(x) < sp_inf() && fabsf(y) < sp_inf() && fabsf(z) < sp_inf())) v[6] = 1.f;
  }
  float reach[HALF];
  if (looks) {  // nearest sampled key of every query, nearest other one of every key
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      reach[i] = sp_sq3(qx[i] - kx, qy[i] - ky, qz[i] - kz);
      const float e = sp_sq3(nx[i] - kx, ny[i] - ky, nz[i] - kz);
      const float dq = sp_warp_min(reach[i]), dk = sp_warp_min(e > 0.f ? e : sp_inf());
      if (lane == 0) least[dir][0][i0 + i][slice] = dq, least[dir][1][i0 + i][slice] = dk;
    }
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
  if (looks) {
    auto min4 = [](const float(&m)[PK_KEYS / 32]) { return fminf(fminf(m[0], m[1]), fminf(m[2], m[3])); };
    // the geometric mean of the spacings: neither an outlier nor a pair of close keys weighs much
    float lg = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) lg += 0.5f * __log2f(fminf(fmaxf(min4(least[dir][1][i]), 1e-30f), 1e30f));
    const float spacing = exp2f(lg / PER);
    int hits = 0;
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const float r = sqrtf(min4(least[dir][0][i0 + i])) + spacing;
      hits += reach[i] <= r * r ? 1 : 0;
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    if (lane == 0) atomicAdd(&near[dir], hits);
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
  g.pad[0] = g.pad[1] = g.pad[2] = 0;
  if (use.prunes) {
    int within[2] = {0, 0};
#pragma unroll
    for (int o = 0; o < CL; ++o) {
      within[0] += remote(near, o)[0];
      within[1] += remote(near, o)[1];
    }
    constexpr int MOST = PK_SAMPLE * PK_KEYS / 2;
    if (within[0] > MOST || (use.both && within[1] > MOST)) g.irregular = 1;
  }
  if (g.irregular) {  // no search looks at the cloud; the same in all blocks, and nobody leaves before all have read
    if (rank == 0 && tid == 0) c.grid[b] = g;
    sync();
    return;
  }

  if (use.resolves) {
    const float half = 0.5f * ext * (1.f / 256.f);
    float x, y, z;
    load_xyz(xyz, pk_key((warp & (PK_KEYS / 32 - 1)) * 32 + lane, N), c.l, x, y, z);
    int same = 0;
    for (int i = warp / (PK_KEYS / 32); i < PER; i += SB_WARPS / (PK_KEYS / 32)) {
      float u, w, r;
      load_xyz(xyz, pk_key((rank * PER + i) * (PK_KEYS / PK_SAMPLE), N), c.l, u, w, r);
      const float e = fmaxf(fmaxf(fabsf(u - x), fabsf(w - y)), fabsf(r - z));
      same += __popc(__ballot_sync(0xffffffffu, e > 0.f && e <= half));
    }
    if (lane == 0 && same) atomicAdd(remote(&close, 0), same);
  }
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
  g.irregular = 2 * (int64_t)*remote(&crowd, 0) > N;  // complete since the last barrier
  if (use.resolves && *remote(&close, 0) * PK_COARSE > PK_SAMPLE * PK_KEYS) g.irregular = 1;
#pragma unroll
  for (int i = 0; i < MINE; ++i) {
    c.table[b * SP_CELLS + c0 + i] = at;
#pragma unroll
    for (int o = 0; o < CL; ++o) {
      remote(hist, o)[c0 + i] = at;
      at += n[o][i];
    }
  }
  sync();  // the last access to another block's shared memory lies behind every block
  if (rank == 0 && tid == 0) c.grid[b] = g;
  if (g.irregular) return;

#pragma unroll 4
  for (int j = beg + tid; j < end; j += SB_THREADS) {
    float x, y, z;
    load_xyz(xyz, j, c.l, x, y, z);
    const int to = atomicAdd(&hist[sp_cell(x, y, z, g)], 1);
    pts[sp_checked(to, N)] = make_float4(x, y, z, __int_as_float(j));
  }
  if (rank == 0) {
    // padding of the last window: NaN distances are never below or at a bound
    for (int j = N + tid; j < c.windows * SP_WINDOW; j += SB_THREADS)
      pts[j] = make_float4(sp_nan(), sp_nan(), sp_nan(), __int_as_float(0x7fffffff));
  }
}

// One warp per window.  Register r of lane l is element 8 l + r of the network, so that a lane ends up
// with a whole leaf and the distances 1, 2, 4 of the network need no exchange.
constexpr int SW_THREADS = 128;

__global__ void __launch_bounds__(SW_THREADS)
spatial_window_kernel(const __grid_constant__ SpPair pair, int64_t windows0, int64_t windows_total) {
  const int lane = threadIdx.x & 31;
  int64_t w = (int64_t)blockIdx.x * (SW_THREADS / 32) + (threadIdx.x >> 5);
  if (w >= windows_total) return;
  const SpCloud &c = pair.c[w >= windows0];
  if (w >= windows0) w -= windows0;
  const SpGrid g = c.grid[w / c.windows];
  if (g.irregular) return;  // no search looks at it
  float4 *p = reinterpret_cast<float4 *>(c.pts) + w * SP_WINDOW;
  unsigned key[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const unsigned e = 32 * r + lane;
    const float4 q = p[e];
    key[r] = ((__float_as_int(q.w) == 0x7fffffff ? 0xffffffu : sp_fine(q.x, q.y, q.z, g)) << 8) | e;  // padding last
  }
#pragma unroll
  for (int k = 2; k <= SP_WINDOW; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j < 8) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int o = r ^ j;
          if (o > r) {
            const bool up = ((8 * lane + r) & k) == 0;
            const unsigned lo = min(key[r], key[o]), hi = max(key[r], key[o]);
            key[r] = up ? lo : hi;
            key[o] = up ? hi : lo;
          }
        }
      } else {
        const bool keep_low = ((8 * lane & k) == 0) == ((8 * lane & j) == 0);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const unsigned other = __shfl_xor_sync(0xffffffffu, key[r], j >> 3);
          key[r] = keep_low ? min(key[r], other) : max(key[r], other);
        }
      }
    }
  }
  float x[8], y[8], z[8];
  int i[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const float4 q = p[key[r] & 255u];
    x[r] = q.x, y[r] = q.y, z[r] = q.z, i[r] = __float_as_int(q.w);
  }
  __syncwarp();  // every point is in registers before its place is written
  float4 *leaf = p + 8 * lane;
  leaf[0] = make_float4(x[0], x[1], x[2], x[3]);
  leaf[1] = make_float4(x[4], x[5], x[6], x[7]);
  leaf[2] = make_float4(y[0], y[1], y[2], y[3]);
  leaf[3] = make_float4(y[4], y[5], y[6], y[7]);
  leaf[4] = make_float4(z[0], z[1], z[2], z[3]);
  leaf[5] = make_float4(z[4], z[5], z[6], z[7]);
  reinterpret_cast<int4 *>(leaf)[6] = make_int4(i[0], i[1], i[2], i[3]);
  reinterpret_cast<int4 *>(leaf)[7] = make_int4(i[4], i[5], i[6], i[7]);
  // boxes (minima and maxima drop NaN; a leaf of nothing but padding gets an empty box)
  float lo[3] = {sp_inf(), sp_inf(), sp_inf()}, hi[3] = {-sp_inf(), -sp_inf(), -sp_inf()};
  int low = 0x7fffffff;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    lo[0] = fminf(lo[0], x[r]), lo[1] = fminf(lo[1], y[r]), lo[2] = fminf(lo[2], z[r]);
    hi[0] = fmaxf(hi[0], x[r]), hi[1] = fmaxf(hi[1], y[r]), hi[2] = fmaxf(hi[2], z[r]);
    low = min(low, i[r]);
  }
  float4 *box = c.boxes + (w * 32 + lane) * 2;
  box[0] = make_float4(lo[0], lo[1], lo[2], hi[0]);
  box[1] = make_float4(hi[1], hi[2], __int_as_float(low), 0.f);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = sp_warp_min(lo[d]);
    hi[d] = sp_warp_max(hi[d]);
  }
  low = __reduce_min_sync(0xffffffffu, low);
  if (lane == 0) {
    c.wbox[2 * w] = make_float4(lo[0], lo[1], lo[2], hi[0]);
    c.wbox[2 * w + 1] = make_float4(hi[1], hi[2], __int_as_float(low), 0.f);
  }
}

// ---------------------------------------------------------------------------------------------
// K <= 4 nearest keys of every query: one warp per 32 consecutive queries, lane = query.
//   1. The leaf at the position of the query's cell in the key cloud bounds its K-th distance.
//   2. The warp walks the windows and, nearest first, their leaves whose boxes come within the largest
//      bound of its queries; a leaf is scanned when at least one lane's own bound reaches its box.
//   3. A scan evaluates exact distances two keys at a time, every lane the same keys, and branches once
//      per leaf.
// Bound by latency and the L1's return path together (0.6 instructions a cycle and scheduler): for two
// clouds of 16384 points a warp visits 6 to 21 windows, tests 30 to 95 leaves and scans 15 to 30 of them.
// 64 x 16384 x 16384, both directions: 0.28 ms on a surface, 0.63 ms in blobs, plus 0.08 ms for the
// order (sweeping all pairs: 5.8 ms; leaves of 32 points and no look-ahead: 0.41 and 0.88 ms).
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
__device__ __forceinline__ void sp_scan(const float *__restrict__ leaf, float2 nx, float2 ny, float2 nz, float2 one,
                                        SpList<K> &list) {
  float2 d[4];
  sp_leaf_dist(leaf, nx, ny, nz, one, d);
  const float m = sp_min8(d);
  if (m <= list.d[K - 1]) {
    int i[8];
    sp_leaf_index(leaf, i);
    if constexpr (K == 1) {  // only the smallest of the eight can enter: its lowest index
      int at = 0x7fffffff;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        at = min(at, d[u].x == m ? i[2 * u] : 0x7fffffff);
        at = min(at, d[u].y == m ? i[2 * u + 1] : 0x7fffffff);
      }
      list.offer(m, at);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (d[u].x <= list.d[K - 1]) list.offer(d[u].x, i[2 * u]);
        if (d[u].y <= list.d[K - 1]) list.offer(d[u].y, i[2 * u + 1]);
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
  int64_t tasks[2];  // query groups of all clouds
  int64_t blocks0;   // blocks of direction 0
};

template <int K, int MODE>
__global__ void __launch_bounds__(SN_THREADS)
spatial_nn_kernel(const __grid_constant__ SpSearch job, double *__restrict__ sums, float eps, float one_) {
  __shared__ double ssum[SN_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rev = blockIdx.x >= job.blocks0;
  const SpCloud &qc = job.c[rev], &kc = job.c[1 - rev];
  const int64_t task = (blockIdx.x - (rev ? job.blocks0 : 0)) * SN_WARPS + warp;
  double total = 0.0;
  if (task < job.tasks[rev]) {
    const int64_t b = task / qc.groups;
    const int first = (int)(task - b * qc.groups) * SP_GROUP;
    const SpGrid g = kc.grid[b];
    if (!(g.irregular | qc.grid[b].irregular)) {
      const float4 q = sp_point(qc.pts + b * (int64_t)qc.windows * SP_WINDOW * 4, first + lane, qc.windows);
      const bool valid = first + lane < qc.N;
      // minima and maxima drop the NaN of padding lanes
      const SpBox qbox = {sp_warp_min(q.x), sp_warp_min(q.y), sp_warp_min(q.z),
                          sp_warp_max(q.x), sp_warp_max(q.y), sp_warp_max(q.z)};
      const float2 one = make_float2(one_, one_);
      const float2 nx = make_float2(-q.x, -q.x), ny = make_float2(-q.y, -q.y), nz = make_float2(-q.z, -q.z);
      const float *kpts = kc.pts + b * (int64_t)kc.windows * SP_WINDOW * 4;
      const float4 *kbox = kc.boxes + b * (int64_t)kc.windows * 64;
      const float4 *kwin = kc.wbox + b * (int64_t)kc.windows * 2;

      // 1. the seed leaf (whole leaves only: it must hold K keys)
      const int *tab = kc.table + b * SP_CELLS;
      const int e = sp_cell(q.x, q.y, q.z, g);
      const int p0 = __ldg(tab + e), p1 = e + 1 < SP_CELLS ? __ldg(tab + e + 1) : kc.N;
      const int seed = min((p0 + p1) >> 4, (kc.N >> 3) - 1);
      SpList<K> list;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        list.d[c] = sp_inf();
        list.i[c] = MODE == SN_CHAMFER ? -1 : 0x7fffffff;
      }
      sp_scan<K>(sp_leaf(kpts, seed, kc.windows), nx, ny, nz, one, list);
      if constexpr (K > 1) {
        // the seeds come again with their leaf: keep their bound only
        const float bound = list.d[K - 1];
#pragma unroll
        for (int c = 0; c < K; ++c) {
          list.d[c] = bound;
          list.i[c] = 0x7fffffff;
        }
      }
      if (!valid) list.d[K - 1] = -1.f;  // never reached by a distance

      // 2. windows and leaves, beginning with the window of a middle query's seed
      const int home = __shfl_sync(0xffffffffu, seed >> 5, min(16, qc.N - first - 1));
      const float mx = 0.5f * (qbox.lx + qbox.hx), my = 0.5f * (qbox.ly + qbox.hy), mz = 0.5f * (qbox.lz + qbox.hz);
      float gb = sp_warp_max(list.d[K - 1]);
      const int chunks = (kc.windows + 31) >> 5;
      int ch = home >> 5;
      for (int cc = 0; cc < chunks; ++cc) {
        const int s = ch * 32 + lane;
        bool hit = false;
        if (s < kc.windows) hit = sp_box_box(qbox, sp_box(kwin + 2 * s)) <= gb;
        unsigned wmask = __ballot_sync(0xffffffffu, hit);
        unsigned begin = cc == 0 ? wmask & (1u << (home & 31)) : 0u;
        while (wmask) {
          const int wl = __ffs(begin ? begin : wmask) - 1;
          begin = 0u;
          wmask &= ~(1u << wl);
          const int l0 = (ch * 32 + wl) * 32;
          const SpBox mine = sp_box(kbox + 2 * (l0 + lane));
          const float reach = sp_box_box(qbox, mine);
          // leaves in ascending distance of their centres from the group's: only an order, any will do
          const float ex = 0.5f * (mine.lx + mine.hx) - mx, ey = 0.5f * (mine.ly + mine.hy) - my,
                      ez = 0.5f * (mine.lz + mine.hz) - mz;
          const unsigned far = 0xffffffffu;
          unsigned key = (__float_as_uint(ex * ex + ey * ey + ez * ez) & 0x7fffffe0u) | lane;
          if (!(reach <= gb)) key = far;
          // the next leaf is picked and its box fetched while the current one is looked at
          unsigned next = __reduce_min_sync(0xffffffffu, key);
          SpBox box = sp_box(kbox + 2 * (l0 + (next & 31)));
          while (next != far) {
            const int l = l0 + (next & 31);
            if (lane == (next & 31)) key = far;
            const SpBox now = box;
            next = __reduce_min_sync(0xffffffffu, key);
            box = sp_box(kbox + 2 * (l0 + (next & 31)));
            const float bd = sp_point_box(q.x, q.y, q.z, now);
            if (!__any_sync(0xffffffffu, bd <= list.d[K - 1])) continue;
            if (!__any_sync(0xffffffffu, bd < list.d[K - 1])) {
              // at the bound itself a leaf matters only if it can win the tie by index
              const int low = __float_as_int(__ldg(reinterpret_cast<const float *>(kbox + 2 * l) + 6));
              if (!__any_sync(0xffffffffu, bd == list.d[K - 1] && low < list.i[K - 1])) continue;
            }
            sp_scan<K>(sp_leaf(kpts, l, kc.windows), nx, ny, nz, one, list);
            gb = sp_warp_max(list.d[K - 1]);
            if (!(reach <= gb)) key = far;
          }
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

int sp_build(const SpCloud &a, const SpCloud *b, int64_t B, const SpUse &use, cudaStream_t st) {
  const int64_t clouds = b ? 2 * B : B;
  const int big = b && b->N > a.N ? b->N : a.N;
  // Blocks per cloud: as many as leave every block an SM of its own (eight: two thirds of the SMs, for clouds of less than
  // 16384 points).  With two blocks per SM the barriers of the cluster take longer than the halved passes save, and small
  // clouds do not fill many blocks.  1 / 2 / 4 / 8 blocks, us: 40 clouds of 2048 10 / 12 / 14 / 26, 16 of 4096 14 / 13 / 11 /
  // 14, 32 of 4096 13 / 13 / 12 / 18, 8 of 6000 - / - / 12 / 11, 16 of 8192 21 / 17 / 13 / 15, 64 of 8192 25 / 21 / 23 / 40,
  // 8 of 16384 36 / 24 / 16 / 13, 40 of 16384 36 / 24 / 26 / 36, 128 of 16384 39 / 43 / 52 / 79, 20 of 65536 124 / 68 / 39 /
  // 40, 16 of 131072 293 / 140 / 76 / 46.
  // Clouds of the smaller side count by their share of the larger one's points (63 of 1343 and 63 of 16251: 36 / 24 by 1 / 2).
  const int64_t weight = b ? B * ((int64_t)a.N + b->N) / big : B, sms = sm_count();
  int CL = 1;
  while (CL < 4 && weight * CL * 2 <= sms && big >= 3000) CL *= 2;
  if (CL == 4 && weight * 8 <= (big >= 16384 ? sms : sms * 2 / 3) && big >= 4096) CL = 8;
  SpPair pair;
  pair.c[0] = a;
  pair.c[1] = b ? *b : a;
  const void *kern = CL == 8   ? (const void *)spatial_sort_kernel<8>
                     : CL == 4 ? (const void *)spatial_sort_kernel<4>
                     : CL == 2 ? (const void *)spatial_sort_kernel<2>
                               : (const void *)spatial_sort_kernel<1>;
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
  SpUse use_ = use;
  void *args[] = {&pair, &B_, &use_};
  if (cudaLaunchKernelExC(&cfg, kern, args) != cudaSuccess) {
    (void)cudaGetLastError();
    return SP_DECLINED;
  }
  const int64_t w0 = B * a.windows, total = w0 + (b ? B * b->windows : 0);
  const int64_t per = SW_THREADS / 32;
  spatial_window_kernel<<<(unsigned)((total + per - 1) / per), SW_THREADS, 0, st>>>(pair, w0, total);
  return check_launch("spatial_window_kernel");
}

int sp_chamfer(const SpCloud &a, const SpCloud &b, int64_t B, float *dist1, int64_t *idx1, float *dist2, int64_t *idx2,
               double *sums, cudaStream_t st) {
  SpSearch job;
  job.c[0] = a, job.c[1] = b;
  job.dist[0] = dist1, job.dist[1] = dist2;
  job.index[0] = index_out(idx1, 0, B * a.N), job.index[1] = index_out(idx2, 0, B * b.N);
  job.tasks[0] = B * a.groups, job.tasks[1] = B * b.groups;
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
  job.tasks[0] = B * q.groups, job.tasks[1] = 0;
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
