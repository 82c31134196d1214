// Ball query over spatially ordered clouds (spatial.cuh).
//
// A block of four warps serves 32 consecutive queries (lane = query):
//   1. leaves whose boxes come within the radius of the group's box go to a list, which is cut to those
//      within the radius of one query (lane = leaf, the queries broadcast from shared memory);
//   2. the listed leaves are scanned, a leaf per warp, and every hit's original index is appended to
//      its query's list;
//   3. a hit's place in the row is the number of hits with a lower index (four threads per query).
// Hits are decided on the exactly rounded distance, and a non-finite point or query has none, whatever
// the boxes say.  Where the balls are dense (as the sort saw it from a sample, or more than SQ_HITS hits
// or SQ_LIST leaves here), or the order is no good (SpGrid::irregular), the block sweeps the keys in
// index order instead, which ends as soon as all rows are full.
//
// 32 x 1024 queries of 8192 keys, 20 hits, k = 32: 0.041 ms plus 0.030 ms for the order (a sweep of all
// keys by the same blocks: 0.137 ms); a third of it is the counting of places, a third the lists.
#include "ball_sweep.cuh"
#include "spatial.cuh"

namespace tk3d {

namespace {

constexpr int SQ_THREADS = 128;
constexpr int SQ_WARPS = SQ_THREADS / 32;
constexpr int SQ_LIST = 512;
constexpr int SQ_HITS = 160;

struct BallSmem {
  unsigned short list[2][SQ_LIST];
  int hit[SQ_HITS][32];  // original indices
};

__global__ void __launch_bounds__(SQ_THREADS, 8)
spatial_ball_kernel(const __grid_constant__ SpCloud qc, const __grid_constant__ SpCloud kc, float r2, int k,
                    IndexOut index, float one_) {
  __shared__ union {
    BallSmem b;
    BallSweepSmem<SQ_WARPS> s;
  } sm;
  __shared__ float4 sq[32];
  __shared__ int cnt[32];
  __shared__ int nlist[2];
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
  const int64_t b = blockIdx.x / qc.groups;
  const int first_q = (int)(blockIdx.x - b * qc.groups) * SP_GROUP;
  bool sweep = kc.grid[b].irregular | qc.grid[b].irregular;
  const bool valid = first_q + lane < qc.N;
  float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (sweep) {  // the pair may not have been ordered at all: queries as they come
    q.w = __int_as_float(valid ? first_q + lane : 0);
    if (valid) load_xyz(qc.xyz + b * 3 * (int64_t)qc.N, first_q + lane, qc.l, q.x, q.y, q.z);
  } else {
    q = sp_point(qc.pts + b * (int64_t)qc.windows * SP_WINDOW * 4, first_q + lane, qc.windows);
  }
  const int64_t row = (b * qc.N + (valid ? __float_as_int(q.w) : 0)) * (int64_t)k;

  if (!sweep) {
    const SpBox qbox = {sp_warp_min(q.x), sp_warp_min(q.y), sp_warp_min(q.z),
                        sp_warp_max(q.x), sp_warp_max(q.y), sp_warp_max(q.z)};
    const float *kpts = kc.pts + b * (int64_t)kc.windows * SP_WINDOW * 4;
    const float4 *kbox = kc.boxes + b * (int64_t)kc.windows * 64;
    const float4 *kwin = kc.wbox + b * (int64_t)kc.windows * 2;
    if (part == 0) {
      cnt[lane] = 0;
      if (lane < 2) nlist[lane] = 0;
      sq[lane] = make_float4(q.x, q.y, q.z, 0.f);  // padding queries are NaN: within reach of nothing
    }
    __syncthreads();

    // ---- 1. leaves within reach
    auto append = [&](bool hit, int l, unsigned short *to, int *total) {
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      int at = 0;
      if (lane == 0 && m) at = atomicAdd(total, __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
      if (hit && at < SQ_LIST) to[at] = (unsigned short)l;
    };
    int turn = 0;
    for (int s0 = 0; s0 < kc.windows; s0 += 32) {
      bool hit = false;
      if (s0 + lane < kc.windows) hit = sp_box_box(qbox, sp_box(kwin + 2 * (s0 + lane))) < r2;
      unsigned wmask = __ballot_sync(0xffffffffu, hit);
      while (wmask) {
        const int l = (s0 + __ffs(wmask) - 1) * 32 + lane;
        wmask &= wmask - 1;
        if ((turn++ & (SQ_WARPS - 1)) != part) continue;
        append(sp_box_box(qbox, sp_box(kbox + 2 * l)) < r2, l, sm.b.list[0], &nlist[0]);
      }
    }
    __syncthreads();
    const int n0 = nlist[0];
    sweep = n0 > SQ_LIST;
    if (!sweep) {
      for (int l0 = part * 32; l0 < n0; l0 += SQ_THREADS) {
        const int l = l0 + lane < n0 ? sm.b.list[0][l0 + lane] : -1;
        bool hit = false;
        if (l >= 0) {
          const SpBox box = sp_box(kbox + 2 * l);
#pragma unroll 4
          for (int e = 0; e < 32; ++e) {
            const float4 w = sq[e];
            // minima and maxima drop NaN: ask the query itself
            hit |= sp_point_box(w.x, w.y, w.z, box) < r2 && w.x == w.x;
          }
        }
        append(hit, l, sm.b.list[1], &nlist[1]);
      }
      __syncthreads();

      // ---- 2. hits
      const int n1 = nlist[1];
      const float2 one = make_float2(one_, one_);
      const float2 nx = make_float2(-q.x, -q.x), ny = make_float2(-q.y, -q.y), nz = make_float2(-q.z, -q.z);
      const float lim = valid ? r2 : 0.f;  // no distance is below 0
#pragma unroll 2
      for (int li = part; li < n1; li += SQ_WARPS) {
        const float *leaf = sp_leaf(kpts, sm.b.list[1][li], kc.windows);
        float2 d[4];
        sp_leaf_dist(leaf, nx, ny, nz, one, d);
        if (sp_min8(d) < lim) {
          int i[8], n = 0;
          sp_leaf_index(leaf, i);
#pragma unroll
          for (int u = 0; u < 4; ++u) n += (d[u].x < lim ? 1 : 0) + (d[u].y < lim ? 1 : 0);
          int at = atomicAdd(&cnt[lane], n);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (((u & 1) ? d[u >> 1].y : d[u >> 1].x) < lim) {
              if (at < SQ_HITS) sm.b.hit[at][lane] = i[u];
              ++at;
            }
          }
        }
      }
      __syncthreads();
      sweep = __any_sync(0xffffffffu, cnt[lane] > SQ_HITS);  // the same in every warp
    }
  }
  if (sweep) {
    __syncthreads();  // the lists are dead
    float x = 0.f, y = 0.f, z = 0.f;
    if (valid) x = q.x, y = q.y, z = q.z;
    ball_sweep<SQ_WARPS>(kc.xyz + b * 3 * (int64_t)kc.N, kc.N, kc.l, x, y, z, valid, r2, k, row, index, sm.s);
    return;
  }

  // ---- 3. rows
  const int n = valid ? cnt[lane] : 0;
  int low = 0x7fffffff;
  for (int o = 0; o < n; ++o) low = min(low, sm.b.hit[o][lane]);
  for (int f = part; f < n; f += SQ_WARPS) {
    const int j = sm.b.hit[f][lane];
    int rank = 0;
#pragma unroll 8
    for (int o = 0; o < n; ++o) rank += sm.b.hit[o][lane] < j ? 1 : 0;
    if (rank < k) index.put(row + rank, j);
  }
  if (valid)
    for (int c = n + part; c < k; c += SQ_WARPS) index.put(row + c, n > 0 ? low : -1);
}

}  // namespace

int ball_query_sweep_f32(const float *query, const float *key, int64_t B, int64_t N1, int64_t N2, float r2, int k,
                         const IndexOut &index, XyzLayout ql, XyzLayout kl, cudaStream_t st);

int sp_ball_query(const float *query, const float *key, int64_t B, int64_t N1, int64_t N2, int channel_first, float r2,
                  int k, void *index, int index32, void *scratch, cudaStream_t st) {
  const int64_t step = sp_batch(B, N1, N2);
  char *at = sp_align_ptr(scratch);
  for (int64_t b0 = 0; b0 < B; b0 += step) {
    const int64_t n = b0 + step < B ? step : B - b0;
    const SpCloud cq = sp_cloud(query + b0 * 3 * N1, channel_first, n, N1, at);
    const SpCloud ck = sp_cloud(key + b0 * 3 * N2, channel_first, n, N2, at + sp_cloud_bytes(n, N1));
    int rc = sp_build(cq, &ck, n, SpUse{false, false, true, k, r2}, st);
    const IndexOut io = index_out((char *)index + b0 * N1 * k * (index32 ? 4 : 8), index32, n * N1 * k);
    if (rc == SP_DECLINED) {
      rc = ball_query_sweep_f32(cq.xyz, ck.xyz, n, N1, N2, r2, k, io, cq.l, ck.l, st);
    } else if (!rc) {
      spatial_ball_kernel<<<(unsigned)(n * cq.groups), SQ_THREADS, 0, st>>>(cq, ck, r2, k, io, 1.0f);
      rc = check_launch("spatial_ball_kernel");
    }
    if (rc) return rc;
  }
  return TK3D_OK;
}

}  // namespace tk3d

TK3D_BOUNDS_TU(spatial_ball)
