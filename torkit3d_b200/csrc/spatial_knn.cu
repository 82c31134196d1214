// k nearest neighbours for 4 < k <= 64 over spatially ordered clouds (spatial.cuh).
//
// The two-pass selection of knn_twopass_kernel (knn.cu) with the key tiles replaced by the leaves
// that can matter.  A block of four warps serves 32 consecutive queries (lane = query) and shares the
// leaves it looks at.
//   1. 2 * NCH seeds around each lane's own position in the key cloud: minima over NCH key classes, a
//      bound at which at least k class minima lie (k distinct keys): tau0.
//   2. The leaves whose boxes come within the largest tau0 of the 32 queries go to a list, which is then
//      cut to those within one query's own tau0 (lane = leaf, the queries broadcast from shared memory:
//      half the cost of a scan, and a group of far-flung queries lists a hundred leaves for each it needs).
//   3. Class minima over the listed leaves give the tight bound tau1 (about 1.3 k keys are below it).
//      Consecutive keys, which are neighbours, always fall into different classes.
//   4. The list is cut to the leaves within one query's tau1; a second sweep records every leaf with a
//      distance at or below the lane's tau1.
//   5. Exact selection among the recorded leaves, by rank; a query whose record overflows (massive
//      ties) falls back to an exact scan of all keys by one warp.
// All distances are the exactly rounded ones (two keys per packed operation), so the bounds need no
// error analysis.  A bound is found by bisection over the class minima, which stay in registers: any
// value with k minima at or below it will do, and eight steps from the smallest minimum come within 1/256 of the
// best (from 0 the keys of a cloud that lies away from the queries could not be told apart, lists overflowed, and
// 16 x 4096 x 4096, k = 16, ten radii away, took 1.03 ms; now 0.087).
//
// 0.5 instructions a cycle and scheduler, bound by latency (barriers of the bisection, gathers of the
// selection): 16 x 4096 x 4096, k = 16: 0.11 ms plus 0.03 ms for the order (two passes over all keys:
// 0.175 ms); 32 x 2048 x 8192, k = 32: 0.16 + 0.03 ms (0.545 ms).
#include "knn_list.cuh"
#include "spatial.cuh"

namespace tk3d {

namespace {

constexpr int SK_THREADS = 128;
constexpr int SK_WARPS = SK_THREADS / 32;
constexpr int SK_LIST = 2048;  // leaves of the second sweep; more than that and it goes over those of the first one
constexpr int SK_STEPS = 8;

template <int QCAP>
constexpr size_t sk_smem_bytes() {
  return (size_t)QCAP * 32 * 8 + SK_LIST * 2;
}

template <int NCH, int QCAP, int MINB>
__global__ void __launch_bounds__(SK_THREADS, MINB)
spatial_knn_kernel(const __grid_constant__ SpCloud qc, const __grid_constant__ SpCloud kc, int k,
                   float *__restrict__ dist, IndexOut index, float one_) {
  constexpr int CPW = NCH / SK_WARPS;  // class minima of one thread
  constexpr int U = CPW / SP_LEAF;     // leaves per round of classes
  constexpr int SEED = NCH / 4;        // seed leaves: two keys per class
  extern __shared__ __align__(16) unsigned char sk_smem[];
  float *cd = reinterpret_cast<float *>(sk_smem);                // [QCAP][32] exact distances
  int *cand = reinterpret_cast<int *>(sk_smem + QCAP * 32 * 4);  // [QCAP][32] leaves, then key indices
  // Leaves within reach of the group, in the place of the candidates; of one query, in the place of the distances; and
  // those of the second sweep.  Tails of a cloud have long lists (65536 points in blobs, k = 16: up to 1500 leaves;
  // a group that went through all 8192 instead took 1.2 ms by itself).
  constexpr int FIRST = QCAP * 64;
  unsigned short *list0 = reinterpret_cast<unsigned short *>(cand), *list1 = reinterpret_cast<unsigned short *>(cd),
                 *list2 = reinterpret_cast<unsigned short *>(sk_smem + QCAP * 32 * 8);
  __shared__ int counts[2][SK_WARPS][32];
  __shared__ float least[SK_WARPS][32];
  __shared__ int ccnt[32], fcnt[32], hcnt[32];
  __shared__ int nlist[3];
  __shared__ float4 sq[32];  // the queries and their bounds
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
  const int64_t b = blockIdx.x / qc.groups;
  const int first_q = (int)(blockIdx.x - b * qc.groups) * SP_GROUP;
  const SpGrid g = kc.grid[b];
  if (g.irregular | qc.grid[b].irregular) return;  // the whole block

  float4 q = sp_point(qc.pts + b * (int64_t)qc.windows * SP_WINDOW * 4, first_q + lane, qc.windows);
  const bool valid = first_q + lane < qc.N;
  const SpBox qbox = {sp_warp_min(q.x), sp_warp_min(q.y), sp_warp_min(q.z),
                      sp_warp_max(q.x), sp_warp_max(q.y), sp_warp_max(q.z)};
  const float fx = __shfl_sync(0xffffffffu, q.x, 0), fy = __shfl_sync(0xffffffffu, q.y, 0),
              fz = __shfl_sync(0xffffffffu, q.z, 0);
  if (!valid) q = make_float4(fx, fy, fz, q.w);  // padding lanes follow the first query and record nothing
  const float2 one = make_float2(one_, one_);
  const float2 nx = make_float2(-q.x, -q.x), ny = make_float2(-q.y, -q.y), nz = make_float2(-q.z, -q.z);
  const float *kpts = kc.pts + b * (int64_t)kc.windows * SP_WINDOW * 4;
  const float4 *kbox = kc.boxes + b * (int64_t)kc.windows * 64;
  const float4 *kwin = kc.wbox + b * (int64_t)kc.windows * 2;

  if (part == 0) {
    ccnt[lane] = fcnt[lane] = hcnt[lane] = 0;
    if (lane < 3) nlist[lane] = 0;
  }

  // a bound with at least k class minima at or below it, starting from `hi`, which is one, and the smallest
  float cmin[CPW];
  auto kth_bound = [&](float hi) {
    float lo = cmin[0];
#pragma unroll
    for (int c = 1; c < CPW; ++c) lo = fminf(lo, cmin[c]);
    least[part][lane] = lo;
    __syncthreads();
    lo = fminf(fminf(least[0][lane], least[1][lane]), fminf(least[2][lane], least[3][lane]));
#pragma unroll 1
    for (int it = 0; it < SK_STEPS; ++it) {
      const float mid = 0.5f * (lo + hi);
      int n = 0;
#pragma unroll
      for (int c = 0; c < CPW; ++c) n += cmin[c] <= mid ? 1 : 0;
      counts[it & 1][part][lane] = n;
      __syncthreads();
      const int t = counts[it & 1][0][lane] + counts[it & 1][1][lane] + counts[it & 1][2][lane] +
                    counts[it & 1][3][lane];
      if (t >= k) hi = mid;
      else lo = mid;
    }
    return hi;
  };
  auto take = [&](const float *leaf, int c0) {  // class minima c0 .. c0 + 7
    float2 d[4];
    sp_leaf_dist(leaf, nx, ny, nz, one, d);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      cmin[c0 + 2 * u] = fminf(cmin[c0 + 2 * u], d[u].x);
      cmin[c0 + 2 * u + 1] = fminf(cmin[c0 + 2 * u + 1], d[u].y);
    }
  };
#pragma unroll
  for (int c = 0; c < CPW; ++c) cmin[c] = pinf();

  // ---- 1. seeds (whole leaves)
  {
    const int *tab = kc.table + b * SP_CELLS;
    const int e = sp_cell(q.x, q.y, q.z, g);
    const int p0 = __ldg(tab + e), p1 = e + 1 < SP_CELLS ? __ldg(tab + e + 1) : kc.N;
    const int seed = min(max(((p0 + p1) >> 4) - SEED / 2, 0), (kc.N >> 3) - SEED);
#pragma unroll
    for (int i = 0; i < SEED / SK_WARPS; ++i)
      take(sp_leaf(kpts, seed + i * SK_WARPS + part, kc.windows), 8 * (i % U));
  }
  float top = cmin[0];
#pragma unroll
  for (int c = 1; c < CPW; ++c) top = fmaxf(top, cmin[c]);
  counts[1][part][lane] = __float_as_int(top);  // distances are >= 0: their patterns order like the values
  __syncthreads();
  top = __int_as_float(max(max(counts[1][0][lane], counts[1][1][lane]), max(counts[1][2][lane], counts[1][3][lane])));
  const float tau0 = kth_bound(top);

  // ---- 2. leaves within reach
  const float gb0 = sp_warp_max(valid ? tau0 : -1.f);
  {
    int turn = 0;
    for (int s0 = 0; s0 < kc.windows; s0 += 32) {
      bool hit = false;
      if (s0 + lane < kc.windows) hit = sp_box_box(qbox, sp_box(kwin + 2 * (s0 + lane))) <= gb0;
      unsigned wmask = __ballot_sync(0xffffffffu, hit);
      while (wmask) {
        const int l = (s0 + __ffs(wmask) - 1) * 32 + lane;
        wmask &= wmask - 1;
        if ((turn++ & (SK_WARPS - 1)) != part) continue;
        hit = sp_box_box(qbox, sp_box(kbox + 2 * l)) <= gb0;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(&nlist[0], __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (hit && at < FIRST) list0[at] = (unsigned short)l;
      }
    }
  }
  if (part == 0) sq[lane] = make_float4(q.x, q.y, q.z, valid ? tau0 : -1.f);
  __syncthreads();
  // leaves of `from` (or all of them) within reach of one of the queries go to `to`
  auto cut = [&](const unsigned short *from, int count, unsigned short *to, int room, int *total) {
    for (int l0 = part * 32; l0 < count; l0 += SK_THREADS) {
      const int l = l0 + lane < count ? (from ? from[l0 + lane] : l0 + lane) : -1;
      bool hit = false;
      if (l >= 0) {
        const SpBox box = sp_box(kbox + 2 * l);
#pragma unroll 4
        for (int e = 0; e < 32; ++e) {
          const float4 w = sq[e];
          hit |= sp_point_box(w.x, w.y, w.z, box) <= w.w;
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      int at = 0;
      if (lane == 0 && m) at = atomicAdd(total, __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
      if (hit && at < room) to[at] = (unsigned short)l;
    }
  };
  const bool most = nlist[0] > FIRST;
  cut(most ? nullptr : list0, most ? kc.windows * 32 : nlist[0], list1, FIRST, &nlist[1]);
  __syncthreads();
  const bool all = nlist[1] > FIRST;
  const int n1 = all ? kc.windows * 32 : nlist[1];

  // ---- 3. class minima over the listed leaves
#pragma unroll
  for (int c = 0; c < CPW; ++c) cmin[c] = pinf();
  for (int li = part; li < n1; li += SK_WARPS * U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = li + u * SK_WARPS;
      if (i < n1) take(sp_leaf(kpts, all ? i : list1[i], kc.windows), 8 * u);
    }
  }
  const float tau1 = kth_bound(tau0);

  // ---- 4. leaves with a distance at or below tau1
  if (part == 0) sq[lane].w = valid ? tau1 : -1.f;
  __syncthreads();
  cut(all ? nullptr : list1, n1, list2, SK_LIST, &nlist[2]);
  __syncthreads();
  const unsigned short *last = nlist[2] <= SK_LIST ? list2 : all ? nullptr : list1;
  const int n2 = nlist[2] <= SK_LIST ? nlist[2] : n1;
  // the next float above tau1 (tau1 >= 0): "below it" is "at or below tau1"
  const float thr = valid ? (tau1 < pinf() ? __int_as_float(__float_as_int(tau1) + 1) : tau1) : -pinf();
  const unsigned cnt_addr = (unsigned)__cvta_generic_to_shared(ccnt + lane);
  const unsigned cand_addr = (unsigned)__cvta_generic_to_shared(cand + lane);
#pragma unroll 2
  for (int li = part; li < n2; li += SK_WARPS) {
    const int leaf = last ? last[li] : li;
    float2 d[4];
    sp_leaf_dist(sp_leaf(kpts, leaf, kc.windows), nx, ny, nz, one, d);
    // padding keys have NaN distances, which the minima drop; a leaf of nothing else gives +inf
    kt_append<32 * 4, QCAP>(fminf(sp_min8(d), pinf()), thr, cnt_addr, cand_addr, leaf);
  }
  __syncthreads();

  // ---- 5. exact selection, four threads per query (as in knn_twopass_kernel)
  const int n = ccnt[lane];
  if (valid && n <= QCAP) {
    int hits = 0;
    for (int c = part; c < n; c += SK_WARPS) {
      const float *leaf = sp_leaf(kpts, cand[c * 32 + lane], kc.windows);
      float2 d2[4];
      int ji[8];
      sp_leaf_dist(leaf, nx, ny, nz, one, d2);
      sp_leaf_index(leaf, ji);
      int first = -1;
      float firstd = pinf();
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = (e & 1) ? d2[e >> 1].y : d2[e >> 1].x;
        if (d < thr) {
          ++hits;
          if (first < 0) {
            first = ji[e];
            firstd = d;
          } else {
            const int row = n + atomicAdd(&fcnt[lane], 1);
            if (row < QCAP) {
              cd[row * 32 + lane] = d;
              cand[row * 32 + lane] = ji[e];
            }
          }
        }
      }
      cd[c * 32 + lane] = firstd;
      cand[c * 32 + lane] = first;
    }
    if (hits) atomicAdd(&hcnt[lane], hits);
  }
  __syncthreads();
  const int rows = n + fcnt[lane];
  const bool listed = n <= QCAP && rows <= QCAP && hcnt[lane] >= k;
  if (valid && listed) {
    const int64_t orow = (b * qc.N + __float_as_int(q.w)) * (int64_t)k;
    float *od = dist + orow;
    for (int f = part; f < rows; f += SK_WARPS) {
      const int j = cand[f * 32 + lane];
      if (j < 0) continue;
      const float d = cd[f * 32 + lane];
      int rank = 0, same = 0;
#pragma unroll 8
      for (int o = 0; o < rows; ++o) {
        const float w = cd[o * 32 + lane];  // empty slots hold +inf
        rank += w < d ? 1 : 0;
        same += w == d ? 1 : 0;
      }
      if (same > 1) {
        for (int o = 0; o < rows; ++o)
          rank += (cd[o * 32 + lane] == d && (unsigned)cand[o * 32 + lane] < (unsigned)j) ? 1 : 0;  // -1 is last
      }
      if (rank < k) {
        od[rank] = d;
        index.put(orow + rank, j);
      }
    }
  }
  // queries whose lists overflowed: one warp each
  unsigned left = __ballot_sync(0xffffffffu, valid && !listed);
  __syncthreads();  // every thread is done with the lists
  int turn = 0;
  while (left) {
    const int fc = __ffs(left) - 1;
    left &= left - 1;
    if ((turn++ & (SK_WARPS - 1)) != part) continue;
    const int fq = __shfl_sync(0xffffffffu, __float_as_int(q.w), fc);
    kt_exact_scan<32>(qc.xyz + b * 3 * (int64_t)qc.N, kc.xyz + b * 3 * (int64_t)kc.N, fq, kc.N, k, qc.l, kc.l, cd + fc,
                      cand + fc, dist, index, (b * qc.N + fq) * (int64_t)k);
  }
}

template <int NCH, int QCAP, int MINB>
int sk_launch(const SpCloud &q, const SpCloud &kc, int64_t B, int k, float *dist, IndexOut index, cudaStream_t st) {
  constexpr size_t smem = sk_smem_bytes<QCAP>();
  if (smem + 2048 > 48 * 1024)
    TK3D_CUDA(raise_smem_limit((const void *)spatial_knn_kernel<NCH, QCAP, MINB>, (int)smem));
  spatial_knn_kernel<NCH, QCAP, MINB><<<(unsigned)(B * q.groups), SK_THREADS, smem, st>>>(q, kc, k, dist, index, 1.0f);
  return check_launch("spatial_knn_kernel");
}

}  // namespace

// 4 < k <= 64
int sp_knn_select(const SpCloud &q, const SpCloud &kc, int64_t B, int k, float *dist, IndexOut index,
                  cudaStream_t st) {
  if (k <= 16) return sk_launch<32, 56, 8>(q, kc, B, k, dist, index, st);
  if (k <= 32) return sk_launch<64, 104, 7>(q, kc, B, k, dist, index, st);
  return sk_launch<128, 192, 4>(q, kc, B, k, dist, index, st);
}

}  // namespace tk3d

TK3D_BOUNDS_TU(spatial_knn)
