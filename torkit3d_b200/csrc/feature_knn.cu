// Brute-force k nearest neighbours in a C-dimensional feature space (DGCNN's dynamic graph:
// torkit3d/models/classification/dgcnn.py:58-61 calls torkit3d/ops/native.py:4-30, cdist + topk,
// on [B, C, N] features).
//
// Squared distance of a (query, key) pair: acc = 0; for c = 0 .. C-1: acc = fma(d_c, d_c, acc) with
// d_c = key_c - query_c -- one rounding per channel, summed in channel order, which a CPU loop with
// fmaf() reproduces bit for bit.  (The reference's cdist goes through a matrix product and is
// itself only accurate to about 1e-6 of |q|^2 + |r|^2.)
//
// With scratch the tensor cores find the pairs that can matter (feature_filter.cu: k <= 48, C <= 128, 256 to 65536 keys);
// this kernel evaluates all pairs, for the calls and the groups of queries that are left.
//
// Every warp owns four queries; the eight warps of a block share tiles of 256 keys, staged 16 channels at
// a time with asynchronous copies into two buffers.  Lane l holds the 4 x 8 distances of its queries to
// keys 2l, 2l + 1 of each 64 in registers and advances two keys per packed operation (eight queries per
// warp halve the loads per operation, but leave 16 warps on an SM, and were 10 % slower).
// Selection: distances that can enter a query's list are appended to a 64-entry buffer in shared
// memory; 32 of them at a time are sorted across the warp's lanes (bitonic, on the 64-bit word of
// distance bits and index) and merged with the list.  A list of 32 * KS entries is kept sorted; a block
// of 32 new entries first meets the topmost 32, of which the lower half stays, and the exchange then
// goes down the list.  Ties go to the lower index; rows come out sorted.
//
// 32 x 1024 x 1024, 64 channels, k = 20: 0.229 ms, point-major tensors 0.298 (0.391 with unpadded rows); one key per
// lane and one candidate at a time into the list took 0.400 and 0.422 ms.  Half of the issue slots are the packed
// operations, the rest mostly selection.
#include <limits.h>

#include "feature_filter.cuh"
#include "tk3d_common.cuh"

namespace tk3d {
namespace {

constexpr int FK_THREADS = 256;
constexpr int FK_WARPS = FK_THREADS / 32;
constexpr int FK_QW = 4;    // queries per warp
constexpr int FK_KT = 256;  // keys per tile
constexpr int FK_CS = 16;   // channels per slice
constexpr int FK_BUF = 64;  // buffered candidates per query: fewer than 32, and up to 32 more
constexpr unsigned FULL = 0xffffffffu;

using u64 = unsigned long long;

// Row lengths: point-major tensors are staged along the channels, sixteen rows at a time, and rows of 256 words would
// meet in one bank; 258 spread sixteen channels of two keys over all banks, 36 those of two queries over half of them.
template <int KS, bool POINTS>
struct FkSmem {
  float k[2][FK_CS][POINTS ? FK_KT + 2 : FK_KT];
  float q[2][FK_CS][POINTS ? FK_QW * FK_WARPS + 4 : FK_QW * FK_WARPS];
  u64 buf[FK_QW * FK_WARPS][FK_BUF];
  u64 list[FK_QW * FK_WARPS][32 * KS];
};

// BYTES (4 or 16) bytes, or zeros where the source does not exist.
template <int BYTES>
__device__ __forceinline__ void fk_copy(float *dst, const float *src, bool there) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "n"(BYTES), "r"(there ? BYTES : 0)
               : "memory");
}

__device__ __forceinline__ u64 fk_exchange(u64 v, int o, bool low) {
  const u64 w = __shfl_xor_sync(FULL, v, o);
  return (w < v) == low ? w : v;
}
// Sorts a bitonic sequence over the lanes.
__device__ __forceinline__ u64 fk_merge(u64 v, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fk_exchange(v, o, (lane & o) == 0);
  return v;
}
__device__ __forceinline__ u64 fk_sort(u64 v, int lane) {
#pragma unroll
  for (int n = 2; n <= 32; n <<= 1)
#pragma unroll
    for (int o = n >> 1; o > 0; o >>= 1) v = fk_exchange(v, o, ((lane & o) == 0) == ((lane & n) == 0));
  return v;
}

// Takes the first 32 buffered candidates (of `n`) into the list; returns the list's k-th entry.
template <int KS>
__device__ __noinline__ u64 fk_flush(u64 *buf, u64 *list, int n, int k, int lane) {
  const u64 none = 0x7f8000007fffffffull;  // (+inf, INT_MAX): orders after every real entry
  __syncwarp();
  u64 v = fk_sort(lane < n ? buf[lane] : none, lane);
  if (lane + 32 < n) buf[lane] = buf[lane + 32];
  v = __shfl_xor_sync(FULL, v, 31);  // descending, against the ascending list
  const u64 top = list[32 * (KS - 1) + lane];
  v = fk_merge(v < top ? v : top, lane);
#pragma unroll
  for (int s = KS - 2; s >= 0; --s) {
    const u64 up = __shfl_xor_sync(FULL, v, 31), mine = list[32 * s + lane];
    list[32 * (s + 1) + lane] = fk_merge(up < mine ? mine : up, lane);
    v = fk_merge(up < mine ? up : mine, lane);
  }
  list[lane] = v;
  __syncwarp();
  return list[k - 1];
}

// KS: list capacity 32 * KS >= k.  LAYOUT: point-major tensors [B, N, C], or channel-first [B, C, N]
// copied by four bytes, or by sixteen (N1 and N2 multiples of four, 16-byte aligned tensors).
enum { FK_POINTS = 0, FK_CHANNELS = 1, FK_CHANNELS16 = 2 };

// LEFT: only the groups that have a query without a result (a negative count, see ff_knn), a block for each.  A template
// argument: as a test of `counts` in every call's loop the kernel took 119 us instead of 114 (2 x 1289 x 1289, 71 channels).
template <int KS, int LAYOUT, bool LEFT>
__global__ void __launch_bounds__(FK_THREADS, KS <= 2 ? 3 : 2)
feature_knn_kernel(const float *__restrict__ query, const float *__restrict__ key, int C, int N1, int N2, int k,
                   float *__restrict__ dist, int64_t *__restrict__ index, int64_t blocks_total,
                   const int *__restrict__ counts) {
  extern __shared__ __align__(16) unsigned char fk_smem[];
  constexpr int QW = FK_QW, V = LAYOUT == FK_CHANNELS16 ? 4 : 1;
  constexpr bool CF = LAYOUT != FK_POINTS;
  using Smem = FkSmem<KS, LAYOUT == FK_POINTS>;
  Smem &sm = *reinterpret_cast<Smem *>(fk_smem);
  constexpr int QT = QW * FK_WARPS;
  static_assert(!LEFT || QT == FF_GROUP, "the filter gives up groups of this size");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunks = (N1 + QT - 1) / QT;
  const int slices = (C + FK_CS - 1) / FK_CS;
  const float pinf = __int_as_float(0x7f800000);

  for (int64_t blk = blockIdx.x; blk < blocks_total; blk += gridDim.x) {
    const int64_t b = blk / chunks;
    const int q0 = (int)(blk % chunks) * QT;
    if (LEFT && !__syncthreads_or(tid < QT && q0 + tid < N1 && counts[b * N1 + q0 + tid] < 0)) return;
    const float *qb = query + b * (int64_t)C * N1;
    const float *kb = key + b * (int64_t)C * N2;
    // slice `s` of the tile at key j0 goes to buffer `to`
    auto stage = [&](int j0, int s, int to) {
      const int c0 = s * FK_CS;
#pragma unroll
      for (int r = 0; r < (FK_CS * QT / V + FK_THREADS - 1) / FK_THREADS; ++r) {
        const int e = (tid + r * FK_THREADS) * V;
        if (FK_CS * QT / V < FK_THREADS && e >= FK_CS * QT) break;
        const int c = CF ? e / QT : e % FK_CS, i = CF ? e % QT : e / FK_CS;
        const bool there = c0 + c < C && q0 + i < N1;
        const int64_t off = CF ? (int64_t)(c0 + c) * N1 + q0 + i : (int64_t)(q0 + i) * C + c0 + c;
        fk_copy<4 * V>(&sm.q[to][c][i], qb + (there ? off : 0), there);
      }
#pragma unroll
      for (int r = 0; r < FK_CS * FK_KT / V / FK_THREADS; ++r) {
        const int e = (tid + r * FK_THREADS) * V;
        const int c = CF ? e / FK_KT : e % FK_CS, j = CF ? e % FK_KT : e / FK_CS;
        const bool there = c0 + c < C && j0 + j < N2;
        const int64_t off = CF ? (int64_t)(c0 + c) * N2 + j0 + j : (int64_t)(j0 + j) * C + c0 + c;
        fk_copy<4 * V>(&sm.k[to][c][j], kb + (there ? off : 0), there);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float thd[QW];
    int thi[QW], cnt[QW];
#pragma unroll
    for (int a = 0; a < QW; ++a) {
      thd[a] = pinf;
      thi[a] = INT_MAX;
      cnt[a] = 0;
#pragma unroll
      for (int s = 0; s < KS; ++s) sm.list[warp * QW + a][32 * s + lane] = 0x7f8000007fffffffull;
    }

    stage(0, 0, 0);
    int at = 0;
    for (int j0 = 0; j0 < N2; j0 += FK_KT) {
      float2 acc[QW][4];
#pragma unroll
      for (int a = 0; a < QW; ++a)
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[a][p] = make_float2(0.f, 0.f);

      for (int s = 0; s < slices; ++s, at ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this slice has landed, and the other buffer has been consumed
        if (s + 1 < slices) stage(j0, s + 1, at ^ 1);
        else if (j0 + FK_KT < N2) stage(j0 + FK_KT, 0, at ^ 1);
#pragma unroll 2
        for (int c = 0; c < FK_CS; ++c) {
          float2 kv[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) kv[p] = *reinterpret_cast<const float2 *>(&sm.k[at][c][64 * p + 2 * lane]);
#pragma unroll
          for (int a0 = 0; a0 < QW; a0 += 4) {
            const float4 qv = *reinterpret_cast<const float4 *>(&sm.q[at][c][warp * QW + a0]);
            const float q[4] = {-qv.x, -qv.y, -qv.z, -qv.w};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              const float2 q2 = make_float2(q[a], q[a]);
#pragma unroll
              for (int p = 0; p < 4; ++p) {
                const float2 df = __fadd2_rn(kv[p], q2);
                acc[a0 + a][p] = __ffma2_rn(df, df, acc[a0 + a][p]);
              }
            }
          }
        }
      }

      // Selection: this warp's queries against the 256 keys of the tile.
#pragma unroll
      for (int a = 0; a < QW; ++a) {
        u64 *buf = sm.buf[warp * QW + a], *list = sm.list[warp * QW + a];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int j = j0 + 64 * (e >> 1) + 2 * lane + (e & 1);
          const float d = (e & 1) ? acc[a][e >> 1].y : acc[a][e >> 1].x;
          const bool in = j < N2 && (d < thd[a] || (d == thd[a] && j < thi[a]));
          const unsigned mask = __ballot_sync(FULL, in);
          if (mask == 0) continue;
          if (in)
            buf[cnt[a] + __popc(mask & ((1u << lane) - 1u))] =
                ((u64)__float_as_uint(d) << 32) | (unsigned)j;  // d >= +0: the bits order like the value
          cnt[a] += __popc(mask);
          if (cnt[a] >= 32) {
            const u64 last = fk_flush<KS>(buf, list, cnt[a], k, lane);
            cnt[a] -= 32;
            thd[a] = __uint_as_float((unsigned)(last >> 32));
            thi[a] = (int)(unsigned)last;
          }
        }
      }
    }

#pragma unroll
    for (int a = 0; a < QW; ++a) {
      const int qi = q0 + warp * QW + a;
      if (qi < N1) {
        u64 *list = sm.list[warp * QW + a];
        if (cnt[a] > 0) fk_flush<KS>(sm.buf[warp * QW + a], list, cnt[a], k, lane);
        float *od = dist + (b * N1 + qi) * (int64_t)k;
        int64_t *oi = index + (b * N1 + qi) * (int64_t)k;
        for (int m = lane; m < k; m += 32) {
          const u64 v = list[m];
          od[m] = __uint_as_float((unsigned)(v >> 32));
          oi[m] = (unsigned)v == 0x7fffffffu ? (int64_t)-1 : (int64_t)(unsigned)v;  // only with NaN inputs
        }
      }
    }
    if (LEFT) return;
    __syncthreads();  // the next task's first slice may land in a buffer that a slower warp still reads
  }
}

template <int KS, bool LEFT>
int launch(const float *query, const float *key, int64_t B, int C, int N1, int N2, int k, bool cf, float *dist,
           int64_t *index, const int *counts, cudaStream_t st) {
  constexpr int QT = FK_QW * FK_WARPS;
  const int64_t total = B * ((N1 + QT - 1) / QT);
  const int64_t cap = (int64_t)sm_count() * 32;
  const unsigned grid = (unsigned)(LEFT || total < cap ? total : cap);
  const size_t smem = cf ? sizeof(FkSmem<KS, false>) : sizeof(FkSmem<KS, true>);
  const bool wide = N1 % 4 == 0 && N2 % 4 == 0 &&
                    ((reinterpret_cast<uintptr_t>(query) | reinterpret_cast<uintptr_t>(key)) & 15) == 0;
  auto kern = !cf    ? feature_knn_kernel<KS, FK_POINTS, LEFT>
              : wide ? feature_knn_kernel<KS, FK_CHANNELS16, LEFT>
                     : feature_knn_kernel<KS, FK_CHANNELS, LEFT>;
  TK3D_CUDA(raise_smem_limit((const void *)kern, (int)smem));
  kern<<<grid, FK_THREADS, smem, st>>>(query, key, C, N1, N2, k, dist, index, total, counts);
  return check_launch("feature_knn_kernel");
}

}  // namespace
}  // namespace tk3d

using namespace tk3d;

namespace tk3d {
namespace {
// Five launches and a scratch buffer against one launch.  On the device, all pairs / filtered, us: 4 x 512 x 512, 16 channels
// (5e7 by the measure below) 21 / 20, 8 x 300 x 300, 100 channels (9.5e7) 39 / 30, 1 x 1024 x 1024, 64 channels (1e8) 53 / 35;
// but a caller that launches an EdgeConv layer's forward and backward waits for its own launches up to about 3e8: 5 x 737 x
// 737, 37 channels (1.9e8) 168 / 186 for the whole pass, 2 x 1289 x 1289, 71 (3.4e8) 170 / 179, 1 x 1780 x 1780, 94 (4e8)
// 242 / 207.
bool ff_pays(int64_t B, int64_t C, int64_t N1, int64_t N2) { return (double)B * N1 * N2 * (C + 32) >= 3.5e8; }
}  // namespace
}  // namespace tk3d

extern "C" size_t tk3d_feature_knn_scratch_bytes(int64_t B, int64_t C, int64_t N1, int64_t N2, int64_t k, int dtype) {
  return dtype == TK3D_F32 && ff_pays(B, C, N1, N2) ? ff_scratch_bytes(B, C, N1, N2, k) : 0;
}

extern "C" int tk3d_feature_knn(const void *query, const void *key, int64_t B, int64_t C, int64_t N1, int64_t N2,
                                int64_t k, int channel_first, void *dist, int64_t *index, int dtype, void *stream) {
  return tk3d_feature_knn_ws(query, key, B, C, N1, N2, k, channel_first, dist, index, nullptr, 0, dtype, stream);
}

extern "C" int tk3d_feature_knn_ws(const void *query, const void *key, int64_t B, int64_t C, int64_t N1, int64_t N2,
                                   int64_t k, int channel_first, void *dist, int64_t *index, void *scratch,
                                   size_t scratch_bytes, int dtype, void *stream) {
  TK3D_RANGE("tk3d_feature_knn");
  TK3D_REQUIRE(dtype == TK3D_F32 || dtype == TK3D_F64, TK3D_ERR_DTYPE, "feature_knn: dtype %d", dtype);
  TK3D_REQUIRE(dtype == TK3D_F32, TK3D_ERR_UNSUPPORTED, "feature_knn: float32 only");
  TK3D_REQUIRE(B >= 0 && N1 >= 0 && N2 >= 0 && C >= 1, TK3D_ERR_SHAPE,
               "feature_knn: bad size (B=%lld C=%lld N1=%lld N2=%lld)", (long long)B, (long long)C, (long long)N1,
               (long long)N2);
  TK3D_REQUIRE(N1 < (1LL << 30) && N2 < (1LL << 30) && C < (1LL << 20), TK3D_ERR_SHAPE,
               "feature_knn: clouds limited to 2^30 points and 2^20 channels");
  TK3D_REQUIRE(k >= 1 && k <= N2, TK3D_ERR_K, "feature_knn: need 1 <= k <= N2 (k=%lld, N2=%lld)", (long long)k,
               (long long)N2);
  TK3D_REQUIRE(k <= 128, TK3D_ERR_UNSUPPORTED, "feature_knn: k up to 128 (got %lld)", (long long)k);
  if (B * N1 == 0) return TK3D_OK;
  TK3D_REQUIRE(query && key && dist && index, TK3D_ERR_NULL, "feature_knn: a pointer is NULL");
  cudaStream_t st = (cudaStream_t)stream;
  const float *q = (const float *)query, *r = (const float *)key;
  const bool cf = channel_first != 0;
  const int *counts = nullptr;
  const size_t need = scratch ? ff_scratch_bytes(B, C, N1, N2, k) : 0;
  if (need != 0 && scratch_bytes >= need && (reinterpret_cast<uintptr_t>(scratch) & 15) == 0) {
    const int rc = ff_knn(q, r, B, (int)C, (int)N1, (int)N2, (int)k, cf, (float *)dist, index, scratch, &counts, st);
    if (rc) return rc;
  }
  float *d = (float *)dist;
  if (counts) {  // k <= 48
    if (k <= 32) return launch<1, true>(q, r, B, (int)C, (int)N1, (int)N2, (int)k, cf, d, index, counts, st);
    return launch<2, true>(q, r, B, (int)C, (int)N1, (int)N2, (int)k, cf, d, index, counts, st);
  }
  if (k <= 32) return launch<1, false>(q, r, B, (int)C, (int)N1, (int)N2, (int)k, cf, d, index, nullptr, st);
  if (k <= 64) return launch<2, false>(q, r, B, (int)C, (int)N1, (int)N2, (int)k, cf, d, index, nullptr, st);
  return launch<4, false>(q, r, B, (int)C, (int)N1, (int)N2, (int)k, cf, d, index, nullptr, st);
}

TK3D_BOUNDS_TU(feature_knn)
