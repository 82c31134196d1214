// Gradients of the row gathers (float32), any number of channels and entries.
//
//     rows[b, index[b,e], c] += gout[b, c, e]     then     gin[b, c, n] = rows[b, n, c]
//
// A kernel reads gout once, tile by tile, turns a tile of [channels][entries] into row pieces in shared memory and adds
// them to rows of [N][channels rounded up to 4] with 16-byte reductions at L2; the rows are then written back channel by
// channel (unrow_kernel, or the plain transposition).  B200, B = 32:
//   scatter_fold_kernel (group_points, set abstraction; 64 channels on): entries of a tile that follow one another with the
//     same index (the padding of a ball repeats its first hit: a third to three quarters of the entries) are summed in
//     registers and reduced once, and what a thread's addresses have in common is computed once.  64 x 8192 <- 1024 x 32
//     (a third padding) 71 -> 65 us, 128 x 512 <- 128 x 64 (two thirds) 49 -> 36.  What bounds it: instructions (0.56 of
//     the issue slots) and the loads' latency between them, not the reductions (the interpolation's gradient reduces 2.4
//     times as many bytes a second); walking over tiles with two buffers did not help (72 to 82 us).
//   scatter_edge_kernel (edge features, lists of up to 128): a tile holds whole queries, and the sums over each query's K
//     entries of both halves of gout come from the same pass.  64 x 1024 <- 1024 x 20: 45 and 76 for the sums apart -> 81 us
//     (335 MB at 4.1 TB/s).  Tiles hold as many queries as make a multiple of four entries, for 16-byte accesses: as many as
//     fit, element by element where that is no multiple, took twice the time (B = 8, K = 14 40 us / 21, 22 78 / 34, 34 133 / 57),
//     and for lists of odd length above 32 or of more than 128 longer than the sums apart (K = 65 348 / 128, 130 1264 / 193).
// Clouds a few at a time, for rows that stay in L2 (32, 16, 8 MB of rows a pass), were no faster: 103, 104, 119, 150 us.
#include "rows.cuh"
#include "scatter.cuh"

namespace tk3d {

namespace {

struct ScatterArgs {
  const float *gout;
  int64_t gstride, E;
  int C, ld;         // channels, floats of a row
  int N;
  float *rows;
  int32_t *status;
  // query sums
  int per;           // entries of a tile
  int M, K, include_query;
  float *gq;
};

// Float (c, e) of a tile: the 16-byte chunk of entries 4g .. 4g + 3 lies at chunk g ^ (c >> 2) of its eight.
__device__ __forceinline__ int sc_at(int c, int e, int TE) { return c * TE + (e ^ (((c >> 2) & 7) << 2)); }

constexpr int SC_NT = 128;

template <bool VEC, typename IndexT>
__global__ void __launch_bounds__(SC_NT, 12) scatter_fold_kernel(const ScatterArgs a, const IndexT *__restrict__ index) {
  constexpr int TE = ROWS_TE, NW = SC_NT / 32;
  extern __shared__ __align__(16) float tile[];  // [ld][TE]
  __shared__ int sid[TE];
  __shared__ uint16_t runs[2][TE];  // single entries and longer runs: first entry | length << 8
  __shared__ int nruns[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ql = lane & 7, el = lane >> 3;
  const int64_t b = blockIdx.y;
  const int64_t e0 = (int64_t)blockIdx.x * TE;
  const int n = (int)min((int64_t)TE, a.E - e0);
  const float *gb = a.gout + b * a.gstride + e0;
  // the index is requested ahead of gout and looked at behind it
  int64_t id = tid < n ? (int64_t)index[TK3D_AT(b * a.E + e0 + tid, gridDim.y * a.E)] : -1;
  if (VEC) {
    // a thread's chunk is the same in every row; rows are 16 apart: (c >> 2) & 7 flips its highest bit
    const int c0 = tid >> 3, e = (tid & 7) << 2;
    const float *src = gb + (int64_t)c0 * a.E + e;
    const int64_t step = 16 * a.E;
    float *dst = tile + c0 * TE;
    const int at = e ^ (((c0 >> 2) & 7) << 2);
    if (e < n) {
      int c = c0;
      for (; c + 48 < a.C; c += 64, src += 4 * step, dst += 64 * TE) {
        const float4 v0 = __ldcs(reinterpret_cast<const float4 *>(src));
        const float4 v1 = __ldcs(reinterpret_cast<const float4 *>(src + step));
        const float4 v2 = __ldcs(reinterpret_cast<const float4 *>(src + 2 * step));
        const float4 v3 = __ldcs(reinterpret_cast<const float4 *>(src + 3 * step));
        *reinterpret_cast<float4 *>(dst + at) = v0;
        *reinterpret_cast<float4 *>(dst + 16 * TE + (at ^ 16)) = v1;
        *reinterpret_cast<float4 *>(dst + 32 * TE + at) = v2;
        *reinterpret_cast<float4 *>(dst + 48 * TE + (at ^ 16)) = v3;
      }
      for (int flip = 0; c < a.C; c += 16, src += step, dst += 16 * TE, flip ^= 16)
        *reinterpret_cast<float4 *>(dst + (at ^ flip)) = __ldcs(reinterpret_cast<const float4 *>(src));
    }
  } else if (lane < n) {
#pragma unroll 8
    for (int c = warp; c < a.C; c += NW) tile[sc_at(c, lane, TE)] = __ldcs(gb + (int64_t)c * a.E + lane);
  }
  for (int i = a.C * TE + tid; i < a.ld * TE; i += SC_NT) tile[i] = 0.f;  // the row's padding channels
  if (warp == 0) {  // runs of one index; lane = entry
    const bool bad = id < 0 || id >= a.N;
    if (bad) id = -1;
    if (bad && lane < n && a.status) atomicOr(a.status, 1);
    sid[lane] = (int)id;
    const int prev = __shfl_up_sync(0xffffffffu, (int)id, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != (int)id);
    const unsigned above = lane == 31 ? 0u : heads >> (lane + 1);
    const int len = above ? __ffs(above) : 32 - lane;
    const bool live = ((heads >> lane) & 1u) && id >= 0;
    const unsigned singles = __ballot_sync(0xffffffffu, live && len == 1);
    const unsigned longer = __ballot_sync(0xffffffffu, live && len > 1);
    if (live) runs[len > 1][__popc((len > 1 ? longer : singles) & ((1u << lane) - 1))] = (uint16_t)(lane | len << 8);
    if (lane == 0) {
      nruns[0] = __popc(singles);
      nruns[1] = __popc(longer);
    }
  }
  __syncthreads();

  const int L = a.ld >> 2;
  float *rb = a.rows + b * (int64_t)a.N * a.ld;
  // single entries, four per warp and step: lane = 8 * el + ql takes the pieces ql, ql + 8, ... of entry el, whose
  // chunks lie in the same place of every row
  const float *mine = tile + 4 * ql * TE;
  for (int i = warp * 4 + el; i < nruns[0]; i += NW * 4) {
    const int s = runs[0][i] & 255;
    float *dst = rb + TK3D_AT(sid[s], a.N) * (int64_t)a.ld + 4 * ql;
    const float *src = mine + (s ^ (ql << 2));
#pragma unroll 2
    for (int q = ql; q < L; q += 8, src += 32 * TE, dst += 32) red_add4(dst, src[0], src[TE], src[2 * TE], src[3 * TE]);
  }
  // longer runs, one per warp: every fourth entry per el
  for (int i = warp; i < nruns[1]; i += NW) {
    const int s = runs[1][i] & 255, len = runs[1][i] >> 8;
    float *dst = rb + TK3D_AT(sid[s], a.N) * (int64_t)a.ld + 4 * ql;
    const float *src = mine;
    for (int q0 = 0; q0 < L; q0 += 8, src += 32 * TE, dst += 32) {
      float x = 0.f, y = 0.f, z = 0.f, w = 0.f;
      if (q0 + ql < L) {
        for (int j = s + el; j < s + len; j += 4) {
          const float *p = src + (j ^ (ql << 2));
          x += p[0];
          y += p[TE];
          z += p[2 * TE];
          w += p[3 * TE];
        }
      }
#pragma unroll
      for (int o = 8; o < 32; o <<= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
        z += __shfl_xor_sync(0xffffffffu, z, o);
        w += __shfl_xor_sync(0xffffffffu, w, o);
      }
      if (el == 0 && q0 + ql < L) red_add4(dst, x, y, z, w);
    }
  }
}

// With query sums.  A block has the entries of a few whole queries, at most 128, in a slab of 32 channels, and those of the
// second half of gout beside them, so that all its loads are under way at once (the second half read as the sums go: 122 us).
// A thread's chunk of four entries is the same in every row, and its rows are 8 apart, which flips bits 1 and 2 of
// (c >> 2) & 7: addresses are constants apart (108 -> 81 us).
constexpr int SE_NT = 256, SE_TE = 128, SE_C = 32;

template <typename IndexT>
__global__ void __launch_bounds__(SE_NT) scatter_edge_kernel(const ScatterArgs a, const IndexT *__restrict__ index) {
  extern __shared__ __align__(16) float tile[];  // [halves][SE_C][SE_TE], then int id[SE_TE]
  constexpr int NW = SE_NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ql = lane & 7, el = lane >> 3;
  const int halves = a.include_query ? 2 : 1;
  int *sid = reinterpret_cast<int *>(tile + halves * SE_C * SE_TE);
  const int64_t b = blockIdx.y;
  const int64_t e0 = (int64_t)blockIdx.x * a.per;
  const int n = (int)min((int64_t)a.per, a.E - e0);  // a multiple of 4
  const int c0 = blockIdx.z * SE_C, nc = min(SE_C, a.C - c0);  // channels of this block
  const float *gb = a.gout + b * a.gstride + (int64_t)c0 * a.E + e0;
  // requested ahead of gout
  const int64_t id0 = tid < n ? (int64_t)index[TK3D_AT(b * a.E + e0 + tid, gridDim.y * a.E)] : -1;
  {
    const int e = lane << 2;
    const float *src = gb + (int64_t)warp * a.E + e;
    const int at = warp * SE_TE + (e ^ ((warp >> 2) << 2));
    const int64_t step = 8 * a.E, other = (int64_t)a.C * a.E;
    float4 v[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (h < halves && e < n && warp + 8 * i < nc)
          v[h][i] = __ldcs(reinterpret_cast<const float4 *>(src + h * other + i * step));
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (h < halves && e < n && warp + 8 * i < nc)
          *reinterpret_cast<float4 *>(tile + ((at + (h * SE_C + 8 * i) * SE_TE) ^ (8 * i))) = v[h][i];
  }
  for (int i = nc * SE_TE + tid; i < ((nc + 3) & ~3) * SE_TE; i += SE_NT) tile[i] = 0.f;  // the row's padding channels
  if (tid < n) {
    const bool out = id0 < 0 || id0 >= a.N;
    sid[tid] = out ? -1 : (int)id0;
    if (out && a.status) atomicOr(a.status, 1);
  }
  __syncthreads();
  const int L = (nc + 3) >> 2;
  float *rb = a.rows + b * (int64_t)a.N * a.ld + c0 + 4 * ql;
  for (int s = warp * 4 + el; s < n; s += NW * 4) {
    const int id = sid[s];
    if (id < 0) continue;
    const float *src = tile + 4 * ql * SE_TE + (s ^ (ql << 2));
    if (ql < L) red_add4(rb + TK3D_AT(id, a.N) * (int64_t)a.ld, src[0], src[SE_TE], src[2 * SE_TE], src[3 * SE_TE]);
  }
  // gq[b,c,m] = sum_k (g[C+c] - g[c]), or minus the sum of the only half
  const int K = a.K, nq = n / K;
  const int64_t m0 = (int64_t)blockIdx.x * (a.per / K);
  const float *second = tile + SE_C * SE_TE;
  for (int u = tid; u < nc * nq; u += SE_NT) {
    const int c = u / nq, m = u - c * nq;
    float sum = 0.f;
    if ((K & 3) == 0) {
      for (int e = m * K; e < m * K + K; e += 4) {
        const float4 g0 = *reinterpret_cast<const float4 *>(tile + sc_at(c, e, SE_TE));
        float4 g1 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.include_query) g1 = *reinterpret_cast<const float4 *>(second + sc_at(c, e, SE_TE));
        sum += g1.x - g0.x;
        sum += g1.y - g0.y;
        sum += g1.z - g0.z;
        sum += g1.w - g0.w;
      }
    } else {
      for (int e = m * K; e < m * K + K; ++e) {
        const int at = sc_at(c, e, SE_TE);
        sum += a.include_query ? second[at] - tile[at] : -tile[at];
      }
    }
    const int64_t at = (b * a.C + c0 + c) * (int64_t)a.M + m0 + m;
    if (TK3D_IN(at, (int64_t)gridDim.y * a.C * a.M)) a.gq[at] = sum;
  }
}

// rows [B][N][ld] -> gin [B][C][N] for any C and N; a block moves 64 points x 64 channels.
__global__ void __launch_bounds__(256)
unrow_kernel(const float *__restrict__ rows, int ld, int C, int N, float *__restrict__ gin) {
  __shared__ __align__(16) float t[64 * 64];  // [channel][point], chunks of four points swizzled
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ql = lane & 7, el = lane >> 3;
  const int64_t b = blockIdx.z;
  const int n0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
  const float *src = rows + b * (int64_t)N * ld;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int g = warp + 8 * i, n = n0 + 4 * g + el;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int q = ql + 8 * j, c = c0 + 4 * q;
      if (n < N && c < ld) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(src + (int64_t)n * ld + c));
        float *p = t + (4 * q) * 64 + (((g ^ q) & 15) << 2) + el;
        p[0] = v.x;
        p[64] = v.y;
        p[128] = v.z;
        p[192] = v.w;
      }
    }
  }
  __syncthreads();
  float *dst = gin + (b * C + c0) * (int64_t)N + n0;
  const int nc = min(64, C - c0), nl = tid & 63;
  if (n0 + nl < N)
    for (int cl = tid >> 6; cl < nc; cl += 4)
      if (TK3D_IN(dst + (int64_t)cl * N + nl - gin, (int64_t)gridDim.z * C * N))
        dst[(int64_t)cl * N + nl] = t[cl * 64 + ((((nl >> 2) ^ (cl >> 2)) & 15) << 2) + (nl & 3)];
}

template <typename IndexT>
int scatter_go(ScatterArgs a, int64_t B, const IndexT *index, cudaStream_t st) {
  const bool aligned = a.E % 4 == 0 && a.gstride % 4 == 0 && (reinterpret_cast<uintptr_t>(a.gout) & 15) == 0;
  if (a.gq) {
    a.per = scatter_edge_entries(a.gout, a.E, a.gstride, a.K);
    const size_t smem = sizeof(float) * (size_t)(a.include_query ? 2 : 1) * SE_C * SE_TE + sizeof(int) * SE_TE;
    const int64_t tiles = (a.E + a.per - 1) / a.per;
    TK3D_REQUIRE(tiles < (1LL << 31), TK3D_ERR_SHAPE, "scatter: too many entries");
    const dim3 grid((unsigned)tiles, (unsigned)B, (unsigned)((a.C + SE_C - 1) / SE_C));
    scatter_edge_kernel<IndexT><<<grid, SE_NT, smem, st>>>(a, index);
    return check_launch("scatter_edge_kernel");
  }
  const size_t smem = sizeof(float) * (size_t)a.ld * ROWS_TE;
  const int64_t tiles = (a.E + ROWS_TE - 1) / ROWS_TE;
  TK3D_REQUIRE(tiles < (1LL << 31), TK3D_ERR_SHAPE, "scatter: too many entries");
  const dim3 grid((unsigned)tiles, (unsigned)B);
  // Folding pays from 64 channels on (8 x 24000 <- 4000 x 16 with 32 channels, a third padding, 23 us without and 29 with it) and
  // from 1e7 elements on, whatever the padding: without / with it, none, a third and two thirds padded, us: 1 x 256 x 128 <-
  // 512 7.4 / 8.3, 8.8, 8.4, 16 x 256 x 512 <- 2048 18 / 18.4, 19.9, 17.5, 64 x 64 x 2048 <- 8192 50 / 46, 48, 44, 16 x 512 x
  // 2048 <- 8192 171 / 139, 169, 155.
  if (aligned && a.C % 4 == 0 && (a.C < 64 || B * a.C * a.E < 10000000)) {
    if (smem > 48 * 1024) TK3D_CUDA(raise_smem_limit((const void *)scatter_rows_vec4_kernel<1, IndexT>, (int)smem));
    scatter_rows_vec4_kernel<1, IndexT><<<grid, ROWS_THREADS, smem, st>>>(a.gout, index, nullptr, a.C, a.N, a.E, a.gstride,
                                                                          a.rows, a.status);
    return check_launch("scatter_rows_vec4_kernel");
  }
  auto kern = aligned ? scatter_fold_kernel<true, IndexT> : scatter_fold_kernel<false, IndexT>;
  if (smem > 48 * 1024) TK3D_CUDA(raise_smem_limit((const void *)kern, (int)smem));
  kern<<<grid, SC_NT, smem, st>>>(a, index);
  return check_launch("scatter_fold_kernel");
}

}  // namespace

bool scatter_ok(int64_t B, int64_t C, int64_t N, int64_t M, int64_t K) {
  return B >= 1 && B <= 65535 && C >= 1 && C <= ROWS_MAX_C && N >= 1 && N < (1LL << 30) && M >= 1 && K >= 1 &&
         M * K < (1LL << 36);
}

int scatter_edge_entries(const void *gout, int64_t E, int64_t gstride, int64_t K) {
  if (K > SE_TE || E % 4 != 0 || gstride % 4 != 0 || (reinterpret_cast<uintptr_t>(gout) & 15) != 0) return 0;
  const int whole = K % 4 == 0 ? 1 : K % 2 == 0 ? 2 : 4;  // queries whose entries are a multiple of 4
  return (int)(SE_TE / (K * whole) * (K * whole));
}

int scatter_launch(const ScatterCall &c, cudaStream_t st) {
  ScatterArgs a;
  a.gout = c.gout;
  a.gstride = c.gstride;
  a.E = c.M * c.K;
  a.C = (int)c.C;
  a.ld = (int)((c.C + 3) & ~(int64_t)3);
  a.N = (int)c.N;
  a.rows = (float *)c.scratch;
  a.status = c.status;
  a.M = (int)c.M;
  a.K = (int)c.K;
  a.include_query = c.include_query;
  a.gq = c.gq;
  TK3D_CUDA(cudaMemsetAsync(c.scratch, 0, scatter_scratch_bytes(c.B, c.C, c.N), st));
  const int rc = c.index_i32 ? scatter_go<int32_t>(a, c.B, (const int32_t *)c.index, st)
                             : scatter_go<int64_t>(a, c.B, (const int64_t *)c.index, st);
  if (rc) return rc;
  if (c.C % 4 == 0 && c.N <= SCATTER_TRANSPOSED) return transpose_bcn(a.rows, c.gin, c.B, c.N, c.C, st);
  const dim3 grid((unsigned)((c.N + 63) / 64), (unsigned)((c.C + 63) / 64), (unsigned)c.B);
  unrow_kernel<<<grid, 256, 0, st>>>(a.rows, a.ld, a.C, a.N, c.gin);
  return check_launch("unrow_kernel");
}

}  // namespace tk3d

TK3D_BOUNDS_TU(scatter)
