// Gathers by channel rows: group_points (float32 and float64) and the set-abstraction front end (float32), clouds whose
// rows fit shared memory twice.  No transposed copy of the features, no scratch.
//
// A block owns a chunk of the E = N2*K index entries of one cloud -- each thread keeps its entries' indices in registers
// for the whole block -- and walks a group of channels.  The N1 features of a channel are one contiguous row of the
// [B,C,N1] tensor: rows are brought into shared memory with cp.async, RB at a time (short rows: one barrier then holds
// for several of them) and double buffered, so that the next ones land while the current ones are gathered; the gather
// itself is a shared-memory read per output element followed by streaming stores.  HBM sees every feature and every
// index once (the row re-reads of neighbouring blocks hit L2) and the output once: 32 x 64 x 8192 -> 1024 x 32 entries
// in 64 us, 5.4 TB/s.  (The mirror image for the backward, rows accumulated with shared-memory float atomics, was 0.18 ms
// against 0.12: a shared-memory float reduction per element is slow.)
// Rows start anywhere: a row is copied to the same offset of a 16-byte line as it has in memory, its ends in single
// elements.  Outputs of four consecutive entries per thread leave as 16-byte stores where E and the addresses allow,
// else lanes hold consecutive entries.  An index outside [0,N1) reads the zero kept behind the row.
#pragma once

#include "tk3d_common.cuh"

namespace tk3d {

template <int BYTES>
__device__ __forceinline__ void cr_cp_async(void *smem, const void *gmem) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem),
                 "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void cr_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cr_cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// The three channels behind the features of a set abstraction: coordinates of the neighbours minus those of the centre.
struct CrXyz {
  const float *points, *cent;  // coordinate d of point j: j * pps + d * pcs
  int pps, pcs, cps, cpc, K, M;
};

// Distance of two rows in shared memory: up to 15 bytes of offset, the row, a zero; whole 16-byte lines.
template <typename T>
__host__ __device__ inline int cr_stride(int N1) {
  constexpr int P = 16 / (int)sizeof(T);
  return (N1 + P + P - 1) / P * P;
}

// R rounds of four entries per thread: a block covers CR_THREADS * 4 * R entries.
template <typename T, typename IndexT, int CR_THREADS, int R, bool VEC, bool XYZ>
__global__ void __launch_bounds__(CR_THREADS)
group_fwd_chanrow_kernel(const T *__restrict__ in, const IndexT *__restrict__ index, int C, int N1, int64_t E, int cg,
                         int RB, T *__restrict__ out, int64_t ostride, int32_t *__restrict__ status, CrXyz xyz) {
  extern __shared__ __align__(16) unsigned char cr_raw[];
  T *cr_rows = reinterpret_cast<T *>(cr_raw);  // [2][RB][stride]
  constexpr int PER16 = 16 / (int)sizeof(T);   // elements per 16-byte copy
  const int tid = threadIdx.x;
  const int64_t b = blockIdx.z;
  const int ctot = XYZ ? C + 3 : C;
  const int c0 = blockIdx.y * cg, c1 = min(ctot, c0 + cg);
  const int64_t e0 = (int64_t)blockIdx.x * (CR_THREADS * 4 * R);
  const int stride = cr_stride<T>(N1);
  const int left = (int)min((int64_t)(CR_THREADS * 4 * R), E - e0);  // entries of this block
  // entry v of round r, within the block
  auto entry = [&](int r, int v) { return VEC ? (r * CR_THREADS + tid) * 4 + v : (r * 4 + v) * CR_THREADS + tid; };

  int id[R][4];
  bool bad = false;
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int e = entry(r, v);
      int64_t j = e < left ? (int64_t)index[TK3D_AT(b * E + e0 + e, gridDim.z * E)] : 0;
      if (j < 0 || j >= N1) {
        j = N1;  // the zero behind the row
        bad = true;
      }
      id[r][v] = (int)j;
    }
  }
  if (bad && status) atomicOr(status, 1);

  // rows of whole 16-byte lines: no ends to copy, and the zeros behind them stay
  bool lines = N1 % PER16 == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
  if constexpr (XYZ) lines = lines && xyz.pps == 1 && (reinterpret_cast<uintptr_t>(xyz.points) & 15) == 0;
  if (lines && tid < 2 * RB) cr_rows[tid * stride + N1] = (T)0;
  // first element of row c and its offset within a 16-byte line
  auto source = [&](int c) -> const T * {
    if constexpr (XYZ) {
      if (c >= C) return xyz.points + b * 3 * (int64_t)N1 + (int64_t)(c - C) * xyz.pcs;
    }
    return in + (b * C + c) * (int64_t)N1;
  };
  auto offset = [&](const T *g) { return (int)((reinterpret_cast<uintptr_t>(g) & 15) / sizeof(T)); };
  auto stage = [&](int c, int buf) {
    for (int k = 0; k < RB && c + k < c1; ++k) {
      const T *g = source(c + k);
      T *d = cr_rows + (buf * RB + k) * stride;
      if (lines) {
        for (int q = tid; q < N1 / PER16; q += CR_THREADS) cr_cp_async<16>(d + PER16 * q, g + PER16 * q);
        continue;
      }
      if constexpr (XYZ) {
        if (c + k >= C && xyz.pps != 1) {
          for (int q = tid; q < N1; q += CR_THREADS) cr_cp_async<sizeof(T)>(d + q, g + (int64_t)q * xyz.pps);
          if (tid == 0) d[N1] = (T)0;
          continue;
        }
      }
      const int o = offset(g), head = min(N1, (PER16 - o) & (PER16 - 1)), body = (N1 - head) / PER16;
      d += o;
      for (int q = tid; q < body; q += CR_THREADS) cr_cp_async<16>(d + head + PER16 * q, g + head + PER16 * q);
      const int done = head + PER16 * body;
      if (tid < head) cr_cp_async<sizeof(T)>(d + tid, g + tid);
      if (tid < N1 - done) cr_cp_async<sizeof(T)>(d + done + tid, g + done + tid);
      if (tid == 0) d[N1] = (T)0;
    }
    cr_cp_commit();
  };
  stage(c0, 0);
  int buf = 0;
  for (int cb = c0; cb < c1; cb += RB, buf ^= 1) {
    if (cb + RB < c1) {
      stage(cb + RB, buf ^ 1);  // the other buffer was released by the barrier that ended the last round
      cr_cp_wait<1>();
    } else {
      cr_cp_wait<0>();
    }
    __syncthreads();
    for (int c = cb; c < min(c1, cb + RB); ++c) {
      const T *row = cr_rows + (buf * RB + c - cb) * stride;
      const bool coord = XYZ && c >= C;
      if (!lines && !(coord && xyz.pps != 1)) row += offset(source(c));
      T *o = out + b * ostride + (int64_t)c * E + e0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (entry(r, 0) >= left) break;
        T v[4] = {row[TK3D_AT(id[r][0], N1 + 1)], row[TK3D_AT(id[r][1], N1 + 1)], row[TK3D_AT(id[r][2], N1 + 1)],
                  row[TK3D_AT(id[r][3], N1 + 1)]};
        if constexpr (XYZ) {
          if (coord) {
            const float *q = xyz.cent + b * 3 * (int64_t)xyz.M + (int64_t)(c - C) * xyz.cpc;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int e = entry(r, k);
              if (e < left) v[k] = __fsub_rn(v[k], __ldg(q + ((unsigned)(e0 + e) / (unsigned)xyz.K) * (int64_t)xyz.cps));
            }
          }
        }
        if constexpr (VEC) {
          const int e = entry(r, 0);
          if (!TK3D_IN(o + e + 3 - out, (int64_t)gridDim.z * ostride)) continue;
          if constexpr (sizeof(T) == 4) {
            __stcs(reinterpret_cast<float4 *>(o + e), make_float4(v[0], v[1], v[2], v[3]));
          } else {
            __stcs(reinterpret_cast<double2 *>(o + e), make_double2(v[0], v[1]));
            __stcs(reinterpret_cast<double2 *>(o + e) + 1, make_double2(v[2], v[3]));
          }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int e = entry(r, k);
            if (e < left && TK3D_IN(o + e - out, (int64_t)gridDim.z * ostride)) __stcs(o + e, v[k]);
          }
        }
      }
    }
    __syncthreads();
  }
}

// Largest cloud: two rows must fit the 227 KB of an SM (24576 floats or 12288 doubles).
constexpr int64_t CR_MAX_ROW_BYTES = 24576 * 4;

inline bool chanrow_ok(int64_t B, int64_t C, int64_t N1, int64_t E, int64_t elem = 4) {
  return N1 >= 256 && N1 * elem <= CR_MAX_ROW_BYTES && E >= 1024 && B <= 65535 && C <= 65532;
}

// Rows that are not whole 16-byte lines, copied in pieces: worth it from 2e6 elements of output and a quarter as many entries as
// points on; below, the direct gather (us, direct / channel rows: 1 x 64 x 1185 -> 18960 4.5 / 5.2, 14 x 12 x 1185 -> 4740 4.1 /
// 5.3, 64 x 12 x 20411 -> 3060 11 / 15; 1 x 64 x 8191 -> 32764 9.1 / 6.6, 64 x 12 x 8191 -> 3276 12.8 / 8.3).
inline bool chanrow_pieces_pay(int64_t B, int64_t C, int64_t N1, int64_t E) {
  return B * C * E >= 2000000 && 4 * E >= N1;
}

// out [B] slabs of ostride elements; XYZ (float32): three more channels behind the C of `in`.
template <bool XYZ, typename T, typename IndexT>
int group_fwd_chanrow(const T *in, const IndexT *index, int64_t B, int64_t C, int64_t N1, int64_t E, T *out,
                      int64_t ostride, int32_t *status, const CrXyz &xyz, cudaStream_t st) {
  const int64_t sms = sm_count(), ctot = C + (XYZ ? 3 : 0);
  // Entries per block: every block of a cloud copies the rows of its channels, so that large calls want many entries, small
  // ones many blocks; rows of 14000 points leave room for one block per SM, which wants more threads.  4096 / 8192 / 16384
  // entries, us: 1 x 131 x 24000 -> 24000 13.6 / 12.0 / 12.4, 4 x 64 x 24000 -> 96000 75 / 46 / 40, 32 x 64 x 12000 -> 12000
  // 46 / 47 / 42, 43 x 12 x 12000 -> 48000 42 / 34 / 39, 8 x 64 x 12000 -> 48000 43 / 35 / 36, 11 x 64 x 8192 -> 32768 35 / 29 /
  // 34, 1 x 131 x 4096 -> 65536 10.6 / 13.7 / 16.5, 1 x 12 x 12000 -> 48000 3.7 / 4.8 / 7.2, 64 x 64 x 300 -> 4800 25 / 20 / 27.
  const int64_t work = B * C * E;
  const bool long_rows = N1 >= 14000 ? work >= 3500000 : N1 >= 9000 && C >= 48 && work >= 10000000;
  const bool many = B * ((E + 8191) / 8192) * 4 >= 3 * sms || (N1 >= 4096 && work >= 10000000);
  const int pick = E > 8192 && long_rows ? 3 : E > 4096 && many ? 2 : 1;
  const int64_t ech = pick == 3 ? 16384 : pick == 2 ? 8192 : 4096;
  const int64_t chunks = (E + ech - 1) / ech;
  // channel groups: enough blocks for about three per SM, as few groups as possible beyond that
  int64_t groups = (3 * sms + B * chunks - 1) / (B * chunks);
  groups = groups < 1 ? 1 : (groups > ctot ? ctot : groups);
  const int cg = (int)((ctot + groups - 1) / groups);
  groups = (ctot + cg - 1) / cg;
  TK3D_REQUIRE(chunks < (1LL << 31), TK3D_ERR_SHAPE, "group_points: too many entries");
  // short rows share a barrier: up to 16 KB of them
  const int64_t rowb = (int64_t)cr_stride<T>((int)N1) * (int64_t)sizeof(T);
  int64_t rb = 16384 / rowb;
  rb = rb < 1 ? 1 : rb > 8 ? 8 : rb;
  rb = rb > cg ? cg : rb;
  const size_t smem = (size_t)(2 * rb * rowb);
  dim3 grid((unsigned)chunks, (unsigned)groups, (unsigned)B);
  const bool vec = E % 4 == 0 && (ostride * sizeof(T)) % 16 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#define TK3D_CR_LAUNCH(NT, RR, VV)                                                                                    \
  {                                                                                                                   \
    if (smem > 48 * 1024)                                                                                             \
      TK3D_CUDA(raise_smem_limit((const void *)group_fwd_chanrow_kernel<T, IndexT, NT, RR, VV, XYZ>, (int)smem));     \
    group_fwd_chanrow_kernel<T, IndexT, NT, RR, VV, XYZ><<<grid, NT, smem, st>>>(                                     \
        in, index, (int)C, (int)N1, E, cg, (int)rb, out, ostride, status, xyz);                                       \
  }
  if (pick == 3) {
    if (vec) TK3D_CR_LAUNCH(512, 8, true) else TK3D_CR_LAUNCH(512, 8, false)
  } else if (pick == 2) {
    if (vec) TK3D_CR_LAUNCH(256, 8, true) else TK3D_CR_LAUNCH(256, 8, false)
  } else {
    if (vec) TK3D_CR_LAUNCH(256, 4, true) else TK3D_CR_LAUNCH(256, 4, false)
  }
#undef TK3D_CR_LAUNCH
  return check_launch("group_fwd_chanrow_kernel");
}

}  // namespace tk3d
