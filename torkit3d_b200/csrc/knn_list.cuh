// Candidate lists of the two-pass neighbour searches (knn.cu over key tiles, spatial_knn.cu over
// ordered leaves): the predicated append, and the exact scan of a query whose list overflowed.
#pragma once

#include "tk3d_common.cuh"

namespace tk3d {

__device__ __forceinline__ float pinf() { return __int_as_float(0x7f800000); }

// Predicated append: if a < thr, claim a slot of the query's list and store v there (when the
// slot exists).  Written in PTX so that it stays five straight-line instructions.
template <int STRIDE_BYTES, int KT_QCAP>
__device__ __forceinline__ void kt_append(float a, float thr, unsigned cnt_addr, unsigned cand_addr, int v) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .pred q;\n\t"
      ".reg .s32 sl;\n\t"
      ".reg .u32 ad;\n\t"
      "setp.ltu.f32 p, %0, %1;\n\t"
      "@p atom.shared.add.s32 sl, [%2], 1;\n\t"
      "setp.lt.and.s32 q, sl, %5, p;\n\t"
      "mad.lo.u32 ad, sl, %6, %3;\n\t"
      "@q st.shared.s32 [ad], %4;\n\t"
      "}" ::"f"(a),
      "f"(thr), "r"(cnt_addr), "r"(cand_addr), "r"(v), "n"(KT_QCAP), "n"(STRIDE_BYTES));
}

// Exact scan of query `fq` by one warp: lanes take 32 consecutive keys at a time; a key that beats
// the current k-th entry is inserted into the sorted list kept in the first k slots of the query's
// column of the candidate lists (col_d / col_i, one slot every QS words; position by counting, entries
// behind it moved up by the lanes together).  Keys arrive in ascending index order, so a key equal to
// the k-th distance never enters a full list and equal distances stay in index order.  A NaN distance
// counts as +inf for the ordering.  The row goes to dist[orow..] / index[orow..].
template <int QS>
__device__ __forceinline__ void kt_exact_scan(const float *__restrict__ queries, const float *__restrict__ rb, int fq,
                                              int N2, int k, XyzLayout ql, XyzLayout kl, float *col_d, int *col_i,
                                              float *__restrict__ dist, const IndexOut &index, int64_t orow) {
  const int lane = threadIdx.x & 31;
  float fx, fy, fz;
  load_xyz(queries, fq, ql, fx, fy, fz);
  int nk = 0;
  float kth = pinf();
  for (int base = 0; base < N2; base += 32) {
    const int j = base + lane;
    float d = pinf();
    if (j < N2) {
      float rx, ry, rz;
      load_xyz(rb, j, kl, rx, ry, rz);
      d = sqdist<float>(rx, ry, rz, fx, fy, fz);
    }
    const float dv = d == d ? d : pinf();  // ordering value
    unsigned mask = __ballot_sync(0xffffffffu, j < N2 && (nk < k || dv < kth));
    while (mask) {
      const int l = __ffs(mask) - 1;
      mask &= mask - 1;
      const float dn = __shfl_sync(0xffffffffu, d, l), dnv = __shfl_sync(0xffffffffu, dv, l);
      if (nk == k && !(dnv < kth)) continue;  // the k-th entry tightened since the ballot
      // position: entries ordering at or before the new key (equal distances hold lower indices)
      int before = 0;
      for (int r = lane; r < nk; r += 32) {
        const float w = col_d[r * QS];
        before += ((w == w ? w : pinf()) <= dnv) ? 1 : 0;
      }
      const int pos = __reduce_add_sync(0xffffffffu, before);
      const int last = nk < k ? nk : k - 1;  // slot that receives the old entry last - 1
      // move entries [pos, last) up by one: read them all, then write them all
      float mv[4];
      int mj[4];
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        const int r = lane + 32 * q4;
        if (r >= pos && r < last) {
          mv[q4] = col_d[r * QS];
          mj[q4] = col_i[r * QS];
        }
      }
      __syncwarp();
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        const int r = lane + 32 * q4;
        if (r >= pos && r < last) {
          col_d[(r + 1) * QS] = mv[q4];
          col_i[(r + 1) * QS] = mj[q4];
        }
      }
      if (lane == 0) {
        col_d[pos * QS] = dn;
        col_i[pos * QS] = base + l;
      }
      __syncwarp();
      if (nk < k) ++nk;
      if (nk == k) {
        const float w = col_d[(k - 1) * QS];
        kth = w == w ? w : pinf();
      }
    }
  }
  float *od = dist + orow;
  for (int c = lane; c < k; c += 32) {
    od[c] = col_d[c * QS];
    index.put(orow + c, col_i[c * QS]);
  }
}

}  // namespace tk3d
