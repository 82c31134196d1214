// Ball query of 32 queries by a block of SPLIT warps, keys swept in index order.
//
// Lane = query, and warp s sweeps the s-th slice of every 256-key tile, so SPLIT times as many warps
// are in flight as with one thread per query.  A thread records the hits of its slice as a bit mask
// (at most 64 keys), the slices' hit counts of the tile are exchanged through shared memory at the
// tile's barrier, and every thread then knows where its hits belong in the query's row (hits of earlier
// tiles + hits of lower slices of this tile) and writes them there: rows come out in ascending key order
// without a merge, for any K.  A query with K hits stops testing, and the block leaves the key loop at
// the first barrier after all its queries are full.
#pragma once

#include "sweep.cuh"

namespace tk3d {

constexpr int BS_TILE = 256;

template <int SPLIT>
struct BallSweepSmem {
  float4 tile[2][BS_TILE];
  int tcount[2][SPLIT][32];
};

// Called by the whole block; lane = query, its row of the output starts at `row`.
template <int SPLIT>
__device__ __forceinline__ void ball_sweep(const float *__restrict__ rb, int N2, XyzLayout kl, float qx, float qy,
                                           float qz, bool valid, float r2, int k, int64_t row, const IndexOut &index,
                                           BallSweepSmem<SPLIT> &sm) {
  constexpr int THREADS = 32 * SPLIT;
  constexpr int PER = BS_TILE / THREADS;
  constexpr int QK = BS_TILE / SPLIT;  // keys per warp per tile (64 or 32)
  static_assert(PER >= 1 && QK <= 64 && QK % 8 == 0, "slice must fit a 64-bit hit mask");
  auto &tile = sm.tile;
  auto &tcount = sm.tcount;
  const int tid = threadIdx.x, lane = tid & 31, part = tid >> 5;
  const float never = __int_as_float(0xff800000);
  const float2 mx[1] = {make_float2(-2.f * qx, -2.f * qx)}, my[1] = {make_float2(-2.f * qy, -2.f * qy)},
               mz[1] = {make_float2(-2.f * qz, -2.f * qz)};
  const float open_thr = sweep_threshold(r2, sweep_qq(qx, qy, qz));
  float thr[1] = {valid ? open_thr : never};
  int done = 0;  // hits of this query in the tiles swept so far (the same number in every warp)
  const int ntiles = (N2 + BS_TILE - 1) / BS_TILE;

  float4 nxt[PER];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int j = t0 + tid + p * THREADS;
      float4 v = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7f800000));
      if (j < N2) {
        float x, y, z;
        load_xyz(rb, j, kl, x, y, z);
        v = make_float4(x, y, z, sweep_key_w(x, y, z));
      }
      nxt[p] = v;
    }
  };
  auto commit = [&](float4 *dst) {
#pragma unroll
    for (int p = 0; p < PER; ++p) sweep_store_key(dst, tid + p * THREADS, nxt[p].x, nxt[p].y, nxt[p].z, nxt[p].w);
  };
  fetch(0);
  commit(tile[0]);
  __syncthreads();
  for (int t = 0; t < ntiles; ++t) {
    const int t0 = t * BS_TILE + part * QK;
    const float4 *tl = tile[t & 1] + part * QK;
    if (t + 1 < ntiles) fetch((t + 1) * BS_TILE);
    unsigned long long mask = 0;
    int cnt = 0;
    const bool was_full = !valid || done >= k;
#pragma unroll 2
    for (int u0 = 0; u0 < QK; u0 += 8) {
      float2 a[4];
      if (__builtin_expect(sweep_group2<1, true>(tl + u0, mx, my, mz, thr, a), 0)) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float av = (u & 1) ? a[u >> 1].y : a[u >> 1].x;
          if (!(av >= thr[0])) {  // padding keys carry +inf; a full row has thr = -inf
            const float4 r = sweep_load_key(tl, u0 + u);
            const float d = sqdist<float>(r.x, r.y, r.z, qx, qy, qz);
            if (d < r2) {
              mask |= 1ull << (u0 + u);
              if (done + ++cnt >= k) thr[0] = never;  // whatever the lower slices found, this row is full
            }
          }
        }
      }
    }
    tcount[t & 1][part][lane] = cnt;
    if (t + 1 < ntiles) commit(tile[(t + 1) & 1]);
    // One barrier per tile; it also votes on "every query of this block was full before this tile"
    // (such a tile recorded no hit anywhere, so nothing is left to write).
    if (__syncthreads_and(was_full)) break;
    int before = 0, total = 0;
#pragma unroll
    for (int s = 0; s < SPLIT; ++s) {
      const int c = tcount[t & 1][s][lane];
      if (s < part) before += c;
      total += c;
    }
    int pos = done + before;
    while (mask != 0 && pos < k) {
      const int bit = __ffsll((long long)mask) - 1;
      mask &= mask - 1;
      index.put(row + pos, t0 + bit);
      ++pos;
    }
    done += total;
    if (done >= k) thr[0] = never;
  }
  __syncthreads();  // the row's first entry, written by whichever warp found it, is visible now
  if (valid && done < k) {
    const int64_t first = done > 0 ? index.get(row) : -1;
    for (int c = done + part; c < k; c += SPLIT) index.put(row + c, first);
  }
}

}  // namespace tk3d
