// k nearest neighbours in a C-dimensional feature space by tensor cores: which keys can be among a query's k nearest is
// decided from a matrix product, and only those pairs (25 for k = 20) get the exact distance of feature_knn.cu.
//
// 1. ff_prep_kernel: every feature, less a common centre (what all have in common would only cost digits: the middle two of
//    four keys, channel by channel), as a sum of two bf16 (its upper and lower half, 2^-17 of it is lost), in the order that
//    tcgen05.mma reads (tiles of 128 points: half, eight channels, point), two bounds of the squared norm, and rows of float32.
// 2. ff_filter_kernel: a block holds 128 queries, the lanes of tensor memory.  Tiles of 128 keys arrive by bulk
//    copies; a . b = ah . bh + ah . bl + al . bh is accumulated in tensor memory, two tiles in flight, while the threads
//    read the tile before: v = |key|^2 - 2 query . key, the distance less the query's own norm.
//    First over all keys: the minima of v's upper bound over 64 classes of keys; their k-th smallest (a sorting network in
//    registers) plus the query's part of the error bounds the k-th neighbour's v.  Then over all keys again: those whose lower
//    bound is below go to the query's list.
// 3. ff_exact_kernel: a warp per query, lane = candidate; exact distances, the nearest kept sorted by (distance, index).
// 4. feature_knn_kernel redoes the groups of 32 queries that have one without a list.
//
// Error of v: let X = |query| + |key|, both less the centre, and count in u = 2^-24 X^2; 2 |a||b| <= X^2 / 2.
//   halves: bf16 has eight digits, so that the upper half is off by 2^-8 of a number at most and both halves by 2^-17; left out
//     are al . bl and what both halves miss, (2^-16 + 2 * 2^-17) of |a||b|, in v twice that: 256 u;
//   product: 3 (C + C / 16) numbers are added, taken to be rounded or truncated at 2^-23 of the sum of magnitudes each;
//   rounding of the norm and of the exact distance, C + 2 u each, of the centred features 2 u, of v, its bounds and the limit 4.
// Together 256 + 5 C + 3 C / 16 + 13 u at most; e = c X^2, c = C * 2^-21 + 1.25 * 2^-16, is 320 + 8 C u (and 2^-110 for what
// underflows).  How the tensor cores round inside a step is written nowhere: what stands behind the product's part are the
// errors measured against 64 bits, at most 0.70, 0.62, 0.41, 0.20 and 0.07 e for 1, 3, 16, 64 and 128 channels (normal,
// rectified, far from the origin, of one sign, channels and points of different size, far points).
// X^2 <= 2 |query|^2 + 2 |key|^2, so that a key's part, 2 c |key|^2, is put into its norm's two bounds: a key far from the
// others widens the bounds of no other (with the largest norm in its place, one key at 100 times the others' distance left
// nothing to filter).  A key with d <= the k-th d has its lower v <= (k-th smallest class minimum) + 4 c |query|^2.
//
// What the filter cannot tell apart it leaves to the kernel for all pairs, and is quick to find out: keys whose norms are not
// finite or vanish (no product is made), queries with a key in reach in 57 or more classes (some 140 keys, more than the
// lists take; with 53 a lattice of ties took 139 instead of 87 us), groups with such a query.  All pairs / the filter in vain,
// us, 32 x 1024 x 1024, 64 channels, k = 20: equal points 185 / 202, not a number 230 / 246, eight tight clusters 230 / 262;
// 16 x 2000 x 2000, 16 channels, k = 16, clusters about as large as the lists 257 / 319.
//
// 32 x 1024 x 1024, 64 channels, k = 20: 229 us by all pairs, 89 now: preparing 7, filter 37, exact distances 41, looking
// for what is left 3; 32 x 2000, 16 channels 388 / 138; 4 x 4096, 64 channels 458 / 117; 32 x 1024, 128 channels, k = 32
// 384 / 220.  The tensor pipe is active for 37 % of the filter; the rest is reading tensor memory (two loads of 32 columns a
// thread and tile), the minima and the comparisons.  With one thread per query it took 61 to 77 us.  The exact distances
// wait for shared memory.
#include "feature_filter.cuh"

namespace tk3d {
namespace {

constexpr int FF_T = 128;        // points of a tile
constexpr int FF_CLASSES = 64;
constexpr int FF_CAP = 64;       // candidates per query
constexpr int FF_MAX_C = 128;
constexpr int FF_MAX_K = 48;     // the 48th of 64 class minima lies near the 89th key
constexpr int FF_CROWD = 57;     // classes with a key in reach of a query that is given up
constexpr float FF_HUGE = 1e37f; // squared norms: no distance below overflows
constexpr int FF_PREP = 32;      // points of a preparing block
constexpr unsigned FULL = 0xffffffffu;
using u64 = unsigned long long;

// One side (queries or keys) in scratch.
struct FfSide {
  unsigned char *tiles;  // [B][tiles][tile_bytes]: halves [2][Cp / 8][128][8] bf16, norms' upper and lower bounds [2][128]
  float *rows;           // [B][N][Cr]
  float *block_max;      // [B][ceil(N / 32)] largest squared norm
};

__host__ __device__ inline int ff_cp(int C) { return (C + 15) / 16 * 16; }
__host__ __device__ inline int ff_cr(int C) { return (C + 3) / 4 * 4; }
__host__ __device__ inline int ff_tile_bytes(int C) { return 2 * ff_cp(C) * FF_T * 2 + 2 * FF_T * 4; }
__host__ __device__ inline int ff_upper(int C) { return ff_tile_bytes(C) - 2 * FF_T * 4; }  // where the bounds lie
__host__ __device__ inline int ff_lower(int C) { return ff_tile_bytes(C) - FF_T * 4; }
__device__ __forceinline__ float ff_error(int C) { return (float)C * 4.76837158e-7f + 1.90734863e-5f; }  // c
__host__ __device__ inline int ff_tiles(int N) { return (N + FF_T - 1) / FF_T; }

// Where a point lies in its tile: tiles are turned against each other, so that points whose indices differ by a multiple of
// 32 -- neighbours in clouds stored row by row -- are spread over the classes.
__device__ __forceinline__ int ff_place(int n) { return (n + 37 * (n / FF_T)) & (FF_T - 1); }
__device__ __forceinline__ int ff_point(int tile, int at) { return tile * FF_T + ((at - 37 * tile) & (FF_T - 1)); }

__device__ __forceinline__ unsigned ff_bf16(float x) {  // nearest bf16, as the upper half of a float
  unsigned r;
  asm("{.reg .b16 h; cvt.rn.bf16.f32 h, %1; mov.b32 %0, {0, h};}" : "=r"(r) : "f"(x));
  return r;
}

// Warp w of a block takes the channel groups w, w + 8, ...; lane = point.
template <bool CF>
__global__ void __launch_bounds__(256)
ff_prep_kernel(const float *__restrict__ in, const float *__restrict__ key, int C, int N, int N2, FfSide s) {
  __shared__ float part[8][FF_PREP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t b = blockIdx.y;
  const int n = blockIdx.x * FF_PREP + lane;  // up to whole tiles
  const int Cp = ff_cp(C), Cr = ff_cr(C), bytes = ff_tile_bytes(C), tiles = ff_tiles(N);
  const bool there = n < N;
  unsigned char *tile = s.tiles + (b * tiles + n / FF_T) * (int64_t)bytes;
  float sum = 0.f;
  for (int g = warp; g < Cp / 8; g += 8) {
    float x[8], mid;  // mid: lane i has the centre's channel 8 g + i % 8
    {
      const int c = 8 * g + (lane & 7);
      const int64_t j = (int64_t)(2 * (lane >> 3) + 1) * N2 / 8;
      mid = 0.f;
      if (c < C) mid = CF ? key[(b * C + c) * (int64_t)N2 + j] : key[(b * N2 + j) * (int64_t)C + c];
      const float other = __shfl_xor_sync(FULL, mid, 8), lo = fminf(mid, other), hi = fmaxf(mid, other);
      mid = 0.5f * (fmaxf(lo, __shfl_xor_sync(FULL, lo, 16)) + fminf(hi, __shfl_xor_sync(FULL, hi, 16)));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = 8 * g + i;
      x[i] = 0.f;
      if (there && c < C) x[i] = CF ? in[(b * C + c) * (int64_t)N + n] : in[(b * N + n) * (int64_t)C + c];
    }
    if (there) {
      float *row = s.rows + (b * N + n) * (int64_t)Cr + 8 * g;
      if (8 * g < Cr) *reinterpret_cast<float4 *>(row) = make_float4(x[0], x[1], x[2], x[3]);
      if (8 * g + 4 < Cr) *reinterpret_cast<float4 *>(row + 4) = make_float4(x[4], x[5], x[6], x[7]);
    }
    unsigned hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float c = __shfl_sync(FULL, mid, i);
      x[i] = there ? x[i] - c : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const unsigned h0 = ff_bf16(x[i]), h1 = ff_bf16(x[i + 1]);
      const unsigned l0 = ff_bf16(x[i] - __uint_as_float(h0)), l1 = ff_bf16(x[i + 1] - __uint_as_float(h1));
      hi[i / 2] = (h0 >> 16) | h1;
      lo[i / 2] = (l0 >> 16) | l1;
      sum = fmaf(x[i], x[i], sum);
      sum = fmaf(x[i + 1], x[i + 1], sum);
    }
    uint4 *dst = reinterpret_cast<uint4 *>(tile) + g * FF_T + ff_place(n);
    dst[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    dst[Cp / 8 * FF_T] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  part[warp][lane] = sum;
  __syncthreads();
  if (warp == 0) {
    sum = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) sum += part[w][lane];
    const float inf = __int_as_float(0x7f800000), e = 2.f * ff_error(C);  // no padding point is ever near
    reinterpret_cast<float *>(tile + ff_upper(C))[ff_place(n)] = there ? fmaf(sum, e, sum) : inf;
    reinterpret_cast<float *>(tile + ff_lower(C))[ff_place(n)] = there ? fmaf(sum, -e, sum) : inf;
    unsigned top = there ? __float_as_uint(sum) & 0x7fffffffu : 0u;  // NaN above infinity above every number
    top = __reduce_max_sync(FULL, top);
    if (lane == 0 && blockIdx.x * FF_PREP < N)
      s.block_max[b * ((N + FF_PREP - 1) / FF_PREP) + blockIdx.x] = __uint_as_float(top);
  }
}

__device__ __forceinline__ unsigned ff_smem(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ff_bar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// Waits for the phase's end, a second at most.
__device__ __forceinline__ bool ff_wait(unsigned bar, unsigned parity) {
  unsigned long long t0 = 0;
  for (int i = 0;; ++i) {
    unsigned done;
    asm volatile(
        "{.reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 63) == 63) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      else if (t - t0 > 1000000000ull) return false;
    }
    if (i >= (1 << 24)) return false;
  }
}
__device__ __forceinline__ void ff_copy(unsigned dst, const void *src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void ff_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// K-major operand without swizzle: eight rows of 16 bytes are contiguous, the next eight rows follow, the next eight
// channels lie 128 rows further on.
__device__ __forceinline__ u64 ff_desc(unsigned addr) {
  return (u64)((addr & 0x3ffffu) >> 4) | (u64)((FF_T * 16) >> 4) << 16 | (u64)(128 >> 4) << 32 | 1ull << 46;
}
__device__ __forceinline__ void ff_mma(unsigned d, u64 a, u64 b, unsigned accumulate) {
  constexpr unsigned idesc = 1u << 4 | 1u << 7 | 1u << 10 | (FF_T >> 3) << 17 | (FF_T >> 4) << 24;  // f32 += bf16 x bf16
  asm volatile(
      "{.reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;}" ::"r"(d), "l"(a),
      "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void ff_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Instructions marked aligned want the whole warp; lanes that took a branch or polled a barrier meet at __syncwarp().
// Requests 32 columns of the warp's lanes; ff_loaded() before they are used.
__device__ __forceinline__ void ff_load32(unsigned taddr, unsigned (&r)[32]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
        "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
        "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
// The registers go through the wait, so that no use of them is moved ahead of it.
__device__ __forceinline__ void ff_loaded(unsigned (&r)[32]) {
  __syncwarp();
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]));
}

// Batcher's odd-even merge sort; steps as template arguments, so that every index is a register.
template <int P, int K>
__device__ __forceinline__ void ff_sort_step(float (&m)[FF_CLASSES]) {
#pragma unroll
  for (int i = 0; i + K < FF_CLASSES; ++i)
    if (i >= K % P && (i - K % P) % (2 * K) < K && i / (2 * P) == (i + K) / (2 * P)) {
      const float lo = fminf(m[i], m[i + K]), hi = fmaxf(m[i], m[i + K]);
      m[i] = lo;
      m[i + K] = hi;
    }
  if constexpr (K > 1) ff_sort_step<P, K / 2>(m);
}
template <int P>
__device__ __forceinline__ void ff_sort(float (&m)[FF_CLASSES]) {
  ff_sort_step<P, P>(m);
  if constexpr (2 * P < FF_CLASSES) ff_sort<2 * P>(m);
}

// Two threads per query, one for each half of a tile's columns, with 32 classes and a list of its own:
// found[b][N1][2] candidates in lists[b][N1][2][FF_CAP], FF_BAD where the query needs the other kernel.
constexpr int FF_THREADS = 2 * FF_T;
constexpr int FF_BAD = 1 << 20;

__global__ void __launch_bounds__(FF_THREADS, 2)
ff_filter_kernel(FfSide qs, FfSide ks, int C, int N1, int N2, int k, unsigned char *__restrict__ lists,
                 int *__restrict__ found) {
  extern __shared__ __align__(1024) unsigned char ff_raw[];  // queries, two tiles of keys, [16][128] minima
  __shared__ __align__(8) unsigned long long bars[5];  // keys arrived [2], product done [2], queries arrived
  __shared__ unsigned tmem_at;
  __shared__ int lost[FF_T / FF_GROUP];  // groups of queries that are redone anyway
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = tid >> 7, row = tid & (FF_T - 1);
  const int64_t b = blockIdx.y;
  const int bytes = ff_tile_bytes(C), lower = ff_cp(C) * FF_T * 2, tiles = ff_tiles(N2), steps = 2 * tiles;
  const unsigned sq = ff_smem(ff_raw), sk = sq + bytes;
  const unsigned char *kt = ks.tiles + b * tiles * (int64_t)bytes;
  const unsigned bar_k = ff_smem(bars), bar_d = ff_smem(bars + 2), bar_q = ff_smem(bars + 4);
  if (tid == 0) {
    for (int i = 0; i < 5; ++i) ff_bar_init(ff_smem(bars + i));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < FF_T / FF_GROUP) lost[tid] = 0;
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ff_smem(&tmem_at)), "r"(2 * FF_T)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_at;

  auto fetch = [&](int s) {  // thread 0: the keys of step s
    ff_expect(bar_k + 8 * (s & 1), bytes);
    ff_copy(sk + (s & 1) * bytes, kt + (int64_t)(s < tiles ? s : s - tiles) * bytes, bytes, bar_k + 8 * (s & 1));
  };
  auto product = [&](int s) -> bool {  // thread 0: step s into its half of tensor memory
    if (!ff_wait(bar_k + 8 * (s & 1), (s >> 1) & 1)) return false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned kh = sk + (s & 1) * bytes, d = tmem + (s & 1) * FF_T;
    for (int c = 0; c < ff_cp(C) / 16; ++c) {
      const unsigned o = c * 2 * FF_T * 16;
      const u64 ah = ff_desc(sq + o), al = ff_desc(sq + lower + o), bh = ff_desc(kh + o), bl = ff_desc(kh + lower + o);
      ff_mma(d, ah, bh, c > 0);
      ff_mma(d, ah, bl, 1);
      ff_mma(d, al, bh, 1);
    }
    ff_commit(bar_d + 8 * (s & 1));
    return true;
  };

  bool ok = true;
  if (tid == 0) {
    ff_expect(bar_q, bytes);
    ff_copy(sq, qs.tiles + (b * ff_tiles(N1) + blockIdx.x) * (int64_t)bytes, bytes, bar_q);
    fetch(0);
    fetch(1);
  }
  // the largest norm of the keys
  float r2 = 0.f;
  {
    unsigned top = 0;
    const int nb = (N2 + FF_PREP - 1) / FF_PREP;
    for (int i = lane; i < nb; i += 32) top = max(top, __float_as_uint(ks.block_max[b * nb + i]));
    r2 = __uint_as_float(__reduce_max_sync(FULL, top));
  }
  auto leave = [&]() {
    if (warp == 0) {
      __syncwarp();
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * FF_T) : "memory");
    }
  };
  ok = ff_wait(bar_q, 0);
  const int q = ff_point(blockIdx.x, row);
  if (!(r2 < FF_HUGE) || r2 < 1e-30f) {  // numbers that overflow or are none, or nothing to tell apart
    if (q < N1) found[(b * N1 + q) * 2 + half] = FF_BAD;
    if (tid == 0) {
      ff_wait(bar_k, 0);
      ff_wait(bar_k + 8, 0);
    }
    __syncthreads();
    leave();
    return;
  }
  if (tid == 0) ok = ok && product(0);
  const float qn = *reinterpret_cast<const float *>(ff_raw + ff_upper(C) + 4 * row);
  float m[FF_CLASSES];  // this thread's 32, and later the other's
#pragma unroll
  for (int i = 0; i < FF_CLASSES; ++i) m[i] = __int_as_float(0x7f800000);
  float limit = 0.f;
  // byte offset in the lists (32 bits: they have 512 MB at most); a list that gets full counts as overflowing
  unsigned at = (unsigned)(((b * N1 + q) * 2 + half) * FF_CAP * 2);
  const unsigned begin = at, end = at + FF_CAP * 2;
  const float2 minus2 = make_float2(-2.f, -2.f);

  // the product of step s: v of this thread's columns i and 32 + i, two at a time
  unsigned r0[32], r1[32];
  const float4 *norm = nullptr;
  auto ready = [&](int s) {
    ok = ok && ff_wait(bar_k + 8 * (s & 1), (s >> 1) & 1) && ff_wait(bar_d + 8 * (s & 1), (s >> 1) & 1);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned ta = tmem + (s & 1) * FF_T + half * 64 + ((unsigned)((warp & 3) * 32) << 16);
    norm = reinterpret_cast<const float4 *>(ff_raw + bytes + (s & 1) * bytes + (s < tiles ? ff_upper(C) : ff_lower(C)));
    norm += half * 16;
    ff_load32(ta, r0);
    ff_load32(ta + 32, r1);
    if (tid == 0 && s + 1 < steps) ok = ok && product(s + 1);
    ff_loaded(r0);
    ff_loaded(r1);
  };
  auto value = [&](const unsigned (&r)[32], int i, float x, float y) {
    return __ffma2_rn(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), minus2, make_float2(x, y));
  };
  auto done = [&](int s) -> bool {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (__syncthreads_or(!ok)) return false;  // this step's tensor memory and norms may be overwritten
    if (tid == 0 && s + 2 < steps) fetch(s + 2);
    return true;
  };

  int s = 0;
  bool going = true;
  for (; going && s < tiles; ++s) {
    ready(s);
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 n0 = norm[i / 4], n1 = norm[8 + i / 4];
      const float2 a0 = value(r0, i, n0.x, n0.y), a1 = value(r0, i + 2, n0.z, n0.w);
      const float2 b0 = value(r1, i, n1.x, n1.y), b1 = value(r1, i + 2, n1.z, n1.w);
      m[i] = fminf(m[i], fminf(a0.x, b0.x));
      m[i + 1] = fminf(m[i + 1], fminf(a0.y, b0.y));
      m[i + 2] = fminf(m[i + 2], fminf(a1.x, b1.x));
      m[i + 3] = fminf(m[i + 3], fminf(a1.y, b1.y));
    }
    going = done(s);
  }
  if (going) {  // all minima are known: the first half's thread gets the second's, 16 at a time, and finds the limit
    float *x = reinterpret_cast<float *>(ff_raw + 3 * bytes) + row;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (half == 1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i * FF_T] = m[16 * h + i];
      }
      __syncthreads();
      if (half == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) m[32 + 16 * h + i] = x[i * FF_T];
      }
      __syncthreads();
    }
    if (half == 0) {
      ff_sort<1>(m);
      const float e = fmaf(4.f * ff_error(C), qn, 1.6e-33f);
#pragma unroll
      for (int i = 0; i < FF_CLASSES; ++i)
        if (i == k - 1) limit = m[i] + e;
      if (m[FF_CROWD - 1] <= limit || !(qn < FF_HUGE)) limit = __int_as_float(0x7f800000);
      *x = limit;
      if (!(fabsf(limit) < 3e38f) && q < N1) lost[(q % FF_T) / FF_GROUP] = 1;
    }
    __syncthreads();
    limit = *x;
  }
  // Neither infinite nor not a number, and a query at all; else nothing is below the limit.
  const bool live = fabsf(limit) < 3e38f && q < N1 && !lost[(q % FF_T) / FF_GROUP];
  const float2 over = live ? make_float2(-limit, -limit) : make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
  if (going && !__syncthreads_or(live)) {  // nothing to look for: the tiles and the product under way, and that is all
    ok = ff_wait(bar_k + 8 * (s & 1), (s >> 1) & 1) && ff_wait(bar_d + 8 * (s & 1), (s >> 1) & 1) &&
         ff_wait(bar_k + 8 * ((s + 1) & 1), ((s + 1) >> 1) & 1);
    __syncthreads();
    s = steps;
  }
  for (; going && s < steps; ++s) {
    ready(s);
    unsigned below0 = 0, below1 = 0;  // signs of v - limit, column 0 in the highest bit
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 n0 = norm[i / 4], n1 = norm[8 + i / 4];
      const float2 a0 = __fadd2_rn(value(r0, i, n0.x, n0.y), over), a1 = __fadd2_rn(value(r0, i + 2, n0.z, n0.w), over);
      const float2 b0 = __fadd2_rn(value(r1, i, n1.x, n1.y), over), b1 = __fadd2_rn(value(r1, i + 2, n1.z, n1.w), over);
      below0 = __funnelshift_l(__float_as_uint(a0.x), below0, 1);
      below1 = __funnelshift_l(__float_as_uint(b0.x), below1, 1);
      below0 = __funnelshift_l(__float_as_uint(a0.y), below0, 1);
      below1 = __funnelshift_l(__float_as_uint(b0.y), below1, 1);
      below0 = __funnelshift_l(__float_as_uint(a1.x), below0, 1);
      below1 = __funnelshift_l(__float_as_uint(b1.x), below1, 1);
      below0 = __funnelshift_l(__float_as_uint(a1.y), below0, 1);
      below1 = __funnelshift_l(__float_as_uint(b1.y), below1, 1);
    }
    u64 below = live ? (u64)below0 << 32 | below1 : 0;
    while (below != 0 && at < end) {
      const int i = __clzll((long long)below);
      below &= ~(0x8000000000000000ull >> i);
      *reinterpret_cast<uint16_t *>(lists + at) = (uint16_t)ff_point(s - tiles, half * 64 + i);
      at += 2;
    }
    going = done(s);
  }
  if (q < N1) found[(b * N1 + q) * 2 + half] = !going || !live || at >= end ? FF_BAD : (int)(at - begin) / 2;
  if (!going) {  // copies and products may still be under way: give them time before the block's memory is given up
    if (tid == 0) {
      for (int i = s - 1; i <= s && i < steps; ++i) {
        ff_wait(bar_k + 8 * (i & 1), (i >> 1) & 1);
        ff_wait(bar_d + 8 * (i & 1), (i >> 1) & 1);
      }
    }
    __syncthreads();
  }
  leave();
}

__device__ __forceinline__ u64 ff_exchange(u64 v, int o, bool low) {
  const u64 w = __shfl_xor_sync(FULL, v, o);
  return (w < v) == low ? w : v;
}

// Sorts a bitonic sequence over the lanes; sorts any.
__device__ __forceinline__ u64 ff_merge32(u64 v, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = ff_exchange(v, o, (lane & o) == 0);
  return v;
}
__device__ __forceinline__ u64 ff_sort32(u64 v, int lane) {
#pragma unroll
  for (int w = 2; w <= 32; w <<= 1)
#pragma unroll
    for (int o = w >> 1; o > 0; o >>= 1) v = ff_exchange(v, o, ((lane & o) == 0) == ((lane & w) == 0));
  return v;
}

// One warp per query.  Up to 32 candidates' rows are copied to shared memory, eight lanes a line, and each lane reads its
// own from there (an odd number of 16-byte pieces apart: no bank conflicts); read in place, every load of a warp touches 32
// lines of L1 (61 us for 32 x 1024 queries of 25 candidates, 64 channels).
constexpr int FF_EXACT = 128;

// WIDE: k > 32, two registers of results per lane.
template <bool WIDE>
__global__ void __launch_bounds__(FF_EXACT)
ff_exact_kernel(FfSide qs, FfSide ks, int C, int N1, int N2, int k, const uint16_t *__restrict__ lists,
                const int *__restrict__ found, int *__restrict__ counts, float *__restrict__ dist,
                int64_t *__restrict__ index) {
  extern __shared__ __align__(1024) unsigned char ff_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q = blockIdx.x * (FF_EXACT / 32) + warp, b = blockIdx.y;
  if (q >= N1) return;
  const int64_t query = (int64_t)b * N1 + q;
  // the lists of the whole group: one without sends all of it to the other kernel
  int2 parts = make_int2(k, 0);
  if ((q & ~(FF_GROUP - 1)) + lane < N1)
    parts = *reinterpret_cast<const int2 *>(found + 2 * ((int64_t)b * N1 + (q & ~(FF_GROUP - 1)) + lane));
  int n = parts.x + parts.y;
  const bool bad = __any_sync(FULL, n > 2 * FF_CAP || n < k);
  parts.x = __shfl_sync(FULL, parts.x, q & (FF_GROUP - 1));
  n = __shfl_sync(FULL, n, q & (FF_GROUP - 1));
  if (lane == 0) counts[query] = bad ? -1 : n;
  if (bad) return;
  const int Cr = ff_cr(C), L = Cr / 4, stride = 16 * (L | 1);
  const char *kb = reinterpret_cast<const char *>(ks.rows + (int64_t)b * N2 * Cr);
  const uint16_t *list = lists + query * 2 * FF_CAP;
  const unsigned char *rows = ff_raw + warp * 33 * stride;  // 32 rows, and the query's
  const unsigned mine = ff_smem(rows);
  if (lane < L)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(mine + 32 * stride + 16 * lane),
                 "l"(reinterpret_cast<const char *>(qs.rows + query * Cr) + 16 * lane)
                 : "memory");
  u64 low = ~0ull, high = ~0ull;  // the nearest 32, and the 32 behind them
  for (int c0 = 0; c0 < n; c0 += 32) {
    const int c = c0 + lane, here = min(32, n - c0);
    int j = 0;
    if (c < n) j = list[c < parts.x ? c : FF_CAP + c - parts.x];
    const unsigned off = (unsigned)TK3D_AT(j, N2) * (unsigned)(Cr * 4);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // four rows a step, eight lanes each
      const int r = 4 * i + (lane >> 3);
      const unsigned o = __shfl_sync(FULL, off, r);
      if (4 * i >= here) break;
      if (r < here) {
        const char *src = kb + o + 16 * (lane & 7);
        const unsigned dst = mine + r * stride + 16 * (lane & 7);
#pragma unroll
        for (int p = 0; p < FF_MAX_C / 4; p += 8)
          if (p + (lane & 7) < L)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * p), "l"(src + 16 * p) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    u64 v = ~0ull;
    if (lane < here) {
      const float4 *kr = reinterpret_cast<const float4 *>(rows + lane * stride);
      const float4 *qv = reinterpret_cast<const float4 *>(rows + 32 * stride);
      float d = 0.f;
#pragma unroll 4
      for (int p = 0; p < L; ++p) {  // channels in order, each rounded once; padding channels add nothing
        const float4 x = kr[p], y = qv[p];
        float t = __fsub_rn(x.x, y.x);
        d = __fmaf_rn(t, t, d);
        t = __fsub_rn(x.y, y.y);
        d = __fmaf_rn(t, t, d);
        t = __fsub_rn(x.z, y.z);
        d = __fmaf_rn(t, t, d);
        t = __fsub_rn(x.w, y.w);
        d = __fmaf_rn(t, t, d);
      }
      v = (u64)__float_as_uint(d) << 32 | (unsigned)j;
    }
    __syncwarp();
    v = ff_sort32(v, lane);
    if (c0 == 0) {
      low = v;
    } else {
      v = __shfl_xor_sync(FULL, v, 31);  // descending, against the ascending list
      if (WIDE) {
        const u64 top = v < high ? v : high;  // the nearest 32 of the upper list and the new ones
        v = __shfl_xor_sync(FULL, ff_merge32(top, lane), 31);
        high = ff_merge32(v < low ? low : v, lane);
      }
      low = ff_merge32(v < low ? v : low, lane);
    }
  }
  float *od = dist + query * k;
  int64_t *oi = index + query * k;
  if (lane < k) {
    od[lane] = __uint_as_float((unsigned)(low >> 32));
    oi[lane] = (int64_t)(unsigned)low;
  }
  if (WIDE && 32 + lane < k) {
    od[32 + lane] = __uint_as_float((unsigned)(high >> 32));
    oi[32 + lane] = (int64_t)(unsigned)high;
  }
}

size_t ff_align(size_t n) { return (n + 255) & ~(size_t)255; }

struct FfLayout {
  FfSide q, k;
  uint16_t *lists;
  int *found, *counts;
  size_t total;
};

FfLayout ff_layout(int64_t B, int C, int N1, int N2, bool same, void *scratch) {
  unsigned char *p = static_cast<unsigned char *>(scratch);
  size_t at = 0;
  auto take = [&](size_t n) {
    unsigned char *r = p ? p + at : nullptr;
    at += ff_align(n);
    return r;
  };
  auto side = [&](int N) {
    FfSide s;
    s.tiles = take((size_t)B * ff_tiles(N) * ff_tile_bytes(C));
    s.rows = (float *)take((size_t)B * N * ff_cr(C) * 4);
    s.block_max = (float *)take((size_t)B * ((N + FF_PREP - 1) / FF_PREP) * 4);
    return s;
  };
  FfLayout l;
  l.k = side(N2);
  l.q = same ? l.k : side(N1);
  l.lists = (uint16_t *)take((size_t)B * N1 * FF_CAP * 4);
  l.found = (int *)take((size_t)B * N1 * 8);
  l.counts = (int *)take((size_t)B * N1 * 4);
  l.total = at;
  return l;
}

int ff_prep(const float *in, const float *key, int64_t B, int C, int N, int N2, bool cf, const FfSide &s, cudaStream_t st) {
  const dim3 grid((unsigned)(ff_tiles(N) * (FF_T / FF_PREP)), (unsigned)B);
  if (cf) ff_prep_kernel<true><<<grid, 256, 0, st>>>(in, key, C, N, N2, s);
  else ff_prep_kernel<false><<<grid, 256, 0, st>>>(in, key, C, N, N2, s);
  return check_launch("ff_prep_kernel");
}

}  // namespace

size_t ff_scratch_bytes(int64_t B, int64_t C, int64_t N1, int64_t N2, int64_t k) {
  if (B < 1 || B > 65535 || C < 1 || C > FF_MAX_C || k < 1 || k > FF_MAX_K || N1 < 1 || N1 > (1 << 24) || N2 < 256 ||
      N2 > 65536)
    return 0;
  const size_t n = ff_layout(B, (int)C, (int)N1, (int)N2, false, nullptr).total;
  return n <= ((size_t)512 << 20) ? n : 0;
}

int ff_knn(const float *query, const float *key, int64_t B, int C, int N1, int N2, int k, bool cf, float *dist, int64_t *index,
           void *scratch, const int **counts, cudaStream_t st) {
  const bool same = query == key && N1 == N2;
  const FfLayout l = ff_layout(B, C, N1, N2, same, scratch);
  int rc = ff_prep(key, key, B, C, N2, N2, cf, l.k, st);
  if (rc) return rc;
  if (!same && (rc = ff_prep(query, key, B, C, N1, N2, cf, l.q, st))) return rc;
  const size_t smem = 3 * (size_t)ff_tile_bytes(C) + 16 * FF_T * 4;
  TK3D_CUDA(raise_smem_limit((const void *)ff_filter_kernel, (int)smem));
  ff_filter_kernel<<<dim3((unsigned)ff_tiles(N1), (unsigned)B), FF_THREADS, smem, st>>>(l.q, l.k, C, N1, N2, k,
                                                                                     (unsigned char *)l.lists, l.found);
  if ((rc = check_launch("ff_filter_kernel"))) return rc;
  const size_t rows = (size_t)(FF_EXACT / 32) * 33 * 16 * (ff_cr(C) / 4 | 1);
  auto exact = k > 32 ? ff_exact_kernel<true> : ff_exact_kernel<false>;
  if (rows > 48 * 1024) TK3D_CUDA(raise_smem_limit((const void *)exact, (int)rows));
  exact<<<dim3((unsigned)((N1 + FF_EXACT / 32 - 1) / (FF_EXACT / 32)), (unsigned)B), FF_EXACT, rows, st>>>(
      l.q, l.k, C, N1, N2, k, l.lists, l.found, l.counts, dist, index);
  *counts = l.counts;
  return check_launch("ff_exact_kernel");
}

}  // namespace tk3d

using namespace tk3d;

extern "C" int tk3d_diag_feature_filter(int64_t B, int64_t C, int64_t N1, int64_t N2, int64_t k, int same,
                                        size_t offset[3]) {
  TK3D_REQUIRE(offset != nullptr, TK3D_ERR_NULL, "diag_feature_filter: offset is NULL");
  TK3D_REQUIRE(ff_scratch_bytes(B, C, N1, N2, k) != 0, TK3D_ERR_SHAPE, "diag_feature_filter: sizes that are not served");
  char *const base = reinterpret_cast<char *>(256);
  const FfLayout l = ff_layout(B, (int)C, (int)N1, (int)N2, same != 0 && N1 == N2, base);
  offset[0] = (size_t)(reinterpret_cast<char *>(l.lists) - base);
  offset[1] = (size_t)(reinterpret_cast<char *>(l.found) - base);
  offset[2] = (size_t)(reinterpret_cast<char *>(l.counts) - base);
  return TK3D_OK;
}

TK3D_BOUNDS_TU(feature_filter)
