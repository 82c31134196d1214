// Gradient of a row gather (group_points, set abstraction, edge features; float32): see scatter.cu.
#pragma once

#include "tk3d_common.cuh"

namespace tk3d {

struct ScatterCall {
  const float *gout = nullptr;  // channels [0,C) of every cloud's slab of gstride elements, E = M*K entries each
  const void *index = nullptr;  // [B][E]
  int index_i32 = 0;
  int64_t B = 0, C = 0, N = 0, M = 0, K = 0, gstride = 0;
  float *gin = nullptr;         // [B][C][N]
  float *gq = nullptr;          // [B][C][M]: sums over each query's K entries, see scatter_edge_entries
  int include_query = 0;
  int32_t *status = nullptr;
  void *scratch = nullptr;      // scatter_scratch_bytes(B, C, N), 16-byte aligned
};

inline size_t scatter_scratch_bytes(int64_t B, int64_t C, int64_t N) {
  return (size_t)B * (size_t)N * (size_t)((C + 3) & ~(int64_t)3) * 4;
}
// Sizes that 16-byte accesses do not fit take the direct kernels while they are small: three launches and a scratch buffer
// cost the caller 7 us more than two (10 x 111 channels, 231 x 36 entries 128 -> 135; 7 x 24, 3557 x 22 192 -> 163).
// Clouds of more points than the transposition takes have their rows written back by unrow_kernel, for few channels a
// small part of a tile: 4 x 2097121 <- 64 x 16 entries 22 us direct and 60 by rows, 4 x 2097121 <- 524288 37 / 77, 64 x
// 4200000 <- 32768 263 / 492, but 16 x 2097121 <- 524288 191 / 117, 32 x 3000001 <- 1600000 1853 / 325.
constexpr int64_t SCATTER_TRANSPOSED = 65535 * 32;  // points: they are a grid's y there
inline bool scatter_pays(int64_t B, int64_t C, int64_t N, int64_t M, int64_t K) {
  if (N > SCATTER_TRANSPOSED && (C < 16 || 4 * M * K < N)) return false;
  return (C % 4 == 0 && (M * K) % 4 == 0) || B * C * M * K >= 12000000;
}
// Whether the sizes are served.
bool scatter_ok(int64_t B, int64_t C, int64_t N, int64_t M, int64_t K);
// Entries of a tile where gq can be summed in the same pass, else 0.
int scatter_edge_entries(const void *gout, int64_t E, int64_t gstride, int64_t K);
int scatter_launch(const ScatterCall &c, cudaStream_t st);

}  // namespace tk3d
