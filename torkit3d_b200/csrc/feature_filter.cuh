// Feature-space neighbours by tensor cores: see feature_filter.cu.
#pragma once

#include "tk3d_common.cuh"

namespace tk3d {

constexpr int FF_GROUP = 32;  // queries that feature_knn_kernel redoes together

// 0 where the sizes are not served.
size_t ff_scratch_bytes(int64_t B, int64_t C, int64_t N1, int64_t N2, int64_t k);
// Distances and indices of all queries but those whose entry in (*counts)[B * N1] is -1, whole groups of FF_GROUP.
int ff_knn(const float *query, const float *key, int64_t B, int C, int N1, int N2, int k, bool cf, float *dist, int64_t *index,
           void *scratch, const int **counts, cudaStream_t st);

}  // namespace tk3d
