// One-row-per-thread k-means assignment (kmeans_rows.cu).
#pragma once
#include "common.cuh"

namespace fl {

// 1 when the CUDA-core assignment takes this kernel for `rows` rows (all rows of a batch).
int kmeans_rows_pick(int64_t rows, int K, int d);
int launch_kmeans_rows(const float* x, int batch, int64_t n, int64_t ldx, int64_t xbs, const float* c, int K, int64_t ldc,
                       int64_t cbs, int d, int32_t* labels, cudaStream_t st);

}  // namespace fl
