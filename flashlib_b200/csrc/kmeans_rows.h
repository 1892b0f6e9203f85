// One-row-per-thread k-means assignment (kmeans_rows.cu).
#pragma once
#include "common.cuh"

namespace fl {

// 1 when the CUDA-core assignment takes this kernel for `rows` rows (all rows of a batch).
int kmeans_rows_pick(int64_t rows, int K, int d);
int launch_kmeans_rows(const float* x, int batch, int64_t n, int64_t ldx, int64_t xbs, const float* c, int K, int64_t ldc,
                       int64_t cbs, int d, int32_t* labels, cudaStream_t st);

// Control words of a Lloyd loop on the device, its centroid step (kmeans_step_kernel) and the host's wait for iteration `want`.
enum { LLOYD_DONE = 0, LLOYD_BLOCKS = 1, LLOYD_SHIFT = 2, LLOYD_WORDS = 4 };
int launch_kmeans_step(float* sums, int32_t* cnts, const float* old_c, float* new_c, int64_t KB, int d, int clear, float tol, int it,
                       int32_t* ctl, int32_t* host, float* shift, cudaStream_t st);
void lloyd_wait(const int32_t* host, int want, cudaStream_t st);

}  // namespace fl
