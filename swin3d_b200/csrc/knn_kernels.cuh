// Host entry points of the KNN kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace s3d {

// thread-per-query scan; root: write distances instead of squared distances; with count (device memory) nothing happens
// unless *count is larger than most
int knn_launch(int K, const float *src, const float *query, const int32_t *src_offset,
               const int32_t *query_offset, int B, int64_t Nq, bool root, int32_t *ret_idx, float *ret_dist,
               cudaStream_t st, const int *count = nullptr, int64_t most = 0);

// warp-per-query scan
bool knn_warp_wanted(int K, int B, int64_t Ns, int64_t Nq);
int knn_launch_warp(int K, const float *src, const float *query, const int32_t *src_offset,
                    const int32_t *query_offset, int B, int64_t Nq, bool root, int32_t *ret_idx, float *ret_dist,
                    cudaStream_t st);

// search over a spatial index
bool knn_tree_supported(int K, int B, int64_t Ns, int64_t Nq);
int64_t knn_tree_bytes(int B, int64_t Ns, int64_t Nq);
int knn_launch_tree(int K, const float *src, const float *query, const int32_t *src_offset,
                    const int32_t *query_offset, int B, int64_t Ns, int64_t Nq, bool root, int32_t *ret_idx,
                    float *ret_dist, void *work, cudaStream_t st);

}  // namespace s3d
