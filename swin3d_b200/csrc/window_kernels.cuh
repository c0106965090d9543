// Host entry points of the window builder.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace s3d {
int64_t window_build_workspace_bytes(int64_t N);
int window_build_launch(const int32_t *coords, const float *feats, int64_t N, int F, int stride,
                        int ws, int shift, int32_t *n2n, float *n_coords, int32_t *w_sizes,
                        int32_t *w2n, int64_t *counts, void *workspace, int64_t workspace_bytes,
                        cudaStream_t st);

// dense grid of windows; bits of counts[3] (0: the results are complete)
constexpr int WD_BAD_RANGE = 1, WD_TOO_SPARSE = 2, WD_REPEATED = 4;
int64_t window_dense_workspace_bytes(int64_t N, int ws);
int window_dense_launch(const int32_t *coords, const float *xyz, int xyz_stride, const float *rest, int rest_stride,
                        int64_t N, int F, int stride, int ws, int shift, int32_t *n2n, float *n_coords, int32_t *w_sizes,
                        int32_t *w2n, int64_t *w2m, int64_t **counts, void *workspace, int64_t workspace_bytes,
                        cudaStream_t st);
}  // namespace s3d
