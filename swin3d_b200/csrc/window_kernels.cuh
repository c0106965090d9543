// Host entry points of the window builder.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace s3d {
int64_t window_build_workspace_bytes(int64_t N);
constexpr int WB_MAX_PASSES = 8;
// radix passes that cover the used bits of the keys; span: max - min of (batch, wx, wy, wz), within the supported range
int window_build_passes(const int *span);
// xyz, rest: the first three and the other F - 3 signals of a voxel, rows of the given strides
int window_build_launch(const int32_t *coords, const float *xyz, int xyz_stride, const float *rest, int rest_stride, int64_t N,
                        int F, int stride, int ws, int shift, int32_t *n2n, float *n_coords, int32_t *w_sizes,
                        int32_t *w2n, int64_t *counts, void *workspace, int64_t workspace_bytes,
                        cudaStream_t st, int passes = WB_MAX_PASSES);

// dense grid of windows; state: 64 bytes of device memory, the keys of -min and max of (batch, wx, wy, wz) (sign bit
// flipped), then counts[4]; bits of counts[3] (0: the results are complete)
constexpr int WD_BAD_RANGE = 1, WD_TOO_SPARSE = 2, WD_REPEATED = 4;
int64_t window_dense_workspace_bytes(int64_t N, int ws);
int window_dense_launch(const int32_t *coords, const float *xyz, int xyz_stride, const float *rest, int rest_stride,
                        int64_t N, int F, int stride, int ws, int shift, int32_t *n2n, float *n_coords, int32_t *w_sizes,
                        int32_t *w2n, int64_t *w2m, uint32_t **state, void *workspace, int64_t workspace_bytes,
                        cudaStream_t st);
}  // namespace s3d
