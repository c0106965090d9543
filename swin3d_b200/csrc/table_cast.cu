// The fp16 copies of a layer's three fp32 tables.  As three torch casts this was three launches of 1.6 us and
// 20 us of host time, more than the attention kernel of a deep stage takes on a small room; the data, 0.1 to
// 2 MB, is never what counts.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/swin3d_b200.h"

namespace s3d {
namespace {

struct Tables {
    const float *src[3];
};

// grid = (x, 3); VEC: sources and destinations are 16- and 8-byte aligned and n is a multiple of four
template <bool VEC>
__global__ void __launch_bounds__(256) cast_tables_kernel(const Tables t, int64_t n, __half *__restrict__ dst)
{
    const float *src = blockIdx.y == 0 ? t.src[0] : (blockIdx.y == 1 ? t.src[1] : t.src[2]);
    __half *out = dst + blockIdx.y * n;
    const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    if (VEC) {
        for (int64_t i = first; i < n / 4; i += step) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(src) + i);
            const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
            reinterpret_cast<uint2 *>(out)[i] = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
        }
    } else {
        for (int64_t i = first; i < n; i += step) out[i] = __float2half_rn(__ldg(src + i));
    }
}

}  // namespace
}  // namespace s3d

extern "C" int s3d_cast_tables(const float *tq, const float *tk, const float *tv, int64_t n, void *dst, void *stream)
{
    if (n < 0) return S3D_ERR_BAD_ARG;
    if (n == 0) return S3D_OK;
    if (!tq || !tk || !tv || !dst) return S3D_ERR_BAD_ARG;
    const bool vec = !((reinterpret_cast<uintptr_t>(tq) | reinterpret_cast<uintptr_t>(tk) | reinterpret_cast<uintptr_t>(tv)) & 15) &&
                     !(reinterpret_cast<uintptr_t>(dst) & 7) && n % 4 == 0;
    const int64_t items = vec ? n / 4 : n;
    const unsigned gx = (unsigned)((items + 255) / 256 < 148 ? (items + 255) / 256 : 148);
    const s3d::Tables t{{tq, tk, tv}};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (vec) s3d::cast_tables_kernel<true><<<dim3(gx, 3), 256, 0, st>>>(t, n, static_cast<__half *>(dst));
    else s3d::cast_tables_kernel<false><<<dim3(gx, 3), 256, 0, st>>>(t, n, static_cast<__half *>(dst));
    return cudaGetLastError() == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}
