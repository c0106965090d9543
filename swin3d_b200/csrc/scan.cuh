// Exclusive scan of an array of counters in place, in two launches: tile sums, then every block adds up
// the sums of the tiles before its own (a few thousand words from L2 at most) and scans its tile.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace s3d {
namespace {

constexpr int SCAN_T = 256, SCAN_PER = 16, SCAN_TILE = SCAN_T * SCAN_PER;   // the array is a whole number of tiles

__global__ void __launch_bounds__(SCAN_T)
scan_tile_sums_kernel(const uint32_t *__restrict__ hist, uint32_t *__restrict__ tile)
{
    const uint4 *p = reinterpret_cast<const uint4 *>(hist + (int64_t)blockIdx.x * SCAN_TILE);
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < SCAN_PER / 4; ++j) {
        const uint4 v = p[j * SCAN_T + threadIdx.x];
        s += v.x + v.y + v.z + v.w;
    }
    __shared__ uint32_t s_w[SCAN_T / 32];
    s = __reduce_add_sync(0xffffffffu, s);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t v = __reduce_add_sync(0xffffffffu, threadIdx.x < SCAN_T / 32 ? s_w[threadIdx.x] : 0u);
        if (threadIdx.x == 0) tile[blockIdx.x] = v;
    }
}

__global__ void __launch_bounds__(SCAN_T)
scan_apply_kernel(uint32_t *__restrict__ hist, const uint32_t *__restrict__ tile)
{
    __shared__ uint32_t s_w[SCAN_T / 32], s_base[SCAN_T / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t before = 0;
    for (int i = threadIdx.x; i < (int)blockIdx.x; i += SCAN_T) before += __ldg(tile + i);
    before = __reduce_add_sync(0xffffffffu, before);
    uint4 *p = reinterpret_cast<uint4 *>(hist + (int64_t)blockIdx.x * SCAN_TILE) + threadIdx.x * (SCAN_PER / 4);
    uint4 v[SCAN_PER / 4];
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < SCAN_PER / 4; ++j) {
        v[j] = p[j];
        sum += v[j].x + v[j].y + v[j].z + v[j].w;
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_w[wid] = incl;
    if (lane == 0) s_base[wid] = before;
    __syncthreads();
    uint32_t run = incl - sum;
#pragma unroll
    for (int w = 0; w < SCAN_T / 32; ++w) run += s_base[w] + (w < wid ? s_w[w] : 0u);
#pragma unroll
    for (int j = 0; j < SCAN_PER / 4; ++j) {
        uint4 o;
        o.x = run; run += v[j].x;
        o.y = run; run += v[j].y;
        o.z = run; run += v[j].z;
        o.w = run; run += v[j].w;
        p[j] = o;
    }
}

inline void scan_in_place(uint32_t *counters, uint32_t *tile, int n_tiles, cudaStream_t st)
{
    scan_tile_sums_kernel<<<(unsigned)n_tiles, SCAN_T, 0, st>>>(counters, tile);
    scan_apply_kernel<<<(unsigned)n_tiles, SCAN_T, 0, st>>>(counters, tile);
}

}  // namespace
}  // namespace s3d
