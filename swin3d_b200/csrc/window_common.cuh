// Which window and cell a voxel falls into; shared by the two window builders.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace s3d {

constexpr int CELL_BITS = 9, W_BITS = 15, B_BITS = 10;       // supported range: batch < 2^10, |window index| < 2^14
constexpr int W_BIAS = 1 << (W_BITS - 1);

struct WindowGrid {
    int stride, ws, shift;
};

struct VoxelWindow {
    int b, wx, wy, wz, cx, cy, cz, cell;
};

__device__ __forceinline__ int floor_div(int a, int b) { const int q = a / b; return a - q * b < 0 ? q - 1 : q; }   // b > 0

// Window = floor((coord + shift*stride) / (ws*stride)) per axis, cell = position inside it,
// cell id = cx*ws^2 + cy*ws + cz.
__device__ __forceinline__ VoxelWindow voxel_window(const int32_t *__restrict__ coords, int64_t i, const WindowGrid &g)
{
    const int4 c = __ldg(reinterpret_cast<const int4 *>(coords) + i);  // b, x, y, z
    const int wstride = g.ws * g.stride;
    const int sx = c.y + g.shift * g.stride, sy = c.z + g.shift * g.stride, sz = c.w + g.shift * g.stride;
    VoxelWindow v;
    v.b = c.x;
    v.wx = floor_div(sx, wstride); v.wy = floor_div(sy, wstride); v.wz = floor_div(sz, wstride);
    v.cx = (sx - v.wx * wstride) / g.stride; v.cy = (sy - v.wy * wstride) / g.stride; v.cz = (sz - v.wz * wstride) / g.stride;
    v.cell = (v.cx * g.ws + v.cy) * g.ws + v.cz;
    return v;
}

__device__ __forceinline__ bool voxel_in_range(const VoxelWindow &v)
{
    const int bx = v.wx + W_BIAS, by = v.wy + W_BIAS, bz = v.wz + W_BIAS;
    return v.b >= 0 && v.b < (1 << B_BITS) && bx >= 0 && bx < (1 << W_BITS) && by >= 0 && by < (1 << W_BITS) && bz >= 0 &&
           bz < (1 << W_BITS) && v.cell < (1 << CELL_BITS);
}

}  // namespace s3d
