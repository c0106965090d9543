// Window grouping over a dense grid of windows, for batches whose windows fill a fair part of their
// bounding box and whose voxels are distinct -- what a voxelised scan gives.  Same results as the radix
// sort of window_build.cu, which remains for everything else.
//
// The windows of the box are numbered in (batch, wx, wy, wz) order, which is the order they come out in.
// Every window owns a bit mask of its ws^3 cells.  A voxel sets its bit; a scan over the windows turns
// the masks into first positions (and emits the window lists); the place of a voxel is then the first
// position of its window plus the number of set bits below its own.  No keys, no sort passes: the
// coordinates are read three times (the second and third time mostly from L2), every output is
// written once.
//
// Bound: HBM for large batches (964 k voxels, 9 signals: 74 us for all kernels, 262 us for the radix
// chain), launches for small ones (6 instead of 57).
#include <climits>

#include "common.cuh"
#include "window_common.cuh"
#include "window_kernels.cuh"

namespace s3d {
namespace {

constexpr int WD_THREADS = 256;
constexpr int WD_PER = 4;                                    // windows per thread of the scan
constexpr int WD_TILE = WD_THREADS * WD_PER;

struct WdTile {
    unsigned long long sq;
    uint32_t voxels, windows;
};

struct WdBufs {
    uint32_t *range;       // [8] keys of -min and max of (batch, wx, wy, wz); cleared
    int64_t *counts;       // [4] windows, pairs, largest window, WD_* bits; cleared
    uint32_t *mask;        // [windows][words]; cleared
    uint32_t *start;       // [windows]
    WdTile *tile;
    int64_t cleared, total;
    int64_t cap;           // windows there is room for
    int words;             // mask words per window
};

// Room for 4 mask words per voxel: 964 k voxels of rooms span 127 k windows of 5^3 cells (4 words each).
WdBufs wd_layout(char *base, int64_t N, int ws)
{
    WdBufs b{};
    b.words = (ws * ws * ws + 31) / 32;
    const int64_t words = N * 4 < (1 << 16) ? (1 << 16) : N * 4;
    b.cap = words / b.words;
    int64_t off = 0;
    auto take = [&](int64_t bytes) { const int64_t o = off; off = (off + bytes + 255) / 256 * 256; return base + o; };
    b.range = (uint32_t *)take(64);
    b.counts = (int64_t *)(base + 32);
    b.mask = (uint32_t *)take(words * 4);
    b.cleared = off;
    b.start = (uint32_t *)take(b.cap * 4);
    b.tile = (WdTile *)take((b.cap + WD_TILE - 1) / WD_TILE * (int64_t)sizeof(WdTile));
    b.total = off;
    return b;
}

// The box of windows, from the reduced range.
struct WdBox {
    int lo[4];
    uint32_t n[4];
    bool fits;
    uint32_t total;
};

__device__ __forceinline__ int key_to_int(uint32_t k) { return (int)(k ^ 0x80000000u); }
__device__ __forceinline__ uint32_t int_to_key(int v) { return (uint32_t)v ^ 0x80000000u; }

__device__ __forceinline__ WdBox wd_box(const WdBufs &b)
{
    WdBox x;
    unsigned long long t = 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        x.lo[k] = -key_to_int(__ldg(b.range + k));
        x.n[k] = (uint32_t)(key_to_int(__ldg(b.range + 4 + k)) - x.lo[k] + 1);
    }
    // spans are below 2^16 after the range check (whose violation the host reports): no overflow
#pragma unroll
    for (int k = 0; k < 4; ++k) t *= x.n[k] & 0xffffu;
    x.fits = t <= (unsigned long long)b.cap;
    x.total = x.fits ? (uint32_t)t : 0u;
    return x;
}

__global__ void __launch_bounds__(WD_THREADS)
wd_range_kernel(const int32_t *__restrict__ coords, int64_t N, WindowGrid w, WdBufs b)
{
    uint32_t m[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    bool bad = false;
    for (int64_t i = (int64_t)blockIdx.x * WD_THREADS + threadIdx.x; i < N; i += (int64_t)gridDim.x * WD_THREADS) {
        const VoxelWindow v = voxel_window(coords, i, w);
        const int f[4] = {v.b, v.wx, v.wy, v.wz};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            m[k] = max(m[k], int_to_key(-f[k]));
            m[4 + k] = max(m[4 + k], int_to_key(f[k]));
        }
        bad = bad || !voxel_in_range(v);
    }
    __shared__ uint32_t s_m[8];
    if (threadIdx.x < 8) s_m[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t r = __reduce_max_sync(0xffffffffu, m[k]);
        if ((threadIdx.x & 31) == 0) atomicMax(s_m + k, r);
    }
    __syncthreads();
    if (threadIdx.x < 8) atomicMax(b.range + threadIdx.x, s_m[threadIdx.x]);
    if (bad) atomicOr(reinterpret_cast<unsigned long long *>(b.counts + 3), (unsigned long long)WD_BAD_RANGE);
}

__device__ __forceinline__ uint32_t wd_index(const WdBox &x, const VoxelWindow &v)
{
    return ((((uint32_t)(v.b - x.lo[0]) * x.n[1] + (uint32_t)(v.wx - x.lo[1])) * x.n[2]) + (uint32_t)(v.wy - x.lo[2])) * x.n[3] +
           (uint32_t)(v.wz - x.lo[3]);
}

__global__ void __launch_bounds__(WD_THREADS)
wd_mark_kernel(const int32_t *__restrict__ coords, int64_t N, WindowGrid w, WdBufs b)
{
    if (b.counts[3] & WD_BAD_RANGE) return;
    const WdBox x = wd_box(b);
    if (!x.fits) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(reinterpret_cast<unsigned long long *>(b.counts + 3), (unsigned long long)WD_TOO_SPARSE);
        return;
    }
    const int64_t i = (int64_t)blockIdx.x * WD_THREADS + threadIdx.x;
    if (i >= N) return;
    const VoxelWindow v = voxel_window(coords, i, w);
    const uint32_t bit = 1u << (v.cell & 31);
    const uint32_t old = atomicOr(b.mask + (int64_t)wd_index(x, v) * b.words + (v.cell >> 5), bit);
    if ((old & bit) && !(*(volatile int64_t *)(b.counts + 3) & WD_REPEATED))      // half of a million voxels repeated: 300 us of atomics
        atomicOr(reinterpret_cast<unsigned long long *>(b.counts + 3), (unsigned long long)WD_REPEATED);
}

__device__ __forceinline__ uint32_t wd_count(const WdBufs &b, uint32_t win, uint32_t total)
{
    uint32_t c = 0;
    if (win < total)
        for (int k = 0; k < b.words; ++k) c += __popc(__ldg(b.mask + (int64_t)win * b.words + k));
    return c;
}

__global__ void __launch_bounds__(WD_THREADS)
wd_tile_kernel(WdBufs b)
{
    if (b.counts[3]) return;                                   // the sort takes over
    const uint32_t total = wd_box(b).total;
    if (blockIdx.x * (uint32_t)WD_TILE >= total) return;
    unsigned long long sq = 0;
    uint32_t vox = 0, wins = 0, mx = 0;
#pragma unroll
    for (int j = 0; j < WD_PER; ++j) {
        const uint32_t c = wd_count(b, blockIdx.x * (uint32_t)WD_TILE + j * WD_THREADS + threadIdx.x, total);
        vox += c;
        wins += c != 0;
        sq += (unsigned long long)c * c;
        mx = max(mx, c);
    }
    __shared__ uint32_t s_v[WD_THREADS / 32], s_w[WD_THREADS / 32], s_x[WD_THREADS / 32];
    __shared__ unsigned long long s_q[WD_THREADS / 32];
    vox = __reduce_add_sync(0xffffffffu, vox);
    wins = __reduce_add_sync(0xffffffffu, wins);
    mx = __reduce_max_sync(0xffffffffu, mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) {
        const int k = threadIdx.x >> 5;
        s_v[k] = vox; s_w[k] = wins; s_q[k] = sq; s_x[k] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        WdTile t{0, 0, 0};
        mx = 0;
        for (int k = 0; k < WD_THREADS / 32; ++k) {
            t.voxels += s_v[k]; t.windows += s_w[k]; t.sq += s_q[k];
            mx = max(mx, s_x[k]);
        }
        b.tile[blockIdx.x] = t;
        atomicAdd(reinterpret_cast<unsigned long long *>(b.counts), (unsigned long long)t.windows);
        atomicAdd(reinterpret_cast<unsigned long long *>(b.counts + 1), t.sq);
        atomicMax(reinterpret_cast<long long *>(b.counts + 2), (long long)mx);
    }
}

// First position of every window; the occupied ones go to the window lists.
__global__ void __launch_bounds__(WD_THREADS)
wd_scan_kernel(WdBufs b, int32_t *__restrict__ w_sizes, int32_t *__restrict__ w2n, int64_t *__restrict__ w2m)
{
    if (b.counts[3]) return;
    const uint32_t total = wd_box(b).total;
    const uint32_t base = blockIdx.x * (uint32_t)WD_TILE;
    if (base >= total) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // what lies before this tile
    uint32_t vox = 0, wins = 0;
    unsigned long long sq = 0;
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += WD_THREADS) {
        vox += b.tile[t].voxels;
        wins += b.tile[t].windows;
        sq += b.tile[t].sq;
    }
    uint32_t c[WD_PER], tv = 0, tw = 0;
    unsigned long long tq = 0;
#pragma unroll
    for (int j = 0; j < WD_PER; ++j) {
        c[j] = wd_count(b, base + threadIdx.x * WD_PER + j, total);
        tv += c[j];
        tw += c[j] != 0;
        tq += (unsigned long long)c[j] * c[j];
    }
    uint32_t iv = tv, iw = tw;
    unsigned long long iq = tq;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t yv = __shfl_up_sync(0xffffffffu, iv, o), yw = __shfl_up_sync(0xffffffffu, iw, o);
        const unsigned long long yq = __shfl_up_sync(0xffffffffu, iq, o);
        if (lane >= o) { iv += yv; iw += yw; iq += yq; }
    }
    vox = __reduce_add_sync(0xffffffffu, vox);
    wins = __reduce_add_sync(0xffffffffu, wins);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    __shared__ uint32_t s_v[WD_THREADS / 32], s_w[WD_THREADS / 32], s_bv[WD_THREADS / 32], s_bw[WD_THREADS / 32];
    __shared__ unsigned long long s_q[WD_THREADS / 32], s_bq[WD_THREADS / 32];
    if (lane == 31) { s_v[wid] = iv; s_w[wid] = iw; s_q[wid] = iq; }
    if (lane == 0) { s_bv[wid] = vox; s_bw[wid] = wins; s_bq[wid] = sq; }
    __syncthreads();
    uint32_t rv = iv - tv, rw = iw - tw;
    unsigned long long rq = iq - tq;
#pragma unroll
    for (int k = 0; k < WD_THREADS / 32; ++k) {
        rv += s_bv[k] + (k < wid ? s_v[k] : 0u);
        rw += s_bw[k] + (k < wid ? s_w[k] : 0u);
        rq += s_bq[k] + (k < wid ? s_q[k] : 0ull);
    }
#pragma unroll
    for (int j = 0; j < WD_PER; ++j) {
        const uint32_t win = base + threadIdx.x * WD_PER + j;
        if (win < total) b.start[win] = rv;
        if (c[j]) {
            w_sizes[rw] = (int32_t)c[j];
            w2n[rw] = (int32_t)rv;
            w2m[rw] = (int64_t)rq;
            ++rw;
        }
        rv += c[j];
        rq += (unsigned long long)c[j] * c[j];
    }
}

__global__ void __launch_bounds__(WD_THREADS)
wd_scatter_kernel(const int32_t *__restrict__ coords, const float *__restrict__ xyz, int xyz_stride, const float *__restrict__ rest,
                  int rest_stride, int64_t N, int F, WindowGrid w, WdBufs b,
                  int32_t *__restrict__ n2n, float *__restrict__ n_coords)
{
    if (b.counts[3]) return;
    const WdBox x = wd_box(b);
    const int64_t i = (int64_t)blockIdx.x * WD_THREADS + threadIdx.x;
    if (i >= N) return;
    const VoxelWindow v = voxel_window(coords, i, w);
    const uint32_t win = wd_index(x, v);
    const uint32_t *m = b.mask + (int64_t)win * b.words;
    uint32_t pos = __ldg(b.start + win) + __popc(__ldg(m + (v.cell >> 5)) & ((1u << (v.cell & 31)) - 1u));
    for (int k = 0; k < (v.cell >> 5); ++k) pos += __popc(__ldg(m + k));
    n2n[pos] = (int32_t)i;
    const float *f = xyz + i * xyz_stride, *r = rest + i * rest_stride;
    float *o = n_coords + (int64_t)pos * F;
    o[0] = (float)v.cx + __ldg(f);
    o[1] = (float)v.cy + __ldg(f + 1);
    o[2] = (float)v.cz + __ldg(f + 2);
    for (int j = 3; j < F; ++j) o[j] = __ldg(r + j - 3);
}

}  // namespace

int64_t window_dense_workspace_bytes(int64_t N, int ws) { return wd_layout(nullptr, N, ws).total; }

int window_dense_launch(const int32_t *coords, const float *xyz, int xyz_stride, const float *rest, int rest_stride,
                        int64_t N, int F, int stride, int ws, int shift, int32_t *n2n, float *n_coords, int32_t *w_sizes,
                        int32_t *w2n, int64_t *w2m, uint32_t **state, void *workspace, int64_t workspace_bytes, cudaStream_t st)
{
    const WdBufs b = wd_layout(static_cast<char *>(workspace), N, ws);
    if (workspace_bytes < b.total) return S3D_ERR_WORKSPACE;
    *state = b.range;
    if (cudaMemsetAsync(b.range, 0, (size_t)b.cleared, st) != cudaSuccess) return S3D_ERR_LAUNCH;
    if (N == 0) return S3D_OK;
    const WindowGrid w{stride, ws, shift};
    const unsigned nb = (unsigned)((N + WD_THREADS - 1) / WD_THREADS);
    const unsigned tiles = (unsigned)((b.cap + WD_TILE - 1) / WD_TILE);
    wd_range_kernel<<<nb < 148u * 8u ? nb : 148u * 8u, WD_THREADS, 0, st>>>(coords, N, w, b);
    wd_mark_kernel<<<nb, WD_THREADS, 0, st>>>(coords, N, w, b);
    wd_tile_kernel<<<tiles, WD_THREADS, 0, st>>>(b);
    wd_scan_kernel<<<tiles, WD_THREADS, 0, st>>>(b, w_sizes, w2n, w2m);
    wd_scatter_kernel<<<nb, WD_THREADS, 0, st>>>(coords, xyz, xyz_stride, rest, rest_stride, N, F, w, b, n2n, n_coords);
    return cudaGetLastError() == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}

}  // namespace s3d
