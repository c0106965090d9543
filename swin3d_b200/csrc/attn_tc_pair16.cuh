// Pieces of the kernels that serve two heads of 16 channels per block (half2 entries = two heads).
//
// A product that contracts over channels is one k-step: an mma lane t holds channels 4t, 4t+1 in its first and 4t+2, 4t+3
// in its second half (any split serves as long as both operands use it), so that its part of a row is one 8-byte load.  A product whose columns are channels runs once for the even and once for the odd channels: lane g loads
// channels 2g, 2g+1 of the two rows of a k pair with 4-byte loads and swaps halves, and an accumulator lane ends with
// channels 4t..4t+3.
#pragma once
#include "attn_tc.cuh"
#include "attn_tc_small.cuh"

namespace s3d {
namespace tc {

constexpr int P16_RS = 40;                       // halves per staged voxel row: 32 + 8, so that 8 rows start in different banks
__host__ __device__ constexpr int p16_warps(int D) { return D == 3 ? 11 : 15; }

__device__ __forceinline__ void mma_f32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    mma_k16(d, a[0], a[1], a[2], a[3], b0, b1);
}

// Table rows of a 16-row tile as A operands of the projections: [slot][row g, g + 8], .x / .y = first / second k-step.
struct P16TileA {
    uint2 f[2][2];
    __device__ __forceinline__ void fetch(const __half *T, int HC, int co, const uint16_t *map, int mt, int g, int t)
    {
        const int r0 = map[mt * 16 + g], r1 = map[mt * 16 + g + 8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            f[h][0] = r0 != 0xffff ? __ldg(reinterpret_cast<const uint2 *>(T + (int64_t)r0 * HC + co + h * 16 + 4 * t)) : make_uint2(0, 0);
            f[h][1] = r1 != 0xffff ? __ldg(reinterpret_cast<const uint2 *>(T + (int64_t)r1 * HC + co + h * 16 + 4 * t)) : make_uint2(0, 0);
        }
    }
};

// The same rows as B operands of the hist.T products (k = row in ht_krow order, n = channel): raw[slot][half][first, second
// row of the pair] = channels 2g, 2g + 1.
struct P16TileB {
    uint32_t raw[2][2][2];
    __device__ __forceinline__ void fetch(const __half *T, int HC, int co, const uint16_t *map, int ks, int g, int t)
    {
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int second = 0; second < 2; ++second) {
                const int r = map[ks * 16 + ht_krow(t, half, second)];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    raw[h][half][second] = r != 0xffff ? __ldg(reinterpret_cast<const uint32_t *>(T + (int64_t)r * HC + co + h * 16 + 2 * g)) : 0u;
            }
    }
};

// The operands of the products themselves: b[slot][even / odd channels][half].
struct P16FragB {
    uint32_t b[2][2][2];
    __device__ __forceinline__ explicit P16FragB(const P16TileB &tile)
    {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                b[h][0][half] = pack_lo(tile.raw[h][half][0], tile.raw[h][half][1]);
                b[h][1][half] = pack_hi(tile.raw[h][half][0], tile.raw[h][half][1]);
            }
    }
    __device__ __forceinline__ P16FragB(const uint4 &x, const uint4 &y) : b{{{x.x, x.y}, {x.z, x.w}}, {{y.x, y.y}, {y.z, y.w}}} {}
};

// acc[slot][even / odd channels][m-tile] += A . rows with A from a [32][ES] plane of half2 pair entries: TRANSPOSED = false:
// m = query, k = key (entry [k][m]); true: m = key, k = query (entry [m][k]).
// WORDS: 4-byte words per entry (the half2 comes first).
template <bool TRANSPOSED, int WORDS = 1>
__device__ __forceinline__ void p16_pair_gemm(float (&acc)[2][2][2][4], const uint32_t *e32, const __half *rows, int nk, int g, int t)
{
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
        if (16 * ks < nk) {
            uint32_t b[2][2][2];                               // [slot][parity][half]
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int kh = 0; kh < 2; ++kh) {
                    const int ka = 16 * ks + 2 * t + 8 * kh;
                    const uint32_t u = *reinterpret_cast<const uint32_t *>(rows + ka * P16_RS + h * 16 + 2 * g);
                    const uint32_t w = *reinterpret_cast<const uint32_t *>(rows + (ka + 1) * P16_RS + h * 16 + 2 * g);
                    b[h][0][kh] = pack_lo(u, w);
                    b[h][1][kh] = pack_hi(u, w);
                }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t fa[2][4];
#pragma unroll
                for (int kh = 0; kh < 2; ++kh)
#pragma unroll
                    for (int rr = 0; rr < 2; ++rr) {
                        const int m = 16 * i + g + 8 * rr, ka = 16 * ks + 2 * t + 8 * kh;
                        const uint32_t u = TRANSPOSED ? e32[(m * ES + ka) * WORDS] : e32[(ka * ES + m) * WORDS];
                        const uint32_t w = TRANSPOSED ? e32[(m * ES + ka + 1) * WORDS] : e32[((ka + 1) * ES + m) * WORDS];
                        fa[0][2 * kh + rr] = pack_lo(u, w);
                        fa[1][2 * kh + rr] = pack_hi(u, w);
                    }
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int p = 0; p < 2; ++p) mma_f32(acc[h][p][i], fa[h], b[h][p][0], b[h][p][1]);
            }
        }
    }
}

// Accumulators [slot][parity][m-tile] to a [32][32] array: lane (g, t) holds channels 4t..4t+3 of rows g, g + 8.
__device__ __forceinline__ void p16_store(float *dst, const float (&acc)[2][2][2][4], int g, int t)
{
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int rr = 0; rr < 2; ++rr)
                *reinterpret_cast<float4 *>(dst + (16 * i + g + 8 * rr) * 32 + h * 16 + 4 * t) =
                    make_float4(acc[h][0][i][2 * rr], acc[h][1][i][2 * rr], acc[h][0][i][2 * rr + 1], acc[h][1][i][2 * rr + 1]);
}

__device__ __forceinline__ void p16_zero(float (&acc)[2][2][2][4])
{
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < 2; ++i) acc[h][p][i][0] = acc[h][p][i][1] = acc[h][p][i][2] = acc[h][p][i][3] = 0.f;
}

// Feature fragments of a staged array for the projections: [voxels 8j + g][slot], channels 4t..4t+3.
__device__ __forceinline__ void p16_feat_frag(uint2 (&bf)[4][2], const __half *rows, int nv, int g, int t)
{
    const __half *feat = rows + g * P16_RS + 4 * t;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) bf[j][h] = 8 * j < nv ? *reinterpret_cast<const uint2 *>(feat + 8 * j * P16_RS + h * 16) : make_uint2(0, 0);
}

// One projection unit: the 16 rows of a table tile against 32 voxels, one product per slot and 8 voxels; d[row g / g + 8]
// [2t + e][j] = voxel 8j + 2t + e, both slots.  (Block-diagonal operands, as at head_dim 8, would take two products
// for four voxels: twice the tensor work, and a second rounding of the sum to fp16.)
__device__ __forceinline__ void p16_project(uint32_t (&d)[2][2][4], const P16TileA &a, const uint2 (&bf)[4][2], int nv)
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        d[0][0][j] = d[0][1][j] = d[1][0][j] = d[1][1][j] = 0u;
        if (8 * j < nv) {
            uint32_t x0, x1, y0, y1;
            mma_k16_h(x0, x1, a.f[0][0].x, a.f[0][1].x, a.f[0][0].y, a.f[0][1].y, bf[j][0].x, bf[j][0].y);
            mma_k16_h(y0, y1, a.f[1][0].x, a.f[1][1].x, a.f[1][0].y, a.f[1][1].y, bf[j][1].x, bf[j][1].y);
            d[0][0][j] = pack_lo(x0, y0);
            d[0][1][j] = pack_hi(x0, y0);
            d[1][0][j] = pack_lo(x1, y1);
            d[1][1][j] = pack_hi(x1, y1);
        }
    }
}

// Its stores.  Lane-major [row][qpos(voxel)]: voxels 8j + 2t + e, j = 0..3, are the four columns from 4 (2t + e) on; odd rows
// write e = 1 first, so that the eight lanes of a quarter warp (rows g, g + 1; t = 0..3) cover all 32 banks.
__device__ __forceinline__ void p16_store_lane_major(uint32_t *dst, const uint32_t (&d)[2][2][4], int mt, int g, int t)
{
    const bool od = g & 1;
    uint32_t *r = dst + (mt * 16 + g) * QT + 8 * t;
    const int o0 = od ? 4 : 0, o1 = 4 - o0;
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
        const uint4 a = make_uint4(d[rr][0][0], d[rr][0][1], d[rr][0][2], d[rr][0][3]), b = make_uint4(d[rr][1][0], d[rr][1][1], d[rr][1][2], d[rr][1][3]);
        *reinterpret_cast<uint4 *>(r + rr * 8 * QT + o0) = od ? b : a;
        *reinterpret_cast<uint4 *>(r + rr * 8 * QT + o1) = od ? a : b;
    }
}

// Key-major [voxel][Rp], the first nv voxels rounded up to a multiple of eight; Rp = 4 (mod 16): voxels 2t lie 8 banks apart.
__device__ __forceinline__ void p16_store_key_major(uint32_t *dst, const uint32_t (&d)[2][2][4], int mt, int Rp, int nv, int g, int t)
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (8 * j < nv) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t *p = dst + (8 * j + 2 * t + e) * Rp + mt * 16 + g;
                p[0] = d[0][e][j];
                p[8] = d[1][e][j];
            }
        }
}

// A 16 x 8 block of Y . X^T (both slots): c[row y0 + g / + 8][voxel x0 + 2t / + 1][slot].
__device__ __forceinline__ void p16_dot_block(float (&c)[2][2][2], const __half *Y, int y0, const __half *X, int x0, int g, int t)
{
    const __half *y = Y + (y0 + g) * P16_RS + 4 * t, *x = X + (x0 + g) * P16_RS + 4 * t;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint2 b = *reinterpret_cast<const uint2 *>(x + h * 16);
        const uint2 a0 = *reinterpret_cast<const uint2 *>(y + h * 16), a1 = *reinterpret_cast<const uint2 *>(y + 8 * P16_RS + h * 16);
        float d[4];
        mma_k16_z(d, a0.x, a1.x, a0.y, a1.y, b.x, b.y);
        c[0][0][h] = d[0]; c[0][1][h] = d[1]; c[1][0][h] = d[2]; c[1][1][h] = d[3];
    }
}

// acc += hist(16 rows of k-step ks) . T(the same rows) for the 32 voxels (m).
__device__ __forceinline__ void p16_hist_t(float (&acc)[2][2][2][4], const uint32_t *hist, const P16FragB &tb, int ks, int lane, int g, int t)
{
    uint4 y[4];
    load_hist_rows(y, hist, ks, lane, g, t);       // y[i] = row t + 4i, queries {g, g+8, g+16, g+24}
    const uint32_t a[2][2][4] = {{{pack_lo(y[0].x, y[1].x), pack_lo(y[0].y, y[1].y), pack_lo(y[2].x, y[3].x), pack_lo(y[2].y, y[3].y)},
                                  {pack_lo(y[0].z, y[1].z), pack_lo(y[0].w, y[1].w), pack_lo(y[2].z, y[3].z), pack_lo(y[2].w, y[3].w)}},
                                 {{pack_hi(y[0].x, y[1].x), pack_hi(y[0].y, y[1].y), pack_hi(y[2].x, y[3].x), pack_hi(y[2].y, y[3].y)},
                                  {pack_hi(y[0].z, y[1].z), pack_hi(y[0].w, y[1].w), pack_hi(y[2].z, y[3].z), pack_hi(y[2].w, y[3].w)}}};
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < 2; ++i) mma_f32(acc[h][p][i], a[h][i], tb.b[h][p][0], tb.b[h][p][1]);
}

}  // namespace tc
}  // namespace s3d
