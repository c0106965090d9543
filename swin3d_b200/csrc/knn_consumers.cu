// Consumers of the KNN result, fused so that the [Nq, K, C] gathered tensor is never materialised:
//
//  * inverse-distance interpolation (microsoft/Swin3D, Swin3D/modules/swin3d_layers.py:53-73):
//        w_i = 1/(dist_i + 1e-8),  w_i /= sum_j w_j,  out[q] = sum_i src_feat[idx[q,i]] * w_i
//    with the reference's operation order (weights in fp32, one rounded multiply and one rounded add
//    per neighbour; for fp16 features the running sum is rounded to fp16 after every neighbour, as
//    the reference's in-place `+=` on an fp16 tensor does).  Backward: scatter of dOut * w_i.
//  * neighbourhood max-pool (swin3d_layers.py:302-309): LayerNorm and the bias-free Linear act on
//    each gathered row separately, so they commute with the gather; what is left per query is
//    out[q][c] = max_i g[idx[q,i]][c] with g = linear(norm(src_feat)) evaluated once per SOURCE row.
//    The arg-max source row is kept for the backward scatter (first maximum wins, as MaxPool1d).
//
// Both forwards are row gathers bound by L2 and HBM: a block takes a tile of queries, works out their
// rows and weights once into shared memory, and its threads then run over (query, 16-byte piece), so
// that every lane carries data whatever C is.  (A warp per query with the lanes over the channels
// left 22 of 32 lanes idle at C = 80: 466 against 127 us for 1.6 M queries, fp16, K = 3.)
//
// Two backwards.  The scatter form adds into an fp32 array with reductions in L2 (red.global.add).  The
// gather form (workspace given) first turns idx around -- a counting sort of the Nq * K (query,
// neighbour) entries by source -- and then a thread per (source, 16-byte piece) sums its entries in
// registers: no fp32 array to clear, add into and convert, one store per result.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "scan.cuh"

namespace s3d {
namespace {

constexpr int KC_MAX_K = 64;
constexpr int KC_THREADS = 256;
constexpr int KC_TILE = 64;              // queries per block of the forwards

template <typename T> struct Vec;
template <> struct Vec<float> {
    static constexpr int N = 4;
    using Raw = float4;
    static __device__ __forceinline__ void unpack(const Raw &r, float (&f)[4]) { f[0] = r.x; f[1] = r.y; f[2] = r.z; f[3] = r.w; }
    static __device__ __forceinline__ Raw pack(const float (&f)[4]) { return make_float4(f[0], f[1], f[2], f[3]); }
};
template <> struct Vec<__half> {
    static constexpr int N = 8;
    using Raw = uint4;
    static __device__ __forceinline__ void unpack(const Raw &r, float (&f)[8])
    {
        const __half2 *h = reinterpret_cast<const __half2 *>(&r);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 v = __half22float2(h[i]);
            f[2 * i] = v.x;
            f[2 * i + 1] = v.y;
        }
    }
    static __device__ __forceinline__ Raw pack(const float (&f)[8])
    {
        Raw r;
        __half2 *h = reinterpret_cast<__half2 *>(&r);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
        return r;
    }
};

// Running sum of the reference: fp32 stays fp32, fp16 is rounded to fp16 after every neighbour.
template <typename T> __device__ __forceinline__ float round_acc(float x);
template <> __device__ __forceinline__ float round_acc<float>(float x) { return x; }
template <> __device__ __forceinline__ float round_acc<__half>(float x) { return __half2float(__float2half_rn(x)); }

// Normalised inverse-distance weights of one query, every lane computes the same values.
__device__ __forceinline__ void interp_weights(const float *dist, int K, float (&w)[KC_MAX_K])
{
    float norm = 0.f;
#pragma unroll 4
    for (int i = 0; i < K; ++i) {
        w[i] = __fdiv_rn(1.0f, __fadd_rn(dist[i], 1e-8f));
        norm = __fadd_rn(norm, w[i]);
    }
#pragma unroll 4
    for (int i = 0; i < K; ++i) w[i] = __fdiv_rn(w[i], norm);
}

template <typename T, int KT /*0: runtime K*/>
__global__ void __launch_bounds__(KC_THREADS)
knn_interp_fwd_kernel(const int32_t *__restrict__ idx, const float *__restrict__ dist, const T *__restrict__ src,
                      T *__restrict__ out, int64_t Nq, int Krt, int C)
{
    constexpr int VN = Vec<T>::N;
    using Raw = typename Vec<T>::Raw;
    extern __shared__ int2 s_iw[];                           // [KC_TILE][K] row, weight
    const int K = KT ? KT : Krt;
    const int CV = C / VN;   // C is a whole number of vectors (checked by the entry point)
    const int64_t q0 = (int64_t)blockIdx.x * KC_TILE;
    const int nq = (int)min((int64_t)KC_TILE, Nq - q0);
    if (threadIdx.x < nq) {
        const int64_t q = q0 + threadIdx.x;
        float norm = 0.f;
        int2 *e = s_iw + threadIdx.x * K;
#pragma unroll 4
        for (int i = 0; i < K; ++i) {
            const float w = __fdiv_rn(1.0f, __fadd_rn(__ldg(dist + q * K + i), 1e-8f));
            norm = __fadd_rn(norm, w);
            e[i] = make_int2(__ldg(idx + q * K + i), __float_as_int(w));
        }
#pragma unroll 4
        for (int i = 0; i < K; ++i) e[i].y = __float_as_int(__fdiv_rn(__int_as_float(e[i].y), norm));
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nq * CV; t += KC_THREADS) {
        const int ql = t / CV, cv = t - ql * CV;
        const int2 *e = s_iw + ql * K;
        float acc[VN];
#pragma unroll
        for (int j = 0; j < VN; ++j) acc[j] = 0.f;
#pragma unroll 4
        for (int i = 0; i < K; ++i) {
            const int2 iw = e[i];
            const float w = __int_as_float(iw.y);
            float f[VN];
            Vec<T>::unpack(__ldg(reinterpret_cast<const Raw *>(src + (int64_t)iw.x * C) + cv), f);
#pragma unroll
            for (int j = 0; j < VN; ++j) acc[j] = round_acc<T>(__fadd_rn(acc[j], __fmul_rn(f[j], w)));
        }
        reinterpret_cast<Raw *>(out + (q0 + ql) * C)[cv] = Vec<T>::pack(acc);
    }
}

template <typename T>
__global__ void __launch_bounds__(KC_THREADS)
knn_interp_bwd_kernel(const int32_t *__restrict__ idx, const float *__restrict__ dist, const T *__restrict__ dout,
                      float *__restrict__ dsrc, int64_t Nq, int K, int C)
{
    constexpr int VN = Vec<T>::N;
    using Raw = typename Vec<T>::Raw;
    const int lane = threadIdx.x & 31;
    const int64_t warp0 = (int64_t)blockIdx.x * (KC_THREADS / 32) + (threadIdx.x >> 5);
    const int64_t nwarp = (int64_t)gridDim.x * (KC_THREADS / 32);
    const int CV = C / VN;
    for (int64_t q = warp0; q < Nq; q += nwarp) {
        float w[KC_MAX_K];
        interp_weights(dist + q * K, K, w);
        for (int cv = lane; cv < CV; cv += 32) {
            float g[VN];
            Vec<T>::unpack(__ldg(reinterpret_cast<const Raw *>(dout + q * C) + cv), g);
            for (int i = 0; i < K; ++i) {
                float *dst = dsrc + (int64_t)__ldg(idx + q * K + i) * C + cv * VN;
#pragma unroll
                for (int j = 0; j < VN; j += 4)
                    atomicAdd(reinterpret_cast<float4 *>(dst + j),
                              make_float4(g[j] * w[i], g[j + 1] * w[i], g[j + 2] * w[i], g[j + 3] * w[i]));
            }
        }
    }
}

// A: what is kept of the arg-max, the source row (int32_t) or the position in the query's list (uint8_t).
template <typename T, typename A, int KT /*0: runtime K*/>
__global__ void __launch_bounds__(KC_THREADS)
knn_maxpool_fwd_kernel(const int32_t *__restrict__ idx, const T *__restrict__ g, T *__restrict__ out,
                       A *__restrict__ arg, int64_t Nq, int Krt, int C)
{
    constexpr int VN = Vec<T>::N;
    using Raw = typename Vec<T>::Raw;
    extern __shared__ int32_t s_id[];                        // [KC_TILE][K] (K <= KC_MAX_K; longer lists stay in global memory)
    const int K = KT ? KT : Krt;
    const int CV = C / VN;
    const int64_t q0 = (int64_t)blockIdx.x * KC_TILE;
    const int nq = (int)min((int64_t)KC_TILE, Nq - q0);
    const bool staged = KT || K <= KC_MAX_K;
    if (staged)
        for (int i = threadIdx.x; i < nq * K; i += KC_THREADS) s_id[i] = __ldg(idx + q0 * K + i);
    __syncthreads();
    for (int t = threadIdx.x; t < nq * CV; t += KC_THREADS) {
        const int ql = t / CV, cv = t - ql * CV;
        const int32_t *e = staged ? s_id + ql * K : idx + (q0 + ql) * K;
        float best[VN] = {};
        A who[VN] = {};
#pragma unroll 8
        for (int i = 0; i < K; ++i) {
            const int32_t s = e[i];
            float f[VN];
            Vec<T>::unpack(__ldg(reinterpret_cast<const Raw *>(g + (int64_t)s * C) + cv), f);
#pragma unroll
            for (int j = 0; j < VN; ++j)
                if (i == 0 || f[j] > best[j] || f[j] != f[j]) {   // first maximum wins; NaN propagates
                    best[j] = f[j];
                    who[j] = sizeof(A) == 1 ? (A)i : (A)s;
                }
        }
        reinterpret_cast<Raw *>(out + (q0 + ql) * C)[cv] = Vec<T>::pack(best);
        A *a = arg + (q0 + ql) * C + cv * VN;
#pragma unroll
        for (int j = 0; j < VN; j += 4) {
            if (sizeof(A) == 1) *reinterpret_cast<uchar4 *>(a + j) = make_uchar4(who[j], who[j + 1], who[j + 2], who[j + 3]);
            else *reinterpret_cast<int4 *>(a + j) = make_int4(who[j], who[j + 1], who[j + 2], who[j + 3]);
        }
    }
}

// ---- gather backward -----------------------------------------------------------------------------------
// Workspace: one counter per source (then the start of its entries), tile sums of their scan, the rank
// of every (query, neighbour) among the entries of its source, the entries, the lists of long rows.
//
// A thread sums the entries of a (source, piece) one after the other, which is right for the dozen that a source
// has as a rule and not for thousands (the padding of scenes with fewer than K sources all refers to row 0).  Rows
// of more than LONG_ROW entries go on a list instead; a block takes up to `chunk` of a row's entries, and the last
// block of a row adds the chunks up.  100 k queries, K = 3, 80 channels fp16, 2 k / 20 k / 100 k entries in one row, forward
// and backward: 409 / 3704 / 21414 us by one thread.
constexpr int LONG_ROW = 64;
struct LongRow {
    int source, chunks, first_sum, done;
};
struct Inverse {
    uint32_t *start, *tile, *rank;
    unsigned long long *listed;    // [2] long rows (low half) and chunks (high half) on the lists; sums taken; cleared
    int2 *entry, *chunk_of;        // chunk_of: (long row, chunk of it)
    LongRow *rows;
    float *sums;                   // of the chunks of rows that have several, C each; over rank, which is read no more
    int64_t cleared, total;
    int n_tiles, chunk;
};

Inverse inverse_layout(char *base, int64_t Ns, int64_t Nq, int K)
{
    Inverse v{};
    v.n_tiles = (int)((Ns + 1 + SCAN_TILE - 1) / SCAN_TILE);
    const int64_t n = Nq * K;
    int64_t off = 0;
    auto take = [&](int64_t bytes) { const int64_t o = off; off = (off + bytes + 255) / 256 * 256; return base + o; };
    v.listed = (unsigned long long *)take(16);
    v.start = (uint32_t *)take((int64_t)v.n_tiles * SCAN_TILE * 4);
    v.cleared = off;
    v.tile = (uint32_t *)take((int64_t)v.n_tiles * 4);
    v.rank = (uint32_t *)take(n * 4);
    v.entry = (int2 *)take(n * 8);
    v.rows = (LongRow *)take((n / LONG_ROW + 1) * (int64_t)sizeof(LongRow));
    v.chunk_of = (int2 *)take((n / LONG_ROW + n / 128 + 1) * 8);     // chunks hold 256 entries at least
    v.sums = (float *)v.rank;
    v.total = off;
    return v;
}

__global__ void __launch_bounds__(KC_THREADS)
inverse_count_kernel(const int32_t *__restrict__ idx, int64_t n, Inverse v)
{
    const int64_t e = (int64_t)blockIdx.x * KC_THREADS + threadIdx.x;
    if (e < n) v.rank[e] = atomicAdd(v.start + __ldg(idx + e), 1u);
}

// entries (query, weight)
__global__ void __launch_bounds__(KC_THREADS)
inverse_fill_weights_kernel(const int32_t *__restrict__ idx, const float *__restrict__ dist, int64_t Nq, int K, Inverse v)
{
    const int64_t q = (int64_t)blockIdx.x * KC_THREADS + threadIdx.x;
    if (q >= Nq) return;
    float norm = 0.f;
#pragma unroll 4
    for (int i = 0; i < K; ++i) norm = __fadd_rn(norm, __fdiv_rn(1.0f, __fadd_rn(__ldg(dist + q * K + i), 1e-8f)));
#pragma unroll 4
    for (int i = 0; i < K; ++i) {
        const float w = __fdiv_rn(__fdiv_rn(1.0f, __fadd_rn(__ldg(dist + q * K + i), 1e-8f)), norm);
        const int64_t e = q * K + i;
        v.entry[v.start[__ldg(idx + e)] + v.rank[e]] = make_int2((int)q, __float_as_int(w));
    }
}

// entries (query, position in its list)
__global__ void __launch_bounds__(KC_THREADS)
inverse_fill_slots_kernel(const int32_t *__restrict__ idx, int64_t n, int K, Inverse v)
{
    const int64_t e = (int64_t)blockIdx.x * KC_THREADS + threadIdx.x;
    if (e >= n) return;
    const int q = (int)((uint32_t)e / (uint32_t)K);
    v.entry[v.start[__ldg(idx + e)] + v.rank[e]] = make_int2(q, (int)(e - (int64_t)q * K));
}

// acc += w * dout[q] of an entry                         (SLOT: dout[q] where slot[q] is the entry's)
template <typename T, bool SLOT>
__device__ __forceinline__ void add_entry(float (&acc)[Vec<T>::N], int2 it, const T *__restrict__ dout, const uint8_t *__restrict__ slot, int C, int cv)
{
    constexpr int VN = Vec<T>::N;
    using Raw = typename Vec<T>::Raw;
    if (SLOT) {
        const uint8_t *sp = slot + (int64_t)it.x * C + cv * VN;
        uint32_t sl[VN / 4], any = 0;
        const uint32_t want = 0x01010101u * (uint32_t)it.y;
#pragma unroll
        for (int j = 0; j < VN / 4; ++j) {
            sl[j] = __vcmpeq4(__ldg(reinterpret_cast<const uint32_t *>(sp) + j), want);
            any |= sl[j];
        }
        if (any) {
            float g[VN];
            Vec<T>::unpack(__ldg(reinterpret_cast<const Raw *>(dout + (int64_t)it.x * C) + cv), g);
#pragma unroll
            for (int j = 0; j < VN; ++j) acc[j] += (sl[j / 4] >> (8 * (j & 3))) & 1u ? g[j] : 0.f;
        }
    } else {
        float g[VN];
        Vec<T>::unpack(__ldg(reinterpret_cast<const Raw *>(dout + (int64_t)it.x * C) + cv), g);
        const float w = __int_as_float(it.y);
#pragma unroll
        for (int j = 0; j < VN; ++j) acc[j] = fmaf(g[j], w, acc[j]);
    }
}

// dsrc[s] = sum over the entries of s of w * dout[q]          (SLOT: of dout[q] where slot[q] is the entry's)
template <typename T, bool SLOT>
__global__ void __launch_bounds__(KC_THREADS)
inverse_gather_kernel(const T *__restrict__ dout, const uint8_t *__restrict__ slot, T *__restrict__ dsrc, int64_t Ns, int C, Inverse v)
{
    constexpr int VN = Vec<T>::N;
    using Raw = typename Vec<T>::Raw;
    const int CV = C / VN;
    const int64_t t = (int64_t)blockIdx.x * KC_THREADS + threadIdx.x;
    const int64_t s = t / CV;
    if (s >= Ns) return;
    const int cv = (int)(t - s * CV);
    const uint32_t e0 = __ldg(v.start + s), e1 = __ldg(v.start + s + 1);
    if (e1 - e0 > LONG_ROW) {
        if (cv == 0) {
            const int chunks = (int)((e1 - e0 + v.chunk - 1) / v.chunk);
            const unsigned long long at = atomicAdd(v.listed, ((unsigned long long)chunks << 32) | 1ull);
            const int row = (int)(uint32_t)at, first = (int)(at >> 32);
            v.rows[row] = LongRow{(int)s, chunks, chunks > 1 ? (int)atomicAdd(v.listed + 1, (unsigned long long)chunks) : 0, 0};
            for (int k = 0; k < chunks; ++k) v.chunk_of[first + k] = make_int2(row, k);
        }
        return;
    }
    float acc[VN];
#pragma unroll
    for (int j = 0; j < VN; ++j) acc[j] = 0.f;
#pragma unroll 4
    for (uint32_t e = e0; e < e1; ++e) add_entry<T, SLOT>(acc, __ldg(v.entry + e), dout, slot, C, cv);
    reinterpret_cast<Raw *>(dsrc + s * C)[cv] = Vec<T>::pack(acc);
}

// The rows on the list: a block per chunk of a row's entries, groups of threads with a piece per thread.
template <typename T, bool SLOT>
__global__ void __launch_bounds__(KC_THREADS)
inverse_long_rows_kernel(const T *__restrict__ dout, const uint8_t *__restrict__ slot, T *__restrict__ dsrc, int C, Inverse v)
{
    constexpr int VN = Vec<T>::N;
    using Raw = typename Vec<T>::Raw;
    __shared__ float s_acc[KC_THREADS][VN];
    __shared__ int s_last;
    const int n_chunks = (int)(*v.listed >> 32);
    const int CV = C / VN, wide = CV < KC_THREADS ? CV : KC_THREADS, groups = KC_THREADS / wide;
    const int grp = threadIdx.x / wide, piece = threadIdx.x - grp * wide;
    for (int c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const int2 of = v.chunk_of[c];
        LongRow *row = v.rows + of.x;
        const uint32_t end = __ldg(v.start + row->source + 1), e0 = __ldg(v.start + row->source) + (uint32_t)of.y * v.chunk;
        const uint32_t e1 = min(end, e0 + v.chunk);
        const bool alone = row->chunks == 1;
        for (int cv = piece; cv - piece < CV; cv += wide) {      // the same number of rounds for every thread
            float acc[VN];
#pragma unroll
            for (int j = 0; j < VN; ++j) acc[j] = 0.f;
            if (grp < groups && cv < CV)
#pragma unroll 4
                for (uint32_t e = e0 + grp; e < e1; e += groups) add_entry<T, SLOT>(acc, __ldg(v.entry + e), dout, slot, C, cv);
#pragma unroll
            for (int j = 0; j < VN; ++j) s_acc[threadIdx.x][j] = acc[j];
            __syncthreads();
            if (grp == 0 && cv < CV) {
                for (int g = 1; g < groups; ++g)
#pragma unroll
                    for (int j = 0; j < VN; ++j) acc[j] += s_acc[g * wide + piece][j];
                if (alone) reinterpret_cast<Raw *>(dsrc + (int64_t)row->source * C)[cv] = Vec<T>::pack(acc);
                else
#pragma unroll
                    for (int j = 0; j < VN; ++j) v.sums[(int64_t)(row->first_sum + of.y) * C + cv * VN + j] = acc[j];
            }
            __syncthreads();
        }
        if (alone) continue;
        // the block that finishes a row's last chunk adds them up
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(&row->done, 1) == row->chunks - 1;
        __syncthreads();
        if (s_last) {
            __threadfence();
            const float *sums = v.sums + (int64_t)row->first_sum * C;
            for (int cv = threadIdx.x; cv < CV; cv += KC_THREADS) {
                float acc[VN];
#pragma unroll
                for (int j = 0; j < VN; ++j) acc[j] = 0.f;
#pragma unroll 4
                for (int k = 0; k < row->chunks; ++k)
#pragma unroll
                    for (int j = 0; j < VN; ++j) acc[j] += __ldcg(sums + (int64_t)k * C + cv * VN + j);
                reinterpret_cast<Raw *>(dsrc + (int64_t)row->source * C)[cv] = Vec<T>::pack(acc);
            }
        }
        __syncthreads();
    }
}

template <typename T>
__global__ void __launch_bounds__(KC_THREADS)
knn_maxpool_bwd_kernel(const int32_t *__restrict__ arg, const T *__restrict__ dout, float *__restrict__ dg,
                       int64_t total, int C)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
        const int c = (int)(e % C);
        atomicAdd(dg + (int64_t)__ldg(arg + e) * C + c, (float)dout[e]);
    }
}

int grid_for(int64_t warps_needed)
{
    static int sms_of[64] = {0};
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
        if (!sms_of[dev] && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) sms_of[dev] = sms;
        if (sms_of[dev]) sms = sms_of[dev];
    }
    const int64_t blocks = (warps_needed + KC_THREADS / 32 - 1) / (KC_THREADS / 32);
    const int64_t cap = (int64_t)sms * 8;     // 8 resident blocks of 256 threads per SM
    return (int)(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

unsigned blocks_of(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

template <typename T>
void launch_interp_fwd(const int32_t *idx, const float *dist, const void *src, void *out, int64_t Nq, int K, int C, cudaStream_t st)
{
    const unsigned grid = blocks_of(Nq, KC_TILE);
    const size_t smem = (size_t)KC_TILE * K * sizeof(int2);
    if (K == 3) knn_interp_fwd_kernel<T, 3><<<grid, KC_THREADS, smem, st>>>(idx, dist, (const T *)src, (T *)out, Nq, K, C);
    else knn_interp_fwd_kernel<T, 0><<<grid, KC_THREADS, smem, st>>>(idx, dist, (const T *)src, (T *)out, Nq, K, C);
}

template <typename T, typename A>
void launch_maxpool_fwd(const int32_t *idx, const void *g, void *out, A *arg, int64_t Nq, int K, int C, cudaStream_t st)
{
    const unsigned grid = blocks_of(Nq, KC_TILE);
    const size_t smem = K <= KC_MAX_K ? (size_t)KC_TILE * K * sizeof(int32_t) : 0;
    if (K == 16) knn_maxpool_fwd_kernel<T, A, 16><<<grid, KC_THREADS, smem, st>>>(idx, (const T *)g, (T *)out, arg, Nq, K, C);
    else knn_maxpool_fwd_kernel<T, A, 0><<<grid, KC_THREADS, smem, st>>>(idx, (const T *)g, (T *)out, arg, Nq, K, C);
}

template <typename T, bool SLOT>
void launch_gather_as(const uint8_t *slot, const void *dout, void *dsrc, int64_t Ns, int64_t n, int C, const Inverse &v, cudaStream_t st)
{
    inverse_gather_kernel<T, SLOT><<<blocks_of(Ns * (C / Vec<T>::N), KC_THREADS), KC_THREADS, 0, st>>>((const T *)dout, slot, (T *)dsrc, Ns, C, v);
    if (n > LONG_ROW) {
        const int64_t most = n / LONG_ROW + 1;
        inverse_long_rows_kernel<T, SLOT><<<(unsigned)(most < 148 * 4 ? most : 148 * 4), KC_THREADS, 0, st>>>((const T *)dout, slot, (T *)dsrc, C, v);
    }
}

template <typename T>
void launch_gather(const uint8_t *slot, const void *dout, void *dsrc, int64_t Ns, int64_t n, int C, const Inverse &v, cudaStream_t st)
{
    if (slot) launch_gather_as<T, true>(slot, dout, dsrc, Ns, n, C, v, st);
    else launch_gather_as<T, false>(nullptr, dout, dsrc, Ns, n, C, v, st);
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int last_status() { return cudaGetLastError() == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH; }

}  // namespace
}  // namespace s3d

using namespace s3d;

extern "C" int s3d_knn_interpolate_fwd(const int32_t *idx, const float *dist, const void *src_feat, void *out,
                                       int64_t Nq, int K, int C, int dtype, void *stream)
{
    if (Nq < 0 || K < 1 || K > KC_MAX_K || C < 1 || (dtype != S3D_F32 && dtype != S3D_F16)) return S3D_ERR_BAD_ARG;
    if (Nq == 0) return S3D_OK;
    if (!idx || !dist || !src_feat || !out) return S3D_ERR_BAD_ARG;
    const int vn = dtype == S3D_F32 ? 4 : 8;
    if (C % vn != 0 || !aligned16(src_feat) || !aligned16(out)) return S3D_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == S3D_F32) launch_interp_fwd<float>(idx, dist, src_feat, out, Nq, K, C, st);
    else launch_interp_fwd<__half>(idx, dist, src_feat, out, Nq, K, C, st);
    return last_status();
}

extern "C" int s3d_knn_interpolate_bwd(const int32_t *idx, const float *dist, const void *dout, float *dsrc,
                                       int64_t Nq, int64_t Ns, int K, int C, int dtype, void *stream)
{
    if (Nq < 0 || Ns < 0 || K < 1 || K > KC_MAX_K || C < 1 || (dtype != S3D_F32 && dtype != S3D_F16)) return S3D_ERR_BAD_ARG;
    if (Ns == 0) return S3D_OK;
    if (!dsrc) return S3D_ERR_BAD_ARG;
    const int vn = dtype == S3D_F32 ? 4 : 8;
    if (C % vn != 0 || !aligned16(dout) || !aligned16(dsrc)) return S3D_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(dsrc, 0, (size_t)Ns * C * sizeof(float), st) != cudaSuccess) return S3D_ERR_LAUNCH;
    if (Nq == 0) return S3D_OK;
    if (!idx || !dist || !dout) return S3D_ERR_BAD_ARG;
    const int grid = grid_for(Nq);
    if (dtype == S3D_F32)
        knn_interp_bwd_kernel<float><<<grid, KC_THREADS, 0, st>>>(idx, dist, (const float *)dout, dsrc, Nq, K, C);
    else
        knn_interp_bwd_kernel<__half><<<grid, KC_THREADS, 0, st>>>(idx, dist, (const __half *)dout, dsrc, Nq, K, C);
    return last_status();
}

extern "C" int s3d_knn_maxpool_fwd(const int32_t *idx, const void *g, void *out, int32_t *arg,
                                   int64_t Nq, int K, int C, int dtype, void *stream)
{
    if (Nq < 0 || K < 1 || C < 1 || (dtype != S3D_F32 && dtype != S3D_F16)) return S3D_ERR_BAD_ARG;
    if (Nq == 0) return S3D_OK;
    if (!idx || !g || !out || !arg) return S3D_ERR_BAD_ARG;
    const int vn = dtype == S3D_F32 ? 4 : 8;
    if (C % vn != 0 || !aligned16(g) || !aligned16(out) || !aligned16(arg)) return S3D_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == S3D_F32) launch_maxpool_fwd<float>(idx, g, out, arg, Nq, K, C, st);
    else launch_maxpool_fwd<__half>(idx, g, out, arg, Nq, K, C, st);
    return last_status();
}

extern "C" int s3d_knn_maxpool_bwd(const int32_t *arg, const void *dout, float *dg,
                                   int64_t Nq, int64_t Ns, int C, int dtype, void *stream)
{
    if (Nq < 0 || Ns < 0 || C < 1 || (dtype != S3D_F32 && dtype != S3D_F16)) return S3D_ERR_BAD_ARG;
    if (Ns == 0) return S3D_OK;
    if (!dg) return S3D_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(dg, 0, (size_t)Ns * C * sizeof(float), st) != cudaSuccess) return S3D_ERR_LAUNCH;
    if (Nq == 0) return S3D_OK;
    if (!arg || !dout) return S3D_ERR_BAD_ARG;
    const int64_t total = Nq * C;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t want = (total + KC_THREADS - 1) / KC_THREADS;
    const int grid = (int)(want < (int64_t)sms * 8 ? want : (int64_t)sms * 8);
    if (dtype == S3D_F32)
        knn_maxpool_bwd_kernel<float><<<grid, KC_THREADS, 0, st>>>(arg, (const float *)dout, dg, total, C);
    else
        knn_maxpool_bwd_kernel<__half><<<grid, KC_THREADS, 0, st>>>(arg, (const __half *)dout, dg, total, C);
    return last_status();
}

extern "C" int s3d_knn_maxpool_slots_fwd(const int32_t *idx, const void *g, void *out, uint8_t *slot,
                                         int64_t Nq, int K, int C, int dtype, void *stream)
{
    if (Nq < 0 || K < 1 || K > KC_MAX_K || C < 1 || (dtype != S3D_F32 && dtype != S3D_F16)) return S3D_ERR_BAD_ARG;
    if (Nq == 0) return S3D_OK;
    if (!idx || !g || !out || !slot) return S3D_ERR_BAD_ARG;
    const int vn = dtype == S3D_F32 ? 4 : 8;
    if (C % vn != 0 || !aligned16(g) || !aligned16(out) || !aligned16(slot)) return S3D_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == S3D_F32) launch_maxpool_fwd<float>(idx, g, out, slot, Nq, K, C, st);
    else launch_maxpool_fwd<__half>(idx, g, out, slot, Nq, K, C, st);
    return last_status();
}

extern "C" int64_t s3d_knn_gather_workspace_bytes(int64_t Ns, int64_t Nq, int K)
{
    if (Ns < 1 || Nq < 1 || K < 1 || Nq * K >= (int64_t)1 << 31) return 0;
    return inverse_layout(nullptr, Ns, Nq, K).total;
}

static int gather_impl(const int32_t *idx, const float *dist, const uint8_t *slot, const void *dout, void *dsrc,
                       int64_t Nq, int64_t Ns, int K, int C, int dtype, void *workspace, int64_t workspace_bytes, void *stream)
{
    if (Nq < 0 || Ns < 0 || K < 1 || K > KC_MAX_K || C < 1 || (dtype != S3D_F32 && dtype != S3D_F16)) return S3D_ERR_BAD_ARG;
    if (Ns == 0) return S3D_OK;
    if (!dsrc) return S3D_ERR_BAD_ARG;
    const int vn = dtype == S3D_F32 ? 4 : 8;
    if (C % vn != 0 || !aligned16(dout) || !aligned16(dsrc)) return S3D_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    if (Nq == 0) return cudaMemsetAsync(dsrc, 0, (size_t)Ns * C * (dtype == S3D_F32 ? 4 : 2), st) == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
    if (!idx || (!dist && !slot) || !dout || !workspace) return S3D_ERR_BAD_ARG;
    if (Nq * K >= (int64_t)1 << 31) return S3D_ERR_UNSUPPORTED;
    Inverse v = inverse_layout((char *)workspace, Ns, Nq, K);
    v.chunk = 2 * C > 256 ? 2 * C : 256;                      // at most 2 n / chunk chunks share a row: their sums find room in rank
    if (workspace_bytes < v.total) return S3D_ERR_WORKSPACE;
    if (cudaMemsetAsync(v.listed, 0, (size_t)v.cleared, st) != cudaSuccess) return S3D_ERR_LAUNCH;
    const int64_t n = Nq * K;
    inverse_count_kernel<<<blocks_of(n, KC_THREADS), KC_THREADS, 0, st>>>(idx, n, v);
    scan_in_place(v.start, v.tile, v.n_tiles, st);
    if (slot) inverse_fill_slots_kernel<<<blocks_of(n, KC_THREADS), KC_THREADS, 0, st>>>(idx, n, K, v);
    else inverse_fill_weights_kernel<<<blocks_of(Nq, KC_THREADS), KC_THREADS, 0, st>>>(idx, dist, Nq, K, v);
    if (dtype == S3D_F32) launch_gather<float>(slot, dout, dsrc, Ns, n, C, v, st);
    else launch_gather<__half>(slot, dout, dsrc, Ns, n, C, v, st);
    return last_status();
}

extern "C" int s3d_knn_interpolate_gather_bwd(const int32_t *idx, const float *dist, const void *dout, void *dsrc,
                                              int64_t Nq, int64_t Ns, int K, int C, int dtype, void *workspace,
                                              int64_t workspace_bytes, void *stream)
{
    return gather_impl(idx, dist, nullptr, dout, dsrc, Nq, Ns, K, C, dtype, workspace, workspace_bytes, stream);
}

extern "C" int s3d_knn_maxpool_slots_bwd(const int32_t *idx, const uint8_t *slot, const void *dout, void *dg,
                                         int64_t Nq, int64_t Ns, int K, int C, int dtype, void *workspace,
                                         int64_t workspace_bytes, void *stream)
{
    return gather_impl(idx, nullptr, slot, dout, dg, Nq, Ns, K, C, dtype, workspace, workspace_bytes, stream);
}
