// K-nearest-neighbour search over a spatial index (K <= 16), with the results of the brute-force scan
// in knn.cu, bit for bit.
//
// Both point sets are put into Morton order of a per-scene grid by a counting sort (histogram, scan,
// scatter).  32 consecutive sources are a leaf and 32 leaves a node, each with its bounding box.
// A warp searches for 32 consecutive queries (K > 3: 16, two lanes each), which lie close together:
// the lanes test the boxes of 32 nodes or leaves at a time against the box of the warp's queries, nearest
// first, and a leaf that survives is offered to all its queries with broadcast loads.
//
// Why the results are the same.  (1) The K smallest distances of a query do not depend on the order
// of the scan, and neither do their indices as long as no two candidates at or below the K-th distance
// are equal.  The search sees every candidate whose distance can be <= the K-th: the distance of a
// point from a box is evaluated with the reference's own expression on the per-axis gaps, and
// since every rounded operation of it is monotone in the magnitude of each difference, the bound is
// never above the computed distance of a point inside the box.  (2) When distances do tie -- two of
// the K are equal, or the smallest excluded one equals the K-th -- the reference's answer depends on
// the history of its heap.  The search notices that (it keeps the smallest excluded distance) and puts
// the query on a list; those queries are scanned again in index order with the literal heap.
//
// Bound: instruction issue of the leaf evaluation for K = 3, the merges of the lists and their latency for
// K = 16.  Measured, whole search: 8 scenes x (200 k queries, 50 k sources), K = 3: 0.42 ms, the scan of knn.cu
// 16.9; 4 x (30 k, 120 k), K = 16: 0.37 ms (the scan: 62).
#include <climits>

#include "knn_common.cuh"
#include "knn_kernels.cuh"
#include "scan.cuh"

namespace s3d {
namespace {

constexpr int LEAF = 32;
constexpr int KT_THREADS = 256;
constexpr int SEARCH_THREADS = 128;

struct TreeBufs {
    uint32_t *zero;          // cleared by the launch: bbox, tie counter, then the two cell histograms
    uint32_t *bbox;          // [B][8] order-preserving keys of -min (0..2) and max (4..6)
    int *tie_count;
    uint32_t *hist;          // [2][B * cells]: sources, queries; after the scan the start of every cell
    uint32_t *tile;          // sums of SCAN_TILE cells
    uint32_t *rank;          // [Ns + Nq] position of a point inside its cell
    float *src;              // [leaves][4][32] x, y, z, row number of the sources in cell order, a leaf at a time
    float4 *qry;             // [Nq] x, y, z, row number of the queries in cell order
    float4 *leaf;            // [leaves][2] lowest and highest corner
    float4 *node;            // [nodes][2]
    int32_t *ties;           // [Nq] queries to scan again
    int64_t zero_bytes, total;
    int bits, n_tiles;
};

// Cells per axis: 2^bits.  A leaf should hold a few cells of a surface (4^bits cells or so of a scene are
// occupied); the histograms of all scenes stay below 2^21 cells each so that clearing and scanning
// them costs a few microseconds.
int tree_bits(int B, int64_t Ns)
{
    const int64_t per = Ns / B;
    int bits = per > 65536 ? 7 : (per > 8192 ? 6 : (per > 2048 ? 5 : 4));
    while (bits > 1 && ((int64_t)B << (3 * bits)) > (1 << 21)) --bits;
    return bits;
}

int64_t up(int64_t x) { return (x + 255) / 256 * 256; }

TreeBufs tree_bufs(char *base, int B, int64_t Ns, int64_t Nq)
{
    TreeBufs t{};
    t.bits = tree_bits(B, Ns);
    const int64_t cells = (int64_t)B << (3 * t.bits);
    t.n_tiles = (int)((2 * cells + SCAN_TILE - 1) / SCAN_TILE);
    int64_t off = 0;
    auto take = [&](int64_t bytes) { const int64_t o = off; off = up(off + bytes); return base + o; };
    t.zero = (uint32_t *)take(0);
    t.bbox = (uint32_t *)take((int64_t)B * 32 + 4);
    t.tie_count = (int *)(t.bbox + (int64_t)B * 8);
    t.hist = (uint32_t *)take((int64_t)t.n_tiles * SCAN_TILE * 4);
    t.zero_bytes = off;
    t.tile = (uint32_t *)take((int64_t)t.n_tiles * 4);
    t.rank = (uint32_t *)take((Ns + Nq) * 4);
    t.src = (float *)take((Ns / LEAF + B + 1) * LEAF * 16);
    t.qry = (float4 *)take(Nq * 16);
    t.leaf = (float4 *)take((Ns / LEAF + B + 1) * 32);
    t.node = (float4 *)take((Ns / (LEAF * 32) + B + 1) * 32);
    t.ties = (int32_t *)take(Nq * 4);
    t.total = off;
    return t;
}

// Order-preserving unsigned key of a finite float; 0 stays free for "nothing yet".
__device__ __forceinline__ uint32_t order_key(float x)
{
    const uint32_t u = __float_as_uint(x);
    return (u >> 31) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_order_key(uint32_t k)
{
    return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ bool finite3(float x, float y, float z)
{
    return fabsf(x) < INFINITY && fabsf(y) < INFINITY && fabsf(z) < INFINITY;
}

// Box of a scene's finite points (sources and queries).  grid = (x, B)
__global__ void __launch_bounds__(KT_THREADS)
tree_bbox_kernel(const float *__restrict__ src, const float *__restrict__ query, const int32_t *__restrict__ so,
                 const int32_t *__restrict__ qo, int B, int64_t Nq, uint32_t *__restrict__ bbox)
{
    const int b = blockIdx.y;
    const int64_t s0 = b > 0 ? __ldg(so + b - 1) : 0, s1 = __ldg(so + b);
    const int64_t q0 = b > 0 ? max(__ldg(qo + b - 1), 0) : 0;
    const int64_t q1 = b == B - 1 ? Nq : min((int64_t)__ldg(qo + b), Nq);
    uint32_t k[6] = {0, 0, 0, 0, 0, 0};
    auto see = [&](const float *p) {
        const float x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
        if (finite3(x, y, z)) {
            k[0] = max(k[0], order_key(-x)); k[1] = max(k[1], order_key(-y)); k[2] = max(k[2], order_key(-z));
            k[3] = max(k[3], order_key(x)); k[4] = max(k[4], order_key(y)); k[5] = max(k[5], order_key(z));
        }
    };
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = s0 + first; i < s1; i += step) see(src + i * 3);
    for (int64_t i = q0 + first; i < q1; i += step) see(query + i * 3);
    __shared__ uint32_t s_k[6];
    if (threadIdx.x < 6) s_k[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const uint32_t m = __reduce_max_sync(0xffffffffu, k[i]);
        if ((threadIdx.x & 31) == 0 && m) atomicMax(s_k + i, m);
    }
    __syncthreads();
    if (threadIdx.x < 6 && s_k[threadIdx.x]) atomicMax(bbox + b * 8 + (threadIdx.x < 3 ? threadIdx.x : threadIdx.x + 1), s_k[threadIdx.x]);
}

__device__ __forceinline__ uint32_t spread3(uint32_t v)      // bit i of v -> bit 3i (v < 256)
{
    v = (v | (v << 8)) & 0x00f00fu;
    v = (v | (v << 4)) & 0x0c30c3u;
    return (v | (v << 2)) & 0x249249u;
}

// Morton number of a point's cell in the cubic grid over its scene's box.
__device__ __forceinline__ uint32_t cell_of(float x, float y, float z, const uint32_t *__restrict__ bbox, int b, int bits)
{
    const uint4 lo = __ldg(reinterpret_cast<const uint4 *>(bbox + b * 8)), hi = __ldg(reinterpret_cast<const uint4 *>(bbox + b * 8 + 4));
    if (!lo.x) return 0;                                     // no finite point in the scene
    const float lx = -from_order_key(lo.x), ly = -from_order_key(lo.y), lz = -from_order_key(lo.z);
    const float ext = fmaxf(from_order_key(hi.x) - lx, fmaxf(from_order_key(hi.y) - ly, from_order_key(hi.z) - lz));
    const float n = (float)(1 << bits), inv = ext > 0.f ? n / ext : 0.f, top = n - 1.f;
    auto axis = [&](float v) { return v > 0.f ? (uint32_t)fminf(v, top) : 0u; };   // NaN -> 0
    return spread3(axis((x - lx) * inv)) | (spread3(axis((y - ly) * inv)) << 1) | (spread3(axis((z - lz) * inv)) << 2);
}

// Leaves and nodes of scene b, whose sources start at s0, start at these places of their arrays, which
// leaves room for the partial last one of every scene.
__device__ __forceinline__ int64_t first_leaf(int64_t s0, int b) { return s0 / LEAF + b; }
__device__ __forceinline__ int64_t first_node(int64_t s0, int b) { return s0 / (LEAF * 32) + b; }

// One point per thread, sources then queries.  COUNT: rank inside the cell; otherwise: into cell order.
template <bool COUNT>
__global__ void __launch_bounds__(KT_THREADS)
tree_sort_kernel(const float *__restrict__ src, const float *__restrict__ query, const int32_t *__restrict__ so,
                 const int32_t *__restrict__ qo, int B, int64_t Ns, int64_t Nq, TreeBufs t)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Ns + Nq) return;
    const bool is_q = i >= Ns;
    const int64_t g = is_q ? i - Ns : i;
    const int32_t *off = is_q ? qo : so;
    int b = 0;
    for (; b < B; ++b)
        if (g < __ldg(off + b)) break;
    if (b >= B) {
        if (!is_q) return;                                   // a source beyond the last scene belongs to none
        b = B - 1;
    }
    const float *p = (is_q ? query : src) + g * 3;
    const float x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
    const int64_t cells = (int64_t)B << (3 * t.bits);
    uint32_t *h = t.hist + (is_q ? cells : 0) + ((int64_t)b << (3 * t.bits)) + cell_of(x, y, z, t.bbox, b, t.bits);
    if (COUNT) {
        t.rank[i] = atomicAdd(h, 1u);
        return;
    }
    const uint32_t at = *h + t.rank[i];
    if (is_q) {
        t.qry[at - t.hist[cells]] = make_float4(x, y, z, __int_as_float((int)g));   // the first query cell follows the last source
    } else {
        const uint32_t s0 = t.hist[(int64_t)b << (3 * t.bits)];
        float *o = t.src + (first_leaf(s0, b) + (at - s0) / LEAF) * (4 * LEAF) + (at - s0) % LEAF;
        o[0] = x; o[LEAF] = y; o[2 * LEAF] = z; o[3 * LEAF] = __int_as_float((int)g);
    }
}

// Boxes: a warp makes a leaf, a block (32 warps) a node.  grid = nodes of all scenes, in scene order.
// The places of a partial leaf that hold no source get NaN coordinates, which no comparison lets in.
__global__ void __launch_bounds__(1024)
tree_boxes_kernel(int B, TreeBufs t)
{
    __shared__ float s_lo[3][32], s_hi[3][32];
    int j = blockIdx.x, b = 0;
    int s0 = 0, n = 0;
    for (; b < B; ++b) {
        const int e = (int)__ldg(t.hist + ((int64_t)(b + 1) << (3 * t.bits)));
        n = e - s0;
        const int nodes = (n + LEAF * 32 - 1) / (LEAF * 32);
        if (j < nodes) break;
        j -= nodes;
        s0 = e;
    }
    if (b >= B) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int leaf = j * 32 + wid, at = leaf * LEAF + lane;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    float *p = t.src + (first_leaf(s0, b) + leaf) * (4 * LEAF) + lane;
    if (at < n) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {                        // a NaN never counts
            lo[d] = fminf(lo[d], p[d * LEAF]);
            hi[d] = fmaxf(hi[d], p[d * LEAF]);
        }
    } else if (leaf * LEAF < n) {
        p[0] = p[LEAF] = p[2 * LEAF] = NAN;
    }
    auto reduce = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
    };
    reduce();
    if (lane == 0) {
        if (leaf * LEAF < n) {
            float4 *o = t.leaf + 2 * (first_leaf(s0, b) + leaf);
            o[0] = make_float4(lo[0], lo[1], lo[2], 0.f);
            o[1] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) { s_lo[d][wid] = lo[d]; s_hi[d][wid] = hi[d]; }
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) { lo[d] = s_lo[d][lane]; hi[d] = s_hi[d][lane]; }
        reduce();
        if (lane == 0) {
            float4 *o = t.node + 2 * (first_node(s0, b) + j);
            o[0] = make_float4(lo[0], lo[1], lo[2], 0.f);
            o[1] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
    }
}

// A lower bound of the reference's distance between any point of box [lo, hi] and any query of box
// [ql, qh]: its expression on the gaps (see the head of the file).
__device__ __forceinline__ float box_gap(float lo, float hi, float ql, float qh)
{
    return fmaxf(fmaxf(lo - qh, ql - hi), 0.f);
}
__device__ __forceinline__ float box_dist(const float4 &lo, const float4 &hi, const float (&ql)[3], const float (&qh)[3])
{
    return knn_dist2(box_gap(lo.x, hi.x, ql[0], qh[0]), box_gap(lo.y, hi.y, ql[1], qh[1]), box_gap(lo.z, hi.z, ql[2], qh[2]));
}

// Two candidates per instruction (element 0 in the low half).  The packed operations round each half as
// the scalar ones do, so the distances are those of knn_dist2 bit for bit.
__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void dist2x2(float &d0, float &d1, uint64_t px, uint64_t py, uint64_t pz, uint64_t nx, uint64_t ny, uint64_t nz)
{
    asm("{\n\t.reg .b64 x, y, z;\n\t"
        "add.rn.f32x2 x, %2, %5;\n\t"
        "add.rn.f32x2 y, %3, %6;\n\t"
        "add.rn.f32x2 z, %4, %7;\n\t"
        "mul.rn.f32x2 y, y, y;\n\t"
        "fma.rn.f32x2 y, x, x, y;\n\t"
        "fma.rn.f32x2 y, z, z, y;\n\t"
        "mov.b64 {%0, %1}, y;\n\t}"
        : "=f"(d0), "=f"(d1) : "l"(px), "l"(py), "l"(pz), "l"(nx), "l"(ny), "l"(nz));
}

// The KL smallest distances of a query, ascending, in registers; the first KL - K entries are -1 when
// K < KL.  ex = smallest distance that was offered and is not among them.
template <int KL>
struct TopK {
    float d[KL];
    int i[KL];
    float ex;
    __device__ __forceinline__ void init(int K)
    {
#pragma unroll
        for (int j = 0; j < KL; ++j) {
            d[j] = j < KL - K ? -1.f : KNN_FAR;
            i[j] = 0;
        }
        ex = INFINITY;
    }
    __device__ __forceinline__ float top() const { return d[KL - 1]; }
    // x < top()
    __device__ __forceinline__ void insert(float x, int id)
    {
        ex = fminf(ex, d[KL - 1]);
#pragma unroll
        for (int j = KL - 1; j > 0; --j) {
            const bool below = x < d[j - 1], here = x < d[j];
            d[j] = below ? d[j - 1] : (here ? x : d[j]);
            i[j] = below ? i[j - 1] : (here ? id : i[j]);
        }
        if (x < d[0]) { d[0] = x; i[0] = id; }
    }
    // the eight candidates (x, id), unsorted, INFINITY where there is none: sort them, keep the KL smallest of
    // both lists (a bitonic sequence), sort that
    __device__ __forceinline__ void merge8(float (&x)[8], int (&id)[8])
    {
        static_assert(KL == 8 || KL == 16, "a power of two");
        constexpr int net[19][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3}, {4, 6}, {5, 7}, {1, 2}, {5, 6},
                                    {0, 4}, {1, 5}, {2, 6}, {3, 7}, {2, 4}, {3, 5}, {1, 2}, {3, 4}, {5, 6}};
#pragma unroll
        for (int k = 0; k < 19; ++k) order(x[net[k][0]], x[net[k][1]], id[net[k][0]], id[net[k][1]]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            order(d[KL - 1 - j], x[j], i[KL - 1 - j], id[j]);
            ex = fminf(ex, x[j]);
        }
        sort_bitonic();
    }
    // the KL smallest of this lane's list and that of lane ^ h, in both lanes
    __device__ __forceinline__ void merge_lane(int h)
    {
        float od[KL];
        int oi[KL];
#pragma unroll
        for (int j = 0; j < KL; ++j) {
            od[j] = __shfl_xor_sync(0xffffffffu, d[KL - 1 - j], h);
            oi[j] = __shfl_xor_sync(0xffffffffu, i[KL - 1 - j], h);
        }
        ex = fminf(ex, __shfl_xor_sync(0xffffffffu, ex, h));
#pragma unroll
        for (int j = 0; j < KL; ++j) {
            order(d[j], od[j], i[j], oi[j]);
            ex = fminf(ex, od[j]);
        }
        sort_bitonic();
    }
    static __device__ __forceinline__ void order(float &a, float &b, int &ia, int &ib)
    {
        const bool swap = b < a;
        const float lo = fminf(a, b), hi = fmaxf(a, b);
        const int il = swap ? ib : ia, ih = swap ? ia : ib;
        a = lo; b = hi; ia = il; ib = ih;
    }
    __device__ __forceinline__ void sort_bitonic()
    {
#pragma unroll
        for (int h = KL / 2; h > 0; h /= 2)
#pragma unroll
            for (int j = 0; j < KL; ++j)
                if (!(j & h)) order(d[j], d[j + h], i[j], i[j + h]);
    }
    __device__ __forceinline__ bool tied() const
    {
        bool tie = ex == d[KL - 1] && ex < KNN_FAR;
#pragma unroll
        for (int j = 1; j < KL; ++j) tie = tie || (d[j] == d[j - 1] && d[j] >= 0.f && d[j] < KNN_FAR);
        return tie;
    }
};

// Longer lists do not take their candidates one by one (an insertion costs five instructions per entry,
// for one lane of the warp as for all): a lane parks what beats its K-th distance in shared memory,
// and when a lane has eight or more parked, all lanes merge eight each.
constexpr int QUEUE = 16;

// Long lists are also shared: the SHARE lanes of a query each take their part of every leaf's sources and keep
// their own list.  A lane's K-th distance is a bound of the query's, and so is the largest of the lanes'
// ceil(K / SHARE)-th.  The lists are merged at the end.  A warp then has fewer queries, so a smaller box and
// fewer leaves to look at, and there are more warps.  K = 16, whole search with one lane / two (before queries were
// split at jumps): 4 x (30 k queries in 120 k sources) 940 / 719 us, 40 k in 135 k 674 / 456.  With the split, two /
// four lanes: 374 / 430 and 200 / 200 us, 3 x (16 k in 60 k) 164 / 211, 8 x (6 k in 20 k) 186 / 179, 3 k in 12 k 99 / 104.
constexpr int SHARED = 2;

template <int KL, int SHARE, bool ROOT>
__global__ void __launch_bounds__(SEARCH_THREADS)
tree_search_kernel(int K, const int32_t *__restrict__ qo, int B, int64_t Nq, TreeBufs t,
                   int32_t *__restrict__ ret_idx, float *__restrict__ ret_dist)
{
    constexpr bool PARK = KL >= 8;
    __shared__ float s_qd[PARK ? QUEUE : 1][PARK ? SEARCH_THREADS : 1];
    __shared__ int s_qi[PARK ? QUEUE : 1][PARK ? SEARCH_THREADS : 1];
    constexpr int PER = LEAF / SHARE;
    static_assert(PER % 8 == 0 && (SHARE == 1 || PARK), "a lane takes its sources eight at a time");
    const int64_t at = ((int64_t)blockIdx.x * SEARCH_THREADS + threadIdx.x) / SHARE;
    const int lane = threadIdx.x & 31, sub = threadIdx.x % SHARE;
    if (at - lane / SHARE >= Nq) return;                     // the whole warp
    float4 q = make_float4(NAN, NAN, NAN, __int_as_float(-1));
    if (at < Nq) q = t.qry[at];
    const int g = __float_as_int(q.w);
    const int scene = g >= 0 ? knn_scene(g, qo, B) : -1;
    TopK<KL> best;
    best.init(sub == 0 ? K : KL);                            // the entries that are -1 come once
    int parked = 0;
    float bound = KNN_FAR;                                   // of the query's K-th distance
    auto tighten = [&]() {
        bound = best.top();
        if constexpr (SHARE > 1) {
            float part = 0.f;
            const int at_part = KL - K + (K + SHARE - 1) / SHARE - 1;
#pragma unroll
            for (int j = 0; j < KL; ++j)
                if (j == at_part) part = best.d[j];
#pragma unroll
            for (int h = 1; h < SHARE; h *= 2) {
                bound = fminf(bound, __shfl_xor_sync(0xffffffffu, bound, h));
                part = fmaxf(part, __shfl_xor_sync(0xffffffffu, part, h));
            }
            bound = fminf(bound, part);
        }
    };
    // a query that is not finite has no distance below the heap's initial entry
    unsigned todo = __ballot_sync(0xffffffffu, scene >= 0 && finite3(q.x, q.y, q.z));
    while (todo) {
        const int b = __shfl_sync(0xffffffffu, scene, __ffs(todo) - 1);
        unsigned act = __ballot_sync(0xffffffffu, ((todo >> lane) & 1u) && scene == b);
        const int s0 = (int)__ldg(t.hist + ((int64_t)b << (3 * t.bits)));
        const int n = (int)__ldg(t.hist + ((int64_t)(b + 1) << (3 * t.bits))) - s0;
        if (n <= 0) {
            todo &= ~act;
            continue;
        }
        // Box of the queries.  Where the cell order jumps, the box of both sides holds far more leaves than the two
        // boxes, and a leaf costs a test against every query: the queries beyond the widest gap are left for
        // another pass if the extents of the two boxes together are less than 0.4 of that of the one (0.2 / 0.3 / 0.4 /
        // 0.5 / 0.7 / 0.85, K = 16, 4 x (30 k in 120 k): 447 / 385 / 373 / 374 / 397 / 469 us, 721 without).
        float ql[3], qh[3];
        auto box_of = [&](unsigned lanes, float (&lo)[3], float (&hi)[3]) {
            const float c[3] = {q.x, q.y, q.z};
            const bool in = (lanes >> lane) & 1u;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const uint32_t k = order_key(c[d]);
                lo[d] = from_order_key(__reduce_min_sync(0xffffffffu, in ? k : 0xffffffffu));
                hi[d] = from_order_key(__reduce_max_sync(0xffffffffu, in ? k : 0u));
            }
            return (hi[0] - lo[0]) + (hi[1] - lo[1]) + (hi[2] - lo[2]);
        };
        for (;;) {
            const float ext = box_of(act, ql, qh);
            const unsigned above = act & ~((2u << lane) - 1u);
            const int nx = above ? __ffs(above) - 1 : lane;
            const float gx = fabsf(__shfl_sync(0xffffffffu, q.x, nx) - q.x), gy = fabsf(__shfl_sync(0xffffffffu, q.y, nx) - q.y),
                        gz = fabsf(__shfl_sync(0xffffffffu, q.z, nx) - q.z);
            const uint32_t gap = ((act >> lane) & 1u) ? __float_as_uint(fmaxf(fmaxf(gx, gy), gz)) : 0u;
            const uint32_t most = __reduce_max_sync(0xffffffffu, gap);
            // ext <= ext of the parts + three gaps, so a smaller gap cannot do
            if (most == 0u || __uint_as_float(most) * 5.f < ext) break;
            const int who = __ffs(__ballot_sync(0xffffffffu, gap == most)) - 1;
            const unsigned lower = act & ((2u << who) - 1u);
            float l0[3], h0[3], l1[3], h1[3];
            if (!(box_of(lower, l0, h0) + box_of(act & ~lower, l1, h1) < 0.4f * ext)) break;
            act = lower;
        }
        todo &= ~act;
        const bool mine = (act >> lane) & 1u;
        // the other queries take part as NaN: no comparison holds for them
        const float qx = mine ? q.x : NAN, qy = mine ? q.y : NAN, qz = mine ? q.z : NAN;
        const uint64_t nx = pack2(-qx, -qx), ny = pack2(-qy, -qy), nz = pack2(-qz, -qz);
        const float *points = t.src + first_leaf(s0, b) * (4 * LEAF);
        const float4 *leaves = t.leaf + 2 * first_leaf(s0, b), *nodes = t.node + 2 * first_node(s0, b);
        const int n_leaf = (n + LEAF - 1) / LEAF, n_node = (n_leaf + 31) / 32;

        auto drain = [&]() {
            if constexpr (PARK) {
                while (__any_sync(0xffffffffu, parked > 0)) {
                    float x[8];
                    int id[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const bool in = parked > j;
                        const int from = in ? parked - 1 - j : 0;
                        x[j] = in ? s_qd[from][threadIdx.x] : INFINITY;
                        id[j] = s_qi[from][threadIdx.x];
                    }
                    parked = max(parked - 8, 0);
                    best.merge8(x, id);
                }
                tighten();
            }
        };
        auto visit = [&](int leaf) {
            const float *p = points + leaf * (4 * LEAF) + sub * PER;
#pragma unroll 2
            for (int j = 0; j < PER; j += 8) {
                float d[8];
#pragma unroll
                for (int u = 0; u < 8; u += 4) {
                    const ulonglong2 x = __ldg(reinterpret_cast<const ulonglong2 *>(p + j + u));
                    const ulonglong2 y = __ldg(reinterpret_cast<const ulonglong2 *>(p + LEAF + j + u));
                    const ulonglong2 z = __ldg(reinterpret_cast<const ulonglong2 *>(p + 2 * LEAF + j + u));
                    dist2x2(d[u], d[u + 1], x.x, y.x, z.x, nx, ny, nz);
                    dist2x2(d[u + 2], d[u + 3], x.y, y.y, z.y, nx, ny, nz);
                }
                const float m = fminf(fminf(fminf(d[0], d[1]), fminf(d[2], d[3])), fminf(fminf(d[4], d[5]), fminf(d[6], d[7])));
                if (!__any_sync(0xffffffffu, m < bound)) {
                    best.ex = fminf(best.ex, m);
                    continue;
                }
                int id[8];
#pragma unroll
                for (int u = 0; u < 8; u += 4) {
                    const int4 v = __ldg(reinterpret_cast<const int4 *>(p + 3 * LEAF + j + u));
                    id[u] = v.x; id[u + 1] = v.y; id[u + 2] = v.z; id[u + 3] = v.w;
                }
                if constexpr (PARK) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        if (d[u] < bound) {
                            s_qd[parked][threadIdx.x] = d[u];
                            s_qi[parked][threadIdx.x] = id[u];
                            ++parked;
                        } else {
                            best.ex = fminf(best.ex, d[u]);
                        }
                    }
                    if (__any_sync(0xffffffffu, parked > QUEUE - 8)) drain();
                } else {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const bool in = d[u] < bound;
                        if (!in) best.ex = fminf(best.ex, d[u]);
                        if (__any_sync(0xffffffffu, in) && in) {
                            best.insert(d[u], id[u]);
                            bound = best.top();
                        }
                    }
                }
            }
        };
        // begin with the leaf at the place of the warp's middle query, so that later boxes meet a bound
        int first;
        {
            const int mid = __fns(act, 0, (__popc(act) + 1) / 2);
            const float mx = __shfl_sync(0xffffffffu, q.x, mid), my = __shfl_sync(0xffffffffu, q.y, mid), mz = __shfl_sync(0xffffffffu, q.z, mid);
            const uint32_t start = __ldg(t.hist + ((int64_t)b << (3 * t.bits)) + cell_of(mx, my, mz, t.bbox, b, t.bits));
            first = min((int)start - s0, n - 1) / LEAF;
            visit(first);
            drain();
        }
        // the nearest of the boxes held by the lanes that can still matter; -1 if there is none
        auto nearest = [&](float lb, bool &open) {
            const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, mine ? __float_as_uint(bound) : 0u));
            const bool can = open && lb <= most;
            const uint32_t key = can ? __float_as_uint(lb) : 0xffffffffu;
            const uint32_t m = __reduce_min_sync(0xffffffffu, key);
            if (m == 0xffffffffu) return -1;
            const int who = __ffs(__ballot_sync(0xffffffffu, key == m)) - 1;
            if (lane == who) open = false;
            return who;
        };
        for (int nb = 0; nb < n_node; nb += 32) {
            bool n_open = nb + lane < n_node;
            float n_lb = INFINITY;
            if (n_open) n_lb = box_dist(__ldg(nodes + 2 * (nb + lane)), __ldg(nodes + 2 * (nb + lane) + 1), ql, qh);
            for (;;) {
                const int nd = nearest(n_lb, n_open);
                if (nd < 0) break;
                const int leaf = (nb + nd) * 32 + lane;
                bool l_open = leaf < n_leaf && leaf != first;
                float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
                float l_lb = INFINITY;
                if (l_open) {
                    lo = __ldg(leaves + 2 * leaf);
                    hi = __ldg(leaves + 2 * leaf + 1);
                    l_lb = box_dist(lo, hi, ql, qh);
                }
                for (;;) {
                    const int lf = nearest(l_lb, l_open);
                    if (lf < 0) break;
                    // does any query of its own still need it?
                    const float4 a = make_float4(__shfl_sync(0xffffffffu, lo.x, lf), __shfl_sync(0xffffffffu, lo.y, lf), __shfl_sync(0xffffffffu, lo.z, lf), 0.f);
                    const float4 c = make_float4(__shfl_sync(0xffffffffu, hi.x, lf), __shfl_sync(0xffffffffu, hi.y, lf), __shfl_sync(0xffffffffu, hi.z, lf), 0.f);
                    const float o[3] = {q.x, q.y, q.z};
                    if (__any_sync(0xffffffffu, mine && box_dist(a, c, o, o) <= bound)) visit((nb + nd) * 32 + lf);
                }
            }
        }
        drain();
    }
    if constexpr (SHARE > 1)
#pragma unroll
        for (int h = 1; h < SHARE; h *= 2) best.merge_lane(h);
    if (g < 0) return;
    if (best.tied()) {
        if (sub == 0) t.ties[atomicAdd(t.tie_count, 1)] = g;
        return;
    }
    const bool put_idx = sub == 0, put_dist = sub == SHARE - 1;
    const int64_t o = (int64_t)g * K;
    if (KL == 16 && K == 16 && !((reinterpret_cast<uintptr_t>(ret_idx) | reinterpret_cast<uintptr_t>(ret_dist)) & 15)) {
#pragma unroll
        for (int j = 0; j < KL; j += 4) {
            if (put_idx) reinterpret_cast<int4 *>(ret_idx + o)[j / 4] = make_int4(best.i[j % KL], best.i[(j + 1) % KL], best.i[(j + 2) % KL], best.i[(j + 3) % KL]);
            float4 d = make_float4(best.d[j % KL], best.d[(j + 1) % KL], best.d[(j + 2) % KL], best.d[(j + 3) % KL]);
            if (ROOT) d = make_float4(__fsqrt_rn(d.x), __fsqrt_rn(d.y), __fsqrt_rn(d.z), __fsqrt_rn(d.w));
            if (put_dist) reinterpret_cast<float4 *>(ret_dist + o)[j / 4] = d;
        }
    } else {
#pragma unroll
        for (int j = 0; j < KL; ++j)
            if (j >= KL - K) {
                if (put_idx) ret_idx[o + j - (KL - K)] = best.i[j];
                if (put_dist) ret_dist[o + j - (KL - K)] = ROOT ? __fsqrt_rn(best.d[j]) : best.d[j];
            }
    }
}

// ---- the literal heap, one entry per lane (K <= 32) ---------------------------------------------------------
// Entry i of the reference's heap lives in lane i.  The path a new root sinks along -- always to the larger
// child, the left one when they are equal -- depends on the heap alone, so every lane knows from one ballot
// (bit j: "entry j's right child is strictly larger") whether it is on it.  The new value sinks past every
// entry of the path that is not smaller than it; those move up one step.
struct LaneHeap {
    float h;
    int id;
    unsigned anc, way;       // entries above this one, and on which of them the path turns right to get here
    bool kid, kid2;
    __device__ __forceinline__ void init(int K, int lane)
    {
        h = KNN_FAR;
        id = 0;
        anc = way = 0;
        for (int i = lane; i > 0; i = (i - 1) / 2) {
            anc |= 1u << ((i - 1) / 2);
            if (!(i & 1)) way |= 1u << ((i - 1) / 2);
        }
        kid = 2 * lane + 1 < K;
        kid2 = 2 * lane + 2 < K;
        if (lane >= K) anc = 1u, way = 0xffffffffu;          // never on the path
    }
    __device__ __forceinline__ float root() const { return __shfl_sync(0xffffffffu, h, 0); }
    // d < root()
    __device__ __forceinline__ void replace(float d, int row, int lane)
    {
        const float v1 = __shfl_sync(0xffffffffu, h, (2 * lane + 1) & 31), v2 = __shfl_sync(0xffffffffu, h, (2 * lane + 2) & 31);
        const int i1 = __shfl_sync(0xffffffffu, id, (2 * lane + 1) & 31), i2 = __shfl_sync(0xffffffffu, id, (2 * lane + 2) & 31);
        const bool right = kid2 && v1 < v2;
        const float v = right ? v2 : v1;
        const unsigned turns = __ballot_sync(0xffffffffu, right);
        const bool left_empty = lane == 0 || ((turns & anc) == way && !(d > h));   // this entry moved up
        if (left_empty) {
            const bool up = kid && !(d > v);
            h = up ? v : d;
            id = up ? (right ? i2 : i1) : row;
        }
    }
};

// Result of a literal heap: the reference's heap sort, by lane 0 in shared memory.
template <bool ROOT>
__device__ __forceinline__ void finish_heap(float *heap, int *hidx, int K, int64_t g, int lane, int32_t *__restrict__ ret_idx,
                                            float *__restrict__ ret_dist)
{
    __syncwarp();
    if (lane == 0) knn_heap_sort(heap, hidx, K);
    __syncwarp();
    for (int j = lane; j < K; j += 32) {
        ret_idx[g * K + j] = hidx[j];
        ret_dist[g * K + j] = ROOT ? __fsqrt_rn(heap[j]) : heap[j];
    }
    __syncwarp();
}

// ---- tied queries of the search: a block per query ----------------------------------------------------------
// The heap is a serial chain over the candidates that enter it, several thousand when the sources are in
// spatial order.  Warp 0 runs it; the other warps scan the sources ahead of it, 8 per lane and round, and
// hand over, in index order, those below the heap root of two rounds ago -- all that can still enter.
// A list of more than list_max queries is left to the thread-per-query scan (few_ties).
constexpr int TIE_THREADS = 512, TIE_WARPS = TIE_THREADS / 32 - 1, TIE_PER = 8;

template <bool ROOT>
__global__ void __launch_bounds__(TIE_THREADS)
knn_tie_kernel(int K, const float *__restrict__ src, const float *__restrict__ query, const int32_t *__restrict__ so,
               const int32_t *__restrict__ qo, int B, const int32_t *__restrict__ list, const int *__restrict__ list_count,
               int64_t list_max, int32_t *__restrict__ ret_idx, float *__restrict__ ret_dist)
{
    __shared__ float s_d[2][TIE_WARPS][32 * TIE_PER];
    __shared__ uint16_t s_o[2][TIE_WARPS][32 * TIE_PER];     // offset from the first source of the warp's share
    __shared__ int s_n[2][TIE_WARPS];
    __shared__ float s_root[2];
    __shared__ float s_heap[32];
    __shared__ int s_hidx[32];
    const int total = __ldg(list_count);
    if (total > list_max) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int ROUND = TIE_WARPS * 32 * TIE_PER;
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int64_t g = list[w];
        const int b = knn_scene(g, qo, B);
        const int s0 = b > 0 ? __ldg(so + b - 1) : 0, s1 = __ldg(so + b);
        const int rounds = s1 > s0 ? (s1 - s0 + ROUND - 1) / ROUND : 0;
        __syncthreads();                                     // the previous query is over
        if (threadIdx.x < 2) s_root[threadIdx.x] = KNN_FAR;
        __syncthreads();
        if (wid == 0) {
            LaneHeap heap;
            heap.init(K, lane);
            for (int r = 0; r <= rounds; ++r) {
                if (r > 0) {
                    const int buf = (r - 1) & 1;
                    for (int v = 0; v < TIE_WARPS; ++v) {
                        const int cnt = s_n[buf][v];
                        const int base = s0 + (r - 1) * ROUND + v * (32 * TIE_PER);
                        for (int j = 0; j < cnt; j += 32) {
                            float d = j + lane < cnt ? s_d[buf][v][j + lane] : INFINITY;
                            const int row = base + (j + lane < cnt ? s_o[buf][v][j + lane] : 0);
                            unsigned m;
                            while ((m = __ballot_sync(0xffffffffu, d < heap.root())) != 0) {
                                const int who = __ffs(m) - 1;
                                heap.replace(__shfl_sync(0xffffffffu, d, who), __shfl_sync(0xffffffffu, row, who), lane);
                                if (lane <= who) d = INFINITY;             // earlier ones had their turn
                            }
                        }
                    }
                    if (lane == 0) s_root[buf] = heap.h;
                }
                __syncthreads();
            }
            s_heap[lane] = heap.h;
            s_hidx[lane] = heap.id;
            finish_heap<ROOT>(s_heap, s_hidx, K, g, lane, ret_idx, ret_dist);
        } else {
            const float qx = __ldg(query + g * 3), qy = __ldg(query + g * 3 + 1), qz = __ldg(query + g * 3 + 2);
            const int v = wid - 1;
            for (int r = 0; r <= rounds; ++r) {
                if (r < rounds) {
                    const int buf = r & 1;
                    const float root = s_root[buf];          // after round r - 2
                    const int base = s0 + r * ROUND + v * (32 * TIE_PER);
                    float d[TIE_PER];
#pragma unroll
                    for (int u = 0; u < TIE_PER; ++u) {
                        const int j = base + 32 * u + lane;
                        d[u] = INFINITY;
                        if (j < s1) {
                            const float *p = src + (int64_t)j * 3;
                            d[u] = knn_dist2(__ldg(p) - qx, __ldg(p + 1) - qy, __ldg(p + 2) - qz);
                        }
                    }
                    int cnt = 0;
#pragma unroll
                    for (int u = 0; u < TIE_PER; ++u) {
                        const bool in = d[u] < root;
                        const unsigned m = __ballot_sync(0xffffffffu, in);
                        if (in) {
                            const int at = cnt + __popc(m & ((1u << lane) - 1u));
                            s_d[buf][v][at] = d[u];
                            s_o[buf][v][at] = (uint16_t)(32 * u + lane);
                        }
                        cnt += __popc(m);
                    }
                    if (lane == 0) s_n[buf][v] = cnt;
                }
                __syncthreads();
            }
        }
    }
}

// ---- a warp per query, straight over the scene's sources --------------------------------------------------
// For small problems, where building the index costs more than it saves.  First pass: the smallest distance
// each lane meets on its 32nd of the sources; the K-th smallest of these 32 is a bound of the K-th
// distance, since they belong to different sources.  Second pass: the candidates within the bound, a few
// more than K, go to shared memory, and every one finds its rank by counting.  A distance tie among
// them that reaches into the result, more than 64 of them, or K > 32: scan with the literal heap.
constexpr int WARP_THREADS = 128, WARP_BATCH = 8, WARP_KEEP = 64;

template <bool ROOT>
__global__ void __launch_bounds__(WARP_THREADS)
knn_warp_kernel(int K, const float *__restrict__ src, const float *__restrict__ query, const int32_t *__restrict__ so,
                const int32_t *__restrict__ qo, int B, int64_t Nq, int32_t *__restrict__ ret_idx, float *__restrict__ ret_dist)
{
    static_assert(WARP_KEEP >= S3D_KNN_MAX_K, "the candidates and the heap share the array");
    __shared__ float s_d[WARP_THREADS / 32][WARP_KEEP];
    __shared__ int s_i[WARP_THREADS / 32][WARP_KEEP];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float *keep = s_d[wid];
    int *kidx = s_i[wid];
    const int64_t g = (int64_t)blockIdx.x * (WARP_THREADS / 32) + wid;
    if (g >= Nq) return;
    const int b = knn_scene(g, qo, B);
    const int s0 = b > 0 ? __ldg(so + b - 1) : 0, s1 = __ldg(so + b);
    const float qx = __ldg(query + g * 3), qy = __ldg(query + g * 3 + 1), qz = __ldg(query + g * 3 + 2);
    // distances of WARP_BATCH x 32 sources, source = base + 32 u + lane
    auto batch = [&](int base, float (&d)[WARP_BATCH]) {
#pragma unroll
        for (int u = 0; u < WARP_BATCH; ++u) {
            const int j = base + 32 * u + lane;
            d[u] = INFINITY;
            if (j < s1) {
                const float *p = src + (int64_t)j * 3;
                d[u] = knn_dist2(__ldg(p) - qx, __ldg(p + 1) - qy, __ldg(p + 2) - qz);
            }
        }
    };
    bool exact = K > 32;
    if (!exact) {
        float mn = INFINITY;
        for (int base = s0; base < s1; base += 32 * WARP_BATCH) {
            float d[WARP_BATCH];
            batch(base, d);
#pragma unroll
            for (int u = 0; u < WARP_BATCH; ++u) mn = fminf(mn, d[u]);       // a NaN never counts
        }
        // bitonic sort over the lanes
#pragma unroll
        for (int k = 2; k <= 32; k *= 2)
#pragma unroll
            for (int h = k / 2; h > 0; h /= 2) {
                const float o = __shfl_xor_sync(0xffffffffu, mn, h);
                mn = ((lane & h) != 0) == ((lane & k) == 0) ? fmaxf(mn, o) : fminf(mn, o);
            }
        const float bound = __shfl_sync(0xffffffffu, mn, K - 1);
        int cnt = 0;
        for (int base = s0; base < s1; base += 32 * WARP_BATCH) {
            float d[WARP_BATCH];
            batch(base, d);
#pragma unroll
            for (int u = 0; u < WARP_BATCH; ++u) {
                const bool in = d[u] <= bound && d[u] < KNN_FAR;
                const unsigned m = __ballot_sync(0xffffffffu, in);
                if (m) {
                    const int at = cnt + __popc(m & ((1u << lane) - 1u));
                    if (in && at < WARP_KEEP) {
                        keep[at] = d[u];
                        kidx[at] = base + 32 * u + lane;
                    }
                    cnt += __popc(m);
                }
            }
        }
        __syncwarp();
        exact = cnt > WARP_KEEP;
        if (!exact) {
            const float d0 = lane < cnt ? keep[lane] : INFINITY, d1 = lane + 32 < cnt ? keep[lane + 32] : INFINITY;
            int r0 = 0, r1 = 0, e0 = 0, e1 = 0;
            for (int j = 0; j < cnt; ++j) {
                const float d = keep[j];
                r0 += d < d0; r1 += d < d1;
                e0 += d == d0; e1 += d == d1;
            }
            exact = __any_sync(0xffffffffu, (lane < cnt && r0 < K && e0 > 1) || (lane + 32 < cnt && r1 < K && e1 > 1));
            if (!exact) {
                if (lane < cnt && r0 < K) {
                    ret_idx[g * K + r0] = kidx[lane];
                    ret_dist[g * K + r0] = ROOT ? __fsqrt_rn(d0) : d0;
                }
                if (lane + 32 < cnt && r1 < K) {
                    ret_idx[g * K + r1] = kidx[lane + 32];
                    ret_dist[g * K + r1] = ROOT ? __fsqrt_rn(d1) : d1;
                }
                if (lane < K && lane >= cnt) {                                // fewer candidates than K
                    ret_idx[g * K + lane] = 0;
                    ret_dist[g * K + lane] = ROOT ? __fsqrt_rn(KNN_FAR) : KNN_FAR;
                }
            }
        }
        __syncwarp();
    }
    if (!exact) return;
    if (K <= 32) {
        LaneHeap heap;
        heap.init(K, lane);
        for (int base = s0; base < s1; base += 32 * WARP_BATCH) {
            float d[WARP_BATCH];
            batch(base, d);
#pragma unroll
            for (int u = 0; u < WARP_BATCH; ++u) {
                unsigned m;
                while ((m = __ballot_sync(0xffffffffu, d[u] < heap.root())) != 0) {
                    const int who = __ffs(m) - 1;
                    heap.replace(__shfl_sync(0xffffffffu, d[u], who), base + 32 * u + who, lane);
                    if (lane <= who) d[u] = INFINITY;
                }
            }
        }
        if (lane < K) { keep[lane] = heap.h; kidx[lane] = heap.id; }
    } else {
        for (int j = lane; j < K; j += 32) { keep[j] = KNN_FAR; kidx[j] = 0; }
        __syncwarp();
        for (int base = s0; base < s1; base += 32 * WARP_BATCH) {
            float d[WARP_BATCH];
            batch(base, d);
#pragma unroll
            for (int u = 0; u < WARP_BATCH; ++u) {
                unsigned m;
                while ((m = __ballot_sync(0xffffffffu, d[u] < *(volatile float *)keep)) != 0) {
                    const int who = __ffs(m) - 1;
                    if (lane == who) {
                        keep[0] = d[u];
                        kidx[0] = base + 32 * u + who;
                        knn_sift_down(keep, kidx, 0, K);
                    }
                    if (lane <= who) d[u] = INFINITY;
                    __syncwarp();
                }
            }
        }
    }
    finish_heap<ROOT>(keep, kidx, K, g, lane, ret_idx, ret_dist);
}

}  // namespace

// Row numbers of points are int, and so is the offset of a leaf in the planes (128 floats each; in 64 bits the search for
// K = 3 was 10 % slower): the index serves up to 2^29 points, the thread-per-query scan takes what is larger.  The
// kernels of this file also count past the last row of a scene, by less than one round of the tie kernel, one
// batch of the warp scan or one node.
constexpr int64_t MAX_POINTS = ((int64_t)1 << 29) - (1 << 13);
static_assert((MAX_POINTS + LEAF - 1) / LEAF * (4 * LEAF) <= INT_MAX, "offsets in the planes");
static_assert(MAX_POINTS + TIE_WARPS * 32 * TIE_PER < INT_MAX && MAX_POINTS + 2 * 32 * WARP_BATCH < INT_MAX &&
              MAX_POINTS + LEAF * 32 < INT_MAX, "row numbers");

bool knn_tree_supported(int K, int B, int64_t Ns, int64_t Nq)
{
    return K <= 16 && Ns + Nq <= MAX_POINTS && B <= 65535;
}

bool knn_warp_wanted(int K, int B, int64_t Ns, int64_t Nq)
{
    return Ns <= MAX_POINTS && Nq * (Ns / B) <= 20000000;
}

// Up to this many tied queries get a block each (knn_tie_kernel); with more of them the thread-per-query scan does all
// queries again.  Both kernels read the count, and one of them returns at once.  4 x 120 k sources: a tied query costs 0.40 /
// 0.47 / 0.57 us (K = 3 / 8 / 16), the scan of 4 x 30 k queries 7.0 / 13.4 / 21 ms, which is an eighth, a fifth and three
// tenths of them; fewer than 10,000 queries do not fill the GPU in the scan (2,100 of 120 k sources: 3.1 / 3.5 / 3.8 ms
// against 0.6 / 0.7 / 0.8).  Many ties cost the index on top of the scan: all queries tied, K = 3, 1 to 5 % more than
// the scan alone.
static int64_t few_ties(int K, int64_t Nq)
{
    const int64_t part = K <= 4 ? Nq / 8 : (K <= 8 ? Nq / 5 : Nq * 3 / 10);
    return part > 10000 ? part : 10000;
}

int64_t knn_tree_bytes(int B, int64_t Ns, int64_t Nq) { return tree_bufs(nullptr, B, Ns, Nq).total; }

int knn_launch_warp(int K, const float *src, const float *query, const int32_t *so, const int32_t *qo, int B, int64_t Nq,
                    bool root, int32_t *idx, float *dist, cudaStream_t st)
{
    const unsigned blocks = (unsigned)((Nq + WARP_THREADS / 32 - 1) / (WARP_THREADS / 32));
    if (root) knn_warp_kernel<true><<<blocks, WARP_THREADS, 0, st>>>(K, src, query, so, qo, B, Nq, idx, dist);
    else knn_warp_kernel<false><<<blocks, WARP_THREADS, 0, st>>>(K, src, query, so, qo, B, Nq, idx, dist);
    return cudaGetLastError() == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}

int knn_launch_tree(int K, const float *src, const float *query, const int32_t *so, const int32_t *qo, int B, int64_t Ns,
                    int64_t Nq, bool root, int32_t *idx, float *dist, void *work, cudaStream_t st)
{
    const TreeBufs t = tree_bufs(static_cast<char *>(work), B, Ns, Nq);
    if (cudaMemsetAsync(t.zero, 0, (size_t)t.zero_bytes, st) != cudaSuccess) return S3D_ERR_LAUNCH;
    const int64_t per = (Ns + Nq) / B + 1;
    const unsigned gx = (unsigned)(per / (KT_THREADS * 8) < 1 ? 1 : (per / (KT_THREADS * 8) > 148 ? 148 : per / (KT_THREADS * 8)));
    tree_bbox_kernel<<<dim3(gx, (unsigned)B), KT_THREADS, 0, st>>>(src, query, so, qo, B, Nq, t.bbox);
    const unsigned nb = (unsigned)((Ns + Nq + KT_THREADS - 1) / KT_THREADS);
    tree_sort_kernel<true><<<nb, KT_THREADS, 0, st>>>(src, query, so, qo, B, Ns, Nq, t);
    scan_in_place(t.hist, t.tile, t.n_tiles, st);
    tree_sort_kernel<false><<<nb, KT_THREADS, 0, st>>>(src, query, so, qo, B, Ns, Nq, t);
    tree_boxes_kernel<<<(unsigned)(Ns / (LEAF * 32) + B), 1024, 0, st>>>(B, t);
    const int64_t few = few_ties(K, Nq);
    const int share = K <= 3 ? 1 : SHARED;
    const unsigned blocks = (unsigned)((Nq * share + SEARCH_THREADS - 1) / SEARCH_THREADS);
#define S3D_KNN_SEARCH(KL, SHARE)                                                                                   \
    if (root) tree_search_kernel<KL, SHARE, true><<<blocks, SEARCH_THREADS, 0, st>>>(K, qo, B, Nq, t, idx, dist);   \
    else tree_search_kernel<KL, SHARE, false><<<blocks, SEARCH_THREADS, 0, st>>>(K, qo, B, Nq, t, idx, dist)
    if (K <= 3) { S3D_KNN_SEARCH(3, 1); }
    else if (K <= 8) { S3D_KNN_SEARCH(8, SHARED); }
    else { S3D_KNN_SEARCH(16, SHARED); }
#undef S3D_KNN_SEARCH
    if (cudaGetLastError() != cudaSuccess) return S3D_ERR_LAUNCH;
    const unsigned tie_blocks = (unsigned)(Nq < 148 * 4 ? Nq : 148 * 4);
    if (root) knn_tie_kernel<true><<<tie_blocks, TIE_THREADS, 0, st>>>(K, src, query, so, qo, B, t.ties, t.tie_count, few, idx, dist);
    else knn_tie_kernel<false><<<tie_blocks, TIE_THREADS, 0, st>>>(K, src, query, so, qo, B, t.ties, t.tie_count, few, idx, dist);
    if (cudaGetLastError() != cudaSuccess) return S3D_ERR_LAUNCH;
    return Nq > few ? knn_launch(K, src, query, so, qo, B, Nq, root, idx, dist, st, t.tie_count, few) : S3D_OK;
}

}  // namespace s3d
