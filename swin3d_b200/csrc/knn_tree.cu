// K-nearest-neighbour search over a spatial index (K <= 16), with the results of the brute-force scan
// in knn.cu, bit for bit.
//
// Both point sets are put into Morton order of a per-scene grid by a counting sort (histogram, scan,
// scatter).  32 consecutive sources are a leaf and 32 leaves a node, each with its bounding box.
// A warp searches for 32 consecutive queries, which lie close together: the lanes test the boxes
// of 32 nodes or leaves at a time against the box of the warp's queries, nearest first, and a leaf that
// survives is offered to all 32 queries with one broadcast load per source.
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
// Bound: instruction issue of the leaf evaluation.  Measured (8 scenes x 200 k queries x 50 k sources,
// K = 3; 4 x 30 k x 120 k, K = 16): see knn_launch_tree.
#include "knn_common.cuh"
#include "knn_kernels.cuh"

namespace s3d {
namespace {

constexpr int LEAF = 32;
constexpr int KT_THREADS = 256;
constexpr int SCAN_T = 256, SCAN_PER = 16, SCAN_TILE = SCAN_T * SCAN_PER;
constexpr int SEARCH_THREADS = 128;

struct TreeBufs {
    uint32_t *zero;          // cleared by the launch: bbox, tie counter, then the two cell histograms
    uint32_t *bbox;          // [B][8] order-preserving keys of -min (0..2) and max (4..6)
    int *tie_count;
    uint32_t *hist;          // [2][B * cells]: sources, queries; after the scan the start of every cell
    uint32_t *tile;          // sums of SCAN_TILE cells
    uint32_t *rank;          // [Ns + Nq] position of a point inside its cell
    float4 *pts;             // [Ns + Nq] x, y, z, row number: sources in cell order, then queries
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
    t.pts = (float4 *)take((Ns + Nq) * 16);
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
    if (COUNT) t.rank[i] = atomicAdd(h, 1u);
    else t.pts[*h + t.rank[i]] = make_float4(x, y, z, __int_as_float((int)g));
}

// Exclusive scan of the histograms in two launches: tile sums, then every block adds up the sums of the
// tiles before its own (at most a few thousand words from L2) and scans its tile in place.
__global__ void __launch_bounds__(SCAN_T)
tree_tile_sums_kernel(const uint32_t *__restrict__ hist, uint32_t *__restrict__ tile)
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
tree_scan_kernel(uint32_t *__restrict__ hist, const uint32_t *__restrict__ tile)
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

// Boxes: a warp makes a leaf, a block (32 warps) a node.  grid = nodes of all scenes, in scene order;
// leaves and nodes of scene b, whose sources start at s0, start at s0 / 32 + b and s0 / 1024 + b of
// their arrays, which leaves room for the partial last one of every scene.
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
    if (at < n) {
        const float4 p = t.pts[s0 + at];
        lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);    // a NaN never counts
        hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
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
            float4 *o = t.leaf + 2 * ((int64_t)(s0 / LEAF) + b + leaf);
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
            float4 *o = t.node + 2 * ((int64_t)(s0 / (LEAF * 32)) + b + j);
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
    __device__ __forceinline__ bool tied() const
    {
        bool tie = ex == d[KL - 1] && ex < KNN_FAR;
#pragma unroll
        for (int j = 1; j < KL; ++j) tie = tie || (d[j] == d[j - 1] && d[j] >= 0.f && d[j] < KNN_FAR);
        return tie;
    }
};

template <int KL, bool ROOT>
__global__ void __launch_bounds__(SEARCH_THREADS)
tree_search_kernel(int K, const int32_t *__restrict__ qo, int B, int64_t Nq, TreeBufs t,
                   int32_t *__restrict__ ret_idx, float *__restrict__ ret_dist)
{
    const int64_t at = (int64_t)blockIdx.x * SEARCH_THREADS + threadIdx.x;
    const int lane = threadIdx.x & 31;
    if ((at & ~(int64_t)31) >= Nq) return;                   // the whole warp
    const uint32_t n_src = __ldg(t.hist + ((int64_t)B << (3 * t.bits)));     // the first query cell follows the last source
    float4 q = make_float4(NAN, NAN, NAN, __int_as_float(-1));
    if (at < Nq) q = t.pts[n_src + at];
    const int g = __float_as_int(q.w);
    const int scene = g >= 0 ? knn_scene(g, qo, B) : -1;
    TopK<KL> best;
    best.init(K);
    // a query that is not finite has no distance below the heap's initial entry
    unsigned todo = __ballot_sync(0xffffffffu, scene >= 0 && finite3(q.x, q.y, q.z));
    while (todo) {
        const int b = __shfl_sync(0xffffffffu, scene, __ffs(todo) - 1);
        const bool mine = ((todo >> lane) & 1u) && scene == b;
        const unsigned act = __ballot_sync(0xffffffffu, mine);
        todo &= ~act;
        const int s0 = (int)__ldg(t.hist + ((int64_t)b << (3 * t.bits)));
        const int n = (int)__ldg(t.hist + ((int64_t)(b + 1) << (3 * t.bits))) - s0;
        if (n <= 0) continue;
        // queries of other scenes take part as NaN: no comparison holds for them
        const float qx = mine ? q.x : NAN, qy = mine ? q.y : NAN, qz = mine ? q.z : NAN;
        float ql[3], qh[3];
        {
            const float c[3] = {q.x, q.y, q.z};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const uint32_t k = order_key(c[d]);
                ql[d] = from_order_key(__reduce_min_sync(0xffffffffu, mine ? k : 0xffffffffu));
                qh[d] = from_order_key(__reduce_max_sync(0xffffffffu, mine ? k : 0u));
            }
        }
        const float4 *pts = t.pts + s0;
        const float4 *leaves = t.leaf + 2 * ((int64_t)(s0 / LEAF) + b), *nodes = t.node + 2 * ((int64_t)(s0 / (LEAF * 32)) + b);
        const int n_leaf = (n + LEAF - 1) / LEAF, n_node = (n_leaf + 31) / 32;

        auto offer = [&](const float4 &p) {
            const float d = knn_dist2(p.x - qx, p.y - qy, p.z - qz);
            const bool in = d < best.top();
            if (__any_sync(0xffffffffu, in)) {
                if (in) best.insert(d, __float_as_int(p.w));
                else best.ex = fminf(best.ex, d);
            } else {
                best.ex = fminf(best.ex, d);
            }
        };
        auto visit = [&](int leaf) {
            const float4 *p = pts + leaf * LEAF;
            if ((leaf + 1) * LEAF <= n) {
#pragma unroll 4
                for (int j = 0; j < LEAF; ++j) offer(__ldg(p + j));
            } else {
                for (int j = 0; j < n - leaf * LEAF; ++j) offer(__ldg(p + j));
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
        }
        auto top_max = [&]() { return __uint_as_float(__reduce_max_sync(0xffffffffu, mine ? __float_as_uint(best.top()) : 0u)); };
        // the nearest of the boxes held by the lanes that can still matter; -1 if there is none
        auto nearest = [&](float lb, bool &open) {
            const float most = top_max();                    // by all lanes, open or not
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
                    if (__any_sync(0xffffffffu, mine && box_dist(a, c, o, o) <= best.top())) visit((nb + nd) * 32 + lf);
                }
            }
        }
    }
    if (g < 0) return;
    if (best.tied()) {
        t.ties[atomicAdd(t.tie_count, 1)] = g;
        return;
    }
    const int64_t o = (int64_t)g * K;
    if (KL == 16 && K == 16 && !((reinterpret_cast<uintptr_t>(ret_idx) | reinterpret_cast<uintptr_t>(ret_dist)) & 15)) {
#pragma unroll
        for (int j = 0; j < KL; j += 4) {
            reinterpret_cast<int4 *>(ret_idx + o)[j / 4] = make_int4(best.i[j % KL], best.i[(j + 1) % KL], best.i[(j + 2) % KL], best.i[(j + 3) % KL]);
            float4 d = make_float4(best.d[j % KL], best.d[(j + 1) % KL], best.d[(j + 2) % KL], best.d[(j + 3) % KL]);
            if (ROOT) d = make_float4(__fsqrt_rn(d.x), __fsqrt_rn(d.y), __fsqrt_rn(d.z), __fsqrt_rn(d.w));
            reinterpret_cast<float4 *>(ret_dist + o)[j / 4] = d;
        }
    } else {
#pragma unroll
        for (int j = 0; j < KL; ++j)
            if (j >= KL - K) {
                ret_idx[o + j - (KL - K)] = best.i[j];
                ret_dist[o + j - (KL - K)] = ROOT ? __fsqrt_rn(best.d[j]) : best.d[j];
            }
    }
}

// ---- a warp per query, straight over the scene's sources ------------------------------------------------
// For K <= 32 the warp keeps the sorted list one entry per lane; a distance tie (as above) or a larger
// K makes it scan again with the literal heap (lane 0, in shared memory).  Serves the small problems,
// where building the index costs more than it saves, and the tied queries of the search above
// (LIST: the queries come from a list and are known to tie).
constexpr int WARP_THREADS = 128;
constexpr int WARP_BATCH = 4;

template <bool LIST, bool ROOT>
__global__ void __launch_bounds__(WARP_THREADS)
knn_warp_kernel(int K, const float *__restrict__ src, const float *__restrict__ query, const int32_t *__restrict__ so,
                const int32_t *__restrict__ qo, int B, int64_t Nq, const int32_t *__restrict__ list,
                const int *__restrict__ list_count, int list_max, int32_t *__restrict__ ret_idx, float *__restrict__ ret_dist)
{
    __shared__ float s_heap[WARP_THREADS / 32][S3D_KNN_MAX_K];
    __shared__ int s_hidx[WARP_THREADS / 32][S3D_KNN_MAX_K];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t total = Nq;
    if (LIST) {
        total = __ldg(list_count);
        if (total > list_max) return;                        // too many: the thread-per-query scan takes them
    }
    for (int64_t w = (int64_t)blockIdx.x * (WARP_THREADS / 32) + wid; w < total; w += (int64_t)gridDim.x * (WARP_THREADS / 32)) {
        const int64_t g = LIST ? list[w] : w;
        const int b = knn_scene(g, qo, B);
        const int s0 = b > 0 ? __ldg(so + b - 1) : 0, s1 = __ldg(so + b);
        const float qx = __ldg(query + g * 3), qy = __ldg(query + g * 3 + 1), qz = __ldg(query + g * 3 + 2);
        // one pass over the sources in index order: 32 per step, every candidate that beats top() is handed to
        // take(distance, row) in order
        auto scan = [&](auto top, auto take, auto reject) {
            for (int base = s0; base < s1; base += 32 * WARP_BATCH) {
                float d[WARP_BATCH];
#pragma unroll
                for (int u = 0; u < WARP_BATCH; ++u) {
                    const int j = base + 32 * u + lane;
                    d[u] = INFINITY;
                    if (j < s1) {
                        const float *p = src + (int64_t)j * 3;
                        d[u] = knn_dist2(__ldg(p) - qx, __ldg(p + 1) - qy, __ldg(p + 2) - qz);
                    }
                }
#pragma unroll
                for (int u = 0; u < WARP_BATCH; ++u) {
                    float tp = top();
                    unsigned m = __ballot_sync(0xffffffffu, d[u] < tp);
                    while (m) {
                        const int who = __ffs(m) - 1;
                        const float dd = __shfl_sync(0xffffffffu, d[u], who);
                        take(dd, base + 32 * u + who);
                        if (lane == who) d[u] = INFINITY;
                        tp = top();
                        m = __ballot_sync(0xffffffffu, d[u] < tp);
                    }
                    reject(d[u]);
                }
            }
        };
        bool exact = LIST || K > 32;
        if (!exact) {
            float a = lane < K ? KNN_FAR : INFINITY, ex = INFINITY;
            int ai = 0;
            scan([&]() { return __shfl_sync(0xffffffffu, a, K - 1); },
                 [&](float dd, int row) {
                     const float last = __shfl_sync(0xffffffffu, a, K - 1);
                     ex = fminf(ex, last);
                     const int at = __popc(__ballot_sync(0xffffffffu, a <= dd));
                     const float up_a = __shfl_up_sync(0xffffffffu, a, 1);
                     const int up_i = __shfl_up_sync(0xffffffffu, ai, 1);
                     if (lane < K) {
                         if (lane > at) { a = up_a; ai = up_i; }
                         else if (lane == at) { a = dd; ai = row; }
                     }
                 },
                 [&](float d) { ex = fminf(ex, d); });
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ex = fminf(ex, __shfl_xor_sync(0xffffffffu, ex, o));
            const float before = __shfl_up_sync(0xffffffffu, a, 1), last = __shfl_sync(0xffffffffu, a, K - 1);
            const bool tie = (lane > 0 && lane < K && a == before && a < KNN_FAR) || (last < KNN_FAR && ex == last);
            exact = __any_sync(0xffffffffu, tie);
            if (!exact && lane < K) {
                ret_idx[g * K + lane] = ai;
                ret_dist[g * K + lane] = ROOT ? __fsqrt_rn(a) : a;
            }
        }
        if (exact) {
            float *heap = s_heap[wid];
            int *hidx = s_hidx[wid];
            __syncwarp();
            for (int j = lane; j < K; j += 32) { heap[j] = KNN_FAR; hidx[j] = 0; }
            __syncwarp();
            scan([&]() { return *(volatile float *)heap; },
                 [&](float dd, int row) {
                     if (lane == 0) {
                         heap[0] = dd;
                         hidx[0] = row;
                         knn_sift_down(heap, hidx, 0, K);
                     }
                     __syncwarp();
                 },
                 [&](float) {});
            if (lane == 0) knn_heap_sort(heap, hidx, K);
            __syncwarp();
            for (int j = lane; j < K; j += 32) {
                ret_idx[g * K + j] = hidx[j];
                ret_dist[g * K + j] = ROOT ? __fsqrt_rn(heap[j]) : heap[j];
            }
            __syncwarp();
        }
    }
}

template <bool LIST>
void launch_warp(int K, const float *src, const float *query, const int32_t *so, const int32_t *qo, int B, int64_t Nq,
                 const int32_t *list, const int *count, int list_max, bool root, int32_t *idx, float *dist, unsigned blocks, cudaStream_t st)
{
    if (root) knn_warp_kernel<LIST, true><<<blocks, WARP_THREADS, 0, st>>>(K, src, query, so, qo, B, Nq, list, count, list_max, idx, dist);
    else knn_warp_kernel<LIST, false><<<blocks, WARP_THREADS, 0, st>>>(K, src, query, so, qo, B, Nq, list, count, list_max, idx, dist);
}

}  // namespace

bool knn_tree_supported(int K, int B, int64_t Ns, int64_t Nq)
{
    return K <= 16 && Ns + Nq < ((int64_t)1 << 31) && B <= 65535;
}

bool knn_warp_wanted(int K, int B, int64_t Ns, int64_t Nq)
{
    return Nq * (Ns / B) <= 20000000;
}

int64_t knn_tree_bytes(int B, int64_t Ns, int64_t Nq) { return tree_bufs(nullptr, B, Ns, Nq).total; }

int knn_launch_warp(int K, const float *src, const float *query, const int32_t *so, const int32_t *qo, int B, int64_t Nq,
                    bool root, int32_t *idx, float *dist, cudaStream_t st)
{
    const unsigned blocks = (unsigned)((Nq + WARP_THREADS / 32 - 1) / (WARP_THREADS / 32));
    launch_warp<false>(K, src, query, so, qo, B, Nq, nullptr, nullptr, 0, root, idx, dist, blocks, st);
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
    tree_tile_sums_kernel<<<(unsigned)t.n_tiles, SCAN_T, 0, st>>>(t.hist, t.tile);
    tree_scan_kernel<<<(unsigned)t.n_tiles, SCAN_T, 0, st>>>(t.hist, t.tile);
    tree_sort_kernel<false><<<nb, KT_THREADS, 0, st>>>(src, query, so, qo, B, Ns, Nq, t);
    tree_boxes_kernel<<<(unsigned)(Ns / (LEAF * 32) + B), 1024, 0, st>>>(B, t);
    const unsigned blocks = (unsigned)((Nq + SEARCH_THREADS - 1) / SEARCH_THREADS);
#define S3D_KNN_SEARCH(KL)                                                                                          \
    if (root) tree_search_kernel<KL, true><<<blocks, SEARCH_THREADS, 0, st>>>(K, qo, B, Nq, t, idx, dist);       \
    else tree_search_kernel<KL, false><<<blocks, SEARCH_THREADS, 0, st>>>(K, qo, B, Nq, t, idx, dist)
    if (K <= 3) { S3D_KNN_SEARCH(3); }
    else if (K <= 8) { S3D_KNN_SEARCH(8); }
    else { S3D_KNN_SEARCH(16); }
#undef S3D_KNN_SEARCH
    if (cudaGetLastError() != cudaSuccess) return S3D_ERR_LAUNCH;
    // tied queries: a warp each while they are few, otherwise the thread-per-query scan; both kernels read
    // the count and one of them returns at once
    constexpr int FEW = 16384;
    launch_warp<true>(K, src, query, so, qo, B, Nq, t.ties, t.tie_count, FEW, root, idx, dist, 148 * 8, st);
    if (cudaGetLastError() != cudaSuccess) return S3D_ERR_LAUNCH;
    return Nq > FEW ? knn_launch_list(K, src, query, so, qo, B, Nq, t.ties, t.tie_count, FEW, root, idx, dist, st) : S3D_OK;
}

}  // namespace s3d
