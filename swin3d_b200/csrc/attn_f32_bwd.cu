// Backward of the cRSE window attention in fp32 (head_dim 8 and 16), for windows of any size: the
// factorised single-sweep scheme of attn_tc_bwd_small.cu with fp32 values throughout and one head
// per block.
//
// A window of n voxels is cut into nt = ceil(n / 32) tiles and the work item is a tile pair (query tile i,
// key tile j); items of a row run one after the other in the same block, later shares of dQ, dK, dV are
// added to the rows already written.  In calls of few windows a window's query and key tiles go to different
// blocks (split_windows).  Per item, phases separated by a barrier of the consumer warps:
//   project    P_q = Tq.Q^T, dB = Tv.dO^T as [row][query], P_k = Tk.K^T as [key][row]; lane = voxel with
//              its row in registers, table rows broadcast from a staged 16-row tile
//   scores     lane = query, keys dealt to the warps: q.k and dO.v, D indices, 3*D look-ups, p = exp(s - lse),
//              ds = p (dP - delta); planes p, ds, idx 0-4, idx 5-8 as [key][query], row stride 33
//   clear      the histograms, which reuse the storage of P_q, dB, P_k
//   histogram  warps 0..D-1: histQ += ds, histV += p for their dimension (lanes = queries); the next
//              (D+1)/2: histK += ds (lanes = keys); one warp dQ += ds.K and dK += ds.Q, one dV = p.dO
//   tables     dTq += histQ.Q, dTv += histV.dO, dTk += histK.K: lane = table row, its sum over all windows
//              of the block in registers; lane l starts at voxel l, so the 32 rows of a unit are read
//              from 32 different banks
//   products   dQ += histQ.Tq, dK += histK.Tk: lane = voxel, row tiles dealt to the warps
//   store      reduce over the warps, write or add the rows
// The last two run over whole row tiles, with zeros where no pair touches a row.  Where the other operand is not finite
// (flags found beside the projections, and once per block for the tables) the zeros are passed over
// there, so that a result becomes infinite or NaN only through a pair that reaches it.
// All products are fp32 FMAs, two per instruction (fma.f32x2): no operand is rounded to fewer bits.
// Row numbering and tile skipping as in PermMeta (attn_tc.cuh).
//
// Bound: instruction issue (51 % of the slots with 16 warps per SM; shared memory of 160 to 220 KB allows one
// block) and shared-memory wavefronts (64 % of the pipe).  The generic kernel this replaces recomputes every pair's
// table products channel by channel, twice, and adds a histogram row by row for every (voxel, head): 117 k voxels, 6
// heads of 8 channels, mixed precision 8.40 -> 3.51 ms a training pass.
#include "attn_kernels.cuh"
#include "attn_tc.cuh"
#include "async_stage.cuh"

namespace s3d {
namespace f32 {

using tc::PairConsts;
using tc::PermMeta;
using tc::QT;
using tc::IDX_BITS;

constexpr int STAGES = 2;
constexpr int ES = 33;                                       // row stride of the pair planes
enum { ROLE_Q = 1, ROLE_K = 2 };                             // what an item contributes to: dQ, dTq, dTv; dK, dV, dTk
// head_dim 16 with six signal dimensions: 15 warps leave 128 registers and spill (8 k voxels, 6 heads 1.90 -> 2.15 ms)
__host__ __device__ constexpr int warps_for(int D, int HD) { return D == 3 || (D == 6 && HD == 16) ? 11 : 15; }

// How the warps share the last two kinds of products.  A step of the table gradients reads a voxel row per
// lane, and every 32-row unit a warp holds reuses it: head_dim 8 gives the gradients to 3 * DTW warps
// with up to NDT units each (8 registers a unit) and the hist.T products to the others at the same
// time.  (All warps doing both in turn, one or two units each: 19 k shared-memory wavefronts per item,
// the pipe 80 % busy, 3.39 instead of 2.72 ms for 115 k voxels, 6 heads.)  At head_dim 16 a unit is 16
// registers: every warp takes its share of both, up to three units.
template <int D, int HD>
struct Split {
    static constexpr int NW = warps_for(D, HD);
    static constexpr bool APART = HD == 8;
    static constexpr int DTW = APART ? (D == 3 ? 2 : 3) : NW / 3;                  // gradient warps per table
    static constexpr int NDT = APART ? (D == 3 ? 3 : 4) : 3;                       // 32-row units per warp
    static constexpr int HT0 = APART ? 3 * DTW : 0;                                // first warp of the hist.T products
    static constexpr int SG = (NW - HT0) / 2;                                      // warps per side of them
};
constexpr int row_stride(int hd) { return hd + 4; }          // lanes = voxels read 16-byte pieces without conflicts

struct Smem {
    int R16, Rp;
    int off_pq, off_db, off_pk, off_pl, off_rows, off_c, off_pg, off_st, off_lut, off_map, off_misc, total;
};

template <int D, int HD>
__host__ __device__ inline Smem make_smem(int R, int lut_entries)
{
    constexpr int nw = warps_for(D, HD), hd = HD, rs = row_stride(HD);
    Smem L;
    L.R16 = (R + 15) / 16 * 16;
    L.Rp = L.R16 + 1;                                        // odd: lanes = keys write P_k without conflicts
    const int arr = L.R16 * QT * 4;
    int off = 0;
    L.off_pq = off; off += arr;                              // P_q, later histQ
    L.off_db = off; off += arr;                              // dB, later histV
    L.off_pk = off; off += (32 * L.Rp * 4 + 15) / 16 * 16;   // P_k, later histK
    // the pair planes; over them, once the histograms exist, the partial dQ and dK of the warps
    const int planes = 4 * 32 * ES * 4, part = 2 * Split<D, HD>::SG * 32 * hd * 4;
    L.off_pl = off; off += planes > part ? planes : part;
    L.off_rows = off; off += STAGES * 4 * 32 * rs * 4;       // Q, dO (query tile), K, V (key tile), per stage
    L.off_c = off; off += STAGES * 2 * 32 * 12 * 4;          // coordinates of both tiles, per stage
    L.off_pg = off; off += 3 * 32 * hd * 4;                  // dQ, dV, dK of the pair products
    L.off_st = off; off += nw * 16 * hd * 4;                 // a 16-row table tile per warp
    L.off_lut = off; off += (lut_entries * 2 + 15) / 16 * 16;
    L.off_map = off; off += (L.R16 * 2 + 15) / 16 * 16;      // internal row -> table row
    L.off_misc = off; off += 2048;
    L.total = off;
    return L;
}

struct Params {
    const float *q, *k, *v, *dout, *o, *lse, *tq, *tk, *tv;
    float *dq, *dk, *dv, *dtq, *dtk, *dtv;
    const int32_t *w_sizes, *w2n, *n2n;
    const float *n_coords;
    int64_t W;
    int H;
};

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t dup2(float x)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sum2(uint64_t a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    return x + y;
}

__device__ __forceinline__ bool finite4(const float4 &v)
{
    return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))) < INFINITY && v.x == v.x && v.y == v.y && v.z == v.z && v.w == v.w;
}

// __expf rounds x * log2(e) before the exponential; the rounding error is put back to first order.
__device__ __forceinline__ float exp_rounded_once(float x)
{
    constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
    const float t = x * LOG2E, e = tc::ex2_approx(t);
    return fabsf(t) < 126.f ? fmaf(e, fmaf(x, LOG2E, -t) * LN2, e) : e;
}

// A row of HD floats as HD/2 packed pairs (16-byte loads).
template <int HD>
__device__ __forceinline__ void load_row(uint64_t (&r)[HD / 2], const float *p)
{
#pragma unroll
    for (int i = 0; i < HD / 4; ++i) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p + 4 * i);
        r[2 * i] = v.x;
        r[2 * i + 1] = v.y;
    }
}
template <int HD>
__device__ __forceinline__ void store_row(float *p, const uint64_t (&r)[HD / 2])
{
#pragma unroll
    for (int i = 0; i < HD / 4; ++i) {
        ulonglong2 v;
        v.x = r[2 * i];
        v.y = r[2 * i + 1];
        *reinterpret_cast<ulonglong2 *>(p + 4 * i) = v;
    }
}
template <int HD>
__device__ __forceinline__ float dot_row(const uint64_t (&a)[HD / 2], const float *p)
{
    uint64_t b[HD / 2];
    load_row<HD>(b, p);
    uint64_t s = mul2(a[0], b[0]);
#pragma unroll
    for (int i = 1; i < HD / 2; ++i) s = fma2(a[i], b[i], s);
    return sum2(s);
}
template <int HD>
__device__ __forceinline__ void axpy_row(uint64_t (&acc)[HD / 2], float x, const float *p)
{
    uint64_t b[HD / 2];
    load_row<HD>(b, p);
    const uint64_t xx = dup2(x);
#pragma unroll
    for (int i = 0; i < HD / 2; ++i) acc[i] = fma2(xx, b[i], acc[i]);
}

// A 16-row tile of a table, through the row map: fetched to registers, stored to the warp's buffer.
template <int HD>
struct TableTile {
    float4 f[HD / 8];
    __device__ __forceinline__ void fetch(const float *T, int HC, int co, const uint16_t *map, int mt, int lane)
    {
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) {
            const int e = lane + 32 * j, r = e / (HD / 4), c4 = e % (HD / 4);
            const int row = map[mt * 16 + r];
            f[j] = row != 0xffff ? __ldg(reinterpret_cast<const float4 *>(T + (int64_t)row * HC + co) + c4)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ void put(float *st, int lane) const
    {
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) reinterpret_cast<float4 *>(st)[lane + 32 * j] = f[j];
    }
};

template <int D, int HD>
__global__ void __launch_bounds__((warps_for(D, HD) + 1) * 32, 1)
attn_bwd_f32_kernel(const Params P, const PermMeta pm, const PairConsts pc)
{
    constexpr int NW = warps_for(D, HD), NT = NW * 32;
    constexpr int TG = NW / 3;                   // warps per table (projections and table gradients)
    constexpr int NKW = (D + 1) / 2;             // warps of the key-side histogram, two dimensions each
    constexpr int GEMM_WARP = D + NKW;           // dQ and dK pair products
    constexpr int DV_WARP = (D & 1) ? D + NKW - 1 : D + NKW + 1;
    static_assert(DV_WARP < NW && GEMM_WARP < NW, "not enough warps");
    using SP = Split<D, HD>;
    constexpr int SG = SP::SG, NDT = SP::NDT, DTW = SP::DTW, RS = row_stride(HD);
    constexpr int KPW = (QT + NW - 1) / NW;      // keys per warp in the score phase
    constexpr int HP = HD / 2;
    extern __shared__ __align__(16) unsigned char smem[];
    const Smem L = make_smem<D, HD>(pm.R, pm.D * pm.lut_stride);
    float *s_pq = reinterpret_cast<float *>(smem + L.off_pq);
    float *s_db = reinterpret_cast<float *>(smem + L.off_db);
    float *s_pk = reinterpret_cast<float *>(smem + L.off_pk);
    float *s_hq = s_pq, *s_hv = s_db, *s_hk = s_pk;
    float *s_P = reinterpret_cast<float *>(smem + L.off_pl), *s_DS = s_P + 32 * ES;
    uint32_t *s_W0 = reinterpret_cast<uint32_t *>(s_DS + 32 * ES), *s_W1 = s_W0 + 32 * ES;
    float *s_part = s_P;                                                // [2][SG][32][HD]
    float *s_rows = reinterpret_cast<float *>(smem + L.off_rows);       // [stage][Q,dO,K,V][32][RS]
    float *s_cs = reinterpret_cast<float *>(smem + L.off_c);            // [stage][query tile, key tile][32][12]
    float *s_pg = reinterpret_cast<float *>(smem + L.off_pg);           // [3][32][HD]
    uint16_t *s_lut = reinterpret_cast<uint16_t *>(smem + L.off_lut);
    uint16_t *s_map = reinterpret_cast<uint16_t *>(smem + L.off_map);
    float *s_lses = reinterpret_cast<float *>(smem + L.off_misc);       // [stage][32]
    float *s_dels = s_lses + STAGES * 32;                               // [stage][32]
    int *s_rowi = reinterpret_cast<int *>(s_dels + STAGES * 32);        // [stage][query tile, key tile][32]
    int *s_n = s_rowi + STAGES * 64;                                    // [stage][8]: nq, nk, j > 0, i > 0, used tiles, roles; nq = 0: no more items
    int *s_fail = s_n + STAGES * 8;
    int *s_odd = s_fail + 1;                                            // [0]: bytes, rows of Q, dO, K of the item not finite; [1], [2]: Tq, Tk
    uint64_t *s_full = reinterpret_cast<uint64_t *>(smem + L.off_misc + 1792), *s_empty = s_full + STAGES;

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int head = blockIdx.y, H = P.H, HC = H * HD, co = head * HD;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(s_full + s, 64);         // every producer lane: its stores, its copies
            mbar_init(s_empty + s, NW);
        }
        *s_fail = 0;
        s_odd[0] = s_odd[1] = s_odd[2] = 0;
        mbar_init_fence();
    }
    tc::fill_perm_lut(s_lut, pm, tid, blockDim.x);
    for (int r = tid; r < L.R16; r += blockDim.x) {
        const int row = tc::perm_table_row(pm, r);
        s_map[r] = row < 0 ? (uint16_t)0xffff : (uint16_t)row;
    }
    __syncthreads();
    for (int e = tid; e < L.R16 * (HD / 4); e += blockDim.x) {
        const int row = s_map[e / (HD / 4)];
        if (row != 0xffff) {
            const int64_t o = (int64_t)row * HC + co + e % (HD / 4) * 4;
            if (!finite4(__ldg(reinterpret_cast<const float4 *>(P.tq + o)))) s_odd[1] = 1;
            if (!finite4(__ldg(reinterpret_cast<const float4 *>(P.tk + o)))) s_odd[2] = 1;
        }
    }
    // this block's share: a contiguous range of equal cost
    const bool split = tc::split_windows<(NW + 1) * 32, 7, 8>(P.w_sizes, P.W, smem + L.off_pq);
    int64_t w_begin, w_end;
    int u_begin, u_end;                          // first unit of window w_begin, one past the last of window w_end
    if (split) tc::balanced_units<(NW + 1) * 32>(P.w_sizes, P.W, smem + L.off_pq, tc::UnitsSplit<7, 8>{}, w_begin, w_end, u_begin, u_end);
    else tc::balanced_units<(NW + 1) * 32>(P.w_sizes, P.W, smem + L.off_pq, tc::UnitsWhole{}, w_begin, w_end, u_begin, u_end);

    if (wid == NW) {
        // ================================ producer warp ================================================
        // Sizes of the next window are fetched when a window is opened, row numbers and coordinates of the
        // next item at the end of the current iteration; only lse, dO and O (indexed by the row number)
        // are loaded inside it.
        int64_t w = w_begin - 1;
        int n = 0, base = 0, nt = 0, ts = 0, ti = 0, tj = 0;
        int unit = 0, unit_end = 0, role = 0;              // a window is one unit of both roles, or (halves) 2 nt of one
        bool halves = false;
        int n_nx = 0, base_nx = 0;
        if (w_begin < P.W) {
            n_nx = __ldg(P.w_sizes + w_begin);
            base_nx = __ldg(P.w2n + w_begin);
        }
        bool have = false;
        int nq = 0, nk = 0, rowq = 0, rowk = 0;
        float cq[D], ck[D];
        auto advance = [&]() {
            if (have && (role & ROLE_Q) && tj + 1 < nt) {
                ++tj;
            } else if (have && (role & ROLE_K) && ti + 1 < nt) {
                ++ti;
                if (role & ROLE_Q) tj = 0;
            } else {
                ++unit;
                while (unit >= unit_end) {                 // the next window with voxels
                    ++w;
                    have = w < w_end || (w == w_end && u_end > 0);
                    if (!have) break;
                    n = n_nx;
                    base = base_nx;
                    if (w + 1 < P.W) {
                        n_nx = __ldg(P.w_sizes + w + 1);
                        base_nx = __ldg(P.w2n + w + 1);
                    }
                    nt = (n + QT - 1) / QT;
                    ts = nt > 0 ? (n + nt - 1) / nt : 0;
                    halves = split && nt > 1;
                    unit = w == w_begin ? u_begin : 0;
                    unit_end = w == w_end ? u_end : (halves ? 2 * nt : (nt > 0 ? 1 : 0));
                }
                role = !halves ? ROLE_Q | ROLE_K : (unit < nt ? ROLE_Q : ROLE_K);
                ti = role == ROLE_Q ? unit : 0;
                tj = role == ROLE_K ? unit - nt : 0;
            }
            nq = have ? min(ts, n - ti * ts) : 0;
            nk = have ? min(ts, n - tj * ts) : 0;
            rowq = rowk = 0;
#pragma unroll
            for (int d = 0; d < D; ++d) cq[d] = ck[d] = 0.f;
            if (lane < nq) {
                const int pos = base + ti * ts + lane;
                rowq = __ldg(P.n2n + pos);
#pragma unroll
                for (int d = 0; d < D; ++d) cq[d] = __ldg(P.n_coords + (int64_t)pos * D + d);
            }
            if (lane < nk) {
                const int pos = base + tj * ts + lane;
                rowk = __ldg(P.n2n + pos);
#pragma unroll
                for (int d = 0; d < D; ++d) ck[d] = __ldg(P.n_coords + (int64_t)pos * D + d);
            }
        };
        advance();
        for (int it = 0;; ++it) {
            float ls = 0.f, de = 0.f;
            float4 gd[HD / 4], go[HD / 4];
            if (lane < nq) {
                ls = __ldg(P.lse + (int64_t)rowq * H + head);
                const float4 *a = reinterpret_cast<const float4 *>(P.dout + (int64_t)rowq * HC + co);
                const float4 *b = reinterpret_cast<const float4 *>(P.o + (int64_t)rowq * HC + co);
#pragma unroll
                for (int i = 0; i < HD / 4; ++i) { gd[i] = __ldg(a + i); go[i] = __ldg(b + i); }
            }
            const uint32_t used = tc::item_tile_mask<D>(cq, ck, nq, nk, s_lut, pm, pc, lane);
            if (lane < nq) {
#pragma unroll
                for (int i = 0; i < HD / 4; ++i)
                    de = fmaf(gd[i].x, go[i].x, fmaf(gd[i].y, go[i].y, fmaf(gd[i].z, go[i].z, fmaf(gd[i].w, go[i].w, de))));
            }
            const int s = it % STAGES;
            if (it >= STAGES && !mbar_wait(s_empty + s, ((it / STAGES) - 1) & 1)) {
                g_async_error = 1;
                nq = nk = 0;                                  // tell the consumers to stop
            }
            float *rq = s_rows + s * (4 * 32 * RS);
            float *cs = s_cs + s * 768;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                cs[lane * 12 + d] = cq[d];
                cs[384 + lane * 12 + d] = ck[d];
            }
            s_rowi[s * 64 + lane] = rowq;
            s_rowi[s * 64 + 32 + lane] = rowk;
            s_lses[s * 32 + lane] = ls;
            s_dels[s * 32 + lane] = de;
            if (lane == 0) {
                s_n[s * 8] = nq;
                s_n[s * 8 + 1] = nk;
                s_n[s * 8 + 2] = tj > 0;
                s_n[s * 8 + 3] = ti > 0;
                s_n[s * 8 + 5] = role;
                s_n[s * 8 + 4] = (int)used;
            }
            mbar_arrive(s_full + s);
            stage_rows<HD / 4>(rq, RS, P.q + co, HC, rowq, nq, lane);
            stage_rows<HD / 4>(rq + 32 * RS, RS, P.dout + co, HC, rowq, nq, lane);
            stage_rows<HD / 4>(rq + 64 * RS, RS, P.k + co, HC, rowk, nk, lane);
            stage_rows<HD / 4>(rq + 96 * RS, RS, P.v + co, HC, rowk, nk, lane);
            mbar_arrive_cp_async(s_full + s);
            if (nq == 0) break;
            advance();
        }
        return;
    }

    // ==================================== consumer warps ===============================================
    const int n_mt = L.R16 / 16, Rp = L.Rp;
    // warps [0, TG) serve Tq with Q, [TG, 2 TG) Tv with dO, [2 TG, 3 TG) Tk with K; tiles (projections) and
    // 32-row units (gradients) are dealt round-robin inside a group
    const int tg = wid / TG, wsub = wid - tg * TG;
    const float *Tproj = tg == 0 ? P.tq : (tg == 1 ? P.tv : P.tk);
    const int dtg = wid / DTW, dsub = wid - dtg * DTW;        // table gradients: the same order of tables
    const int side = wid < SP::HT0 ? 2 : (wid - SP::HT0) / SG, ws2 = (wid - SP::HT0) - side * SG;   // hist.T: 0 = histQ.Tq, 1 = histK.Tk
    float *st = reinterpret_cast<float *>(smem + L.off_st) + wid * (16 * HD);
    uint64_t dt_acc[NDT][HP];
#pragma unroll
    for (int u = 0; u < NDT; ++u)
#pragma unroll
        for (int i = 0; i < HP; ++i) dt_acc[u][i] = 0ull;

    int it = 0;
    for (;; ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(s_full + s, (it / STAGES) & 1)) {
            *s_fail = 1;
            g_async_error = 2;
        }
        consumer_sync<NT>();          // the previous item's stores are over; the flag is settled
        const int nq = s_n[s * 8], nk = s_n[s * 8 + 1];
        const bool add_q = s_n[s * 8 + 2] != 0, add_k = s_n[s * 8 + 3] != 0;
        const bool do_q = s_n[s * 8 + 5] & ROLE_Q, do_k = s_n[s * 8 + 5] & ROLE_K;
        const uint32_t used = (uint32_t)s_n[s * 8 + 4];
        if (nq == 0 || *s_fail) break;
        const float *s_q = s_rows + s * (4 * 32 * RS), *s_do = s_q + 32 * RS, *s_k = s_do + 32 * RS, *s_v = s_k + 32 * RS;
        const float *s_c = s_cs + s * 768, *s_ck = s_c + 384;
        const int *s_rowq = s_rowi + s * 64, *s_rowk = s_rowq + 32;
        // ---- projections ------------------------------------------------------------------------------------
        if (tg < 3) {
            uint64_t x[HP];
            load_row<HD>(x, (tg == 0 ? s_q : (tg == 1 ? s_do : s_k)) + lane * RS);
            if (wsub == TG - 1) {                                     // 0 * x is zero for every finite x
                uint64_t z = mul2(x[0], 0ull);
#pragma unroll
                for (int i = 1; i < HP; ++i) z = fma2(x[i], 0ull, z);
                const bool odd = __any_sync(0xffffffffu, sum2(z) != 0.f);
                if (lane == 0) reinterpret_cast<uint8_t *>(s_odd)[tg] = odd;
            }
            TableTile<HD> tile;
            tc::UsedTiles tiles(used, n_mt, wsub, TG);
            int mt = tiles.next();
            if (mt >= 0) tile.fetch(Tproj, HC, co, s_map, mt, lane);
            while (mt >= 0) {
                __syncwarp();
                tile.put(st, lane);
                __syncwarp();
                const int nx = tiles.next();
                if (nx >= 0) tile.fetch(Tproj, HC, co, s_map, nx, lane);
                if (tg < 2) {
                    float *dst = (tg == 0 ? s_pq : s_db) + mt * 16 * QT + lane;
#pragma unroll 4
                    for (int r = 0; r < 16; ++r) dst[r * QT] = dot_row<HD>(x, st + r * HD);
                } else {
                    float *dst = s_pk + lane * Rp + mt * 16;
#pragma unroll 4
                    for (int r = 0; r < 16; ++r) dst[r] = dot_row<HD>(x, st + r * HD);
                }
                mt = nx;
            }
        }
        consumer_sync<NT>();
        // ---- scores: keys wid, wid + NW, ... ; lane = query ---------------------------------------------------
        {
            uint64_t q2[HP], g2[HP];
            load_row<HD>(q2, s_q + lane * RS);
            load_row<HD>(g2, s_do + lane * RS);
            float cx[D];
            tc::load_coords12<D>(s_c + lane * 12, cx);
            const float lse = s_lses[s * 32 + lane], del = s_dels[s * 32 + lane];
            const float *pq_lane = s_pq + lane, *db_lane = s_db + lane;
#pragma unroll
            for (int j = 0; j < KPW; ++j) {
                const int kk = wid + NW * j;
                if (kk < QT) {
                    float p = 0.f, ds = 0.f;
                    uint32_t w0 = 0u, w1 = 0u;                     // zero for keys beyond the window
                    if (kk < nk) {
                        float ck[D];
                        tc::load_coords12<D>(s_ck + kk * 12, ck);
                        const float *pk_row = s_pk + kk * Rp;
                        float b0 = 0.f, b1 = 0.f, b2 = 0.f;      // table terms, small beside the products: summed first
#pragma unroll
                        for (int d = 0; d < D; ++d) {
                            const uint32_t idx = tc::crse_index_pc(cx[d], ck[d], pc.half[d], pc.clamp[d]);
                            const uint32_t row = s_lut[d * pm.lut_stride + idx];
                            b0 += pq_lane[row * QT];
                            b1 += pk_row[row];
                            b2 += db_lane[row * QT];
                            if (d < 5) w0 |= idx << (IDX_BITS * d);
                            else w1 |= idx << (IDX_BITS * (d - 5));
                        }
                        if (lane < nq) {
                            p = exp_rounded_once(dot_row<HD>(q2, s_k + kk * RS) - lse + (b0 + b1));
                            ds = p * (dot_row<HD>(g2, s_v + kk * RS) - del + b2);
                        }
                    }
                    s_P[kk * ES + lane] = p;
                    s_DS[kk * ES + lane] = ds;
                    s_W0[kk * ES + lane] = w0;
                    s_W1[kk * ES + lane] = w1;
                }
            }
        }
        consumer_sync<NT>();
        const int odd_rows = s_odd[0];
        // ---- clear the histograms ------------------------------------------------------------------------------
        for (int i = tid; i < L.R16 * QT / 4; i += NT)                 // 128 16-byte pieces per 16-row tile
            if ((used >> (i >> 7)) & 1u) {
                const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                if (do_q) {
                    reinterpret_cast<float4 *>(s_hq)[i] = z;
                    reinterpret_cast<float4 *>(s_hv)[i] = z;
                }
                if (do_k) reinterpret_cast<float4 *>(s_hk)[i] = z;
            }
        consumer_sync<NT>();
        // ---- histograms and pair products ----------------------------------------------------------------------
        if (wid < D && do_q) {
            // lanes = queries, two keys per step, the next step's entries fetched before this step's stores
            const int d = wid;
            const bool lo = d < 5;
            const int sh = IDX_BITS * (lo ? d : d - 5);
            const float *pcol = s_P + lane, *dcol = s_DS + lane;
            const uint32_t *wcol = (lo ? s_W0 : s_W1) + lane;
            const uint16_t *lut = s_lut + d * pm.lut_stride;
            float *cell = s_hq + lane;
            const int hv = L.R16 * QT;                     // histV follows histQ
            // software pipeline: the rows of this step are known; its cells, the rows of the next step and
            // the pair entries after that are fetched together
            auto row_of = [&](uint32_t x) { return (int)lut[(x >> sh) & ((1u << IDX_BITS) - 1u)] * QT; };
            int r0 = row_of(wcol[0]), r1 = row_of(wcol[ES]);
            uint32_t x0 = wcol[2 * ES], x1 = wcol[3 * ES];
            float p0 = pcol[0], d0 = dcol[0], p1 = pcol[ES], d1 = dcol[ES];
            for (int kk = 0; kk < nk; kk += 2) {           // entries beyond the window are zero
                float *a0 = cell + r0, *a1 = cell + r1;
                const bool second = kk + 1 < nk, same = r1 == r0;
                const float q0 = a0[0], v0 = a0[hv], q1 = a1[0], v1 = a1[hv];
                r0 = row_of(x0); r1 = row_of(x1);
                const float cp0 = p0, cd0 = d0, cp1 = p1, cd1 = d1;
                const int k2 = min(kk + 2, QT - 1) * ES, k3 = min(kk + 3, QT - 1) * ES;
                p0 = pcol[k2]; d0 = dcol[k2];
                p1 = pcol[k3]; d1 = dcol[k3];
                x0 = wcol[min(kk + 4, QT - 1) * ES];
                x1 = wcol[min(kk + 5, QT - 1) * ES];
                const float sq0 = q0 + cd0, sv0 = v0 + cp0;
                const float sq1 = (same ? sq0 : q1) + cd1, sv1 = (same ? sv0 : v1) + cp1;
                a0[0] = sq0; a0[hv] = sv0;
                if (second) { a1[0] = sq1; a1[hv] = sv1; }
            }
        } else if (wid >= D && wid < D + NKW && do_k) {
            // histK += ds ; lanes = keys, the planes are read column-wise
            for (int d = 2 * (wid - D); d < 2 * (wid - D) + 2 && d < D; ++d) {
                const bool lo = d < 5;
                const int sh = IDX_BITS * (lo ? d : d - 5);
                const float *drow = s_DS + lane * ES;
                const uint32_t *wrow = (lo ? s_W0 : s_W1) + lane * ES;
                const uint16_t *lut = s_lut + d * pm.lut_stride;
                float *cell = s_hk + lane;
                auto row_of = [&](uint32_t x) { return (int)lut[(x >> sh) & ((1u << IDX_BITS) - 1u)] * QT; };
                int r0 = row_of(wrow[0]), r1 = row_of(wrow[1]);
                uint32_t x0 = wrow[2], x1 = wrow[3];
                float d0 = drow[0], d1 = drow[1];
                for (int qq = 0; qq < nq; qq += 2) {
                    float *a0 = cell + r0, *a1 = cell + r1;
                    const bool second = qq + 1 < nq, same = r1 == r0;
                    const float c0 = a0[0], c1 = a1[0];
                    r0 = row_of(x0); r1 = row_of(x1);
                    const float cd0 = d0, cd1 = d1;
                    d0 = drow[min(qq + 2, QT - 1)];
                    d1 = drow[min(qq + 3, QT - 1)];
                    x0 = wrow[min(qq + 4, QT - 1)];
                    x1 = wrow[min(qq + 5, QT - 1)];
                    const float s0 = c0 + cd0, s1 = (same ? s0 : c1) + cd1;
                    a0[0] = s0;
                    if (second) a1[0] = s1;
                }
            }
        }
        if (wid == GEMM_WARP) {
            uint64_t acc[HP];
            if (do_q) {
#pragma unroll
                for (int i = 0; i < HP; ++i) acc[i] = 0ull;
#pragma unroll 4
                for (int kk = 0; kk < nk; ++kk) axpy_row<HD>(acc, s_DS[kk * ES + lane], s_k + kk * RS);  // dQ[q] = sum_k ds K[k]
                store_row<HD>(s_pg + lane * HD, acc);
            }
            if (do_k) {
#pragma unroll
                for (int i = 0; i < HP; ++i) acc[i] = 0ull;
#pragma unroll 4
                for (int qq = 0; qq < nq; ++qq) axpy_row<HD>(acc, s_DS[lane * ES + qq], s_q + qq * RS);  // dK[k] = sum_q ds Q[q]
                store_row<HD>(s_pg + (64 + lane) * HD, acc);
            }
        } else if (wid == DV_WARP && do_k) {
            uint64_t acc[HP];
#pragma unroll
            for (int i = 0; i < HP; ++i) acc[i] = 0ull;
#pragma unroll 4
            for (int qq = 0; qq < nq; ++qq) axpy_row<HD>(acc, s_P[lane * ES + qq], s_do + qq * RS);      // dV[k] = sum_q p dO[q]
            store_row<HD>(s_pg + (32 + lane) * HD, acc);
        }
        consumer_sync<NT>();
        // ---- rows of the item that are not finite: NaN to the histogram entries of their pairs, zeros in their place (passing
        // over zero entries in the loop below made every item 3.5 % slower, this 1 %) -------------------------------------------
        if (__builtin_expect(odd_rows, 0)) {
            float *rows = s_rows + s * (4 * 32 * RS);
            float *const X[3] = {rows, rows + 32 * RS, rows + 64 * RS}, *const hist[3] = {s_hq, s_hv, s_hk};
#pragma unroll 1
            for (int e = tid; e < 3 * 32 * HD; e += NT) {
                const int tab = e / (32 * HD), v = e / HD & 31;
                if (fabsf(X[tab][v * RS + e % HD]) < INFINITY || !(tab < 2 ? do_q : do_k)) continue;
#pragma unroll 1
                for (int r = 0; r < L.R16; ++r)
                    if (((used >> (r >> 4)) & 1u) && hist[tab][r * QT + v] != 0.f) hist[tab][r * QT + v] = NAN;
            }
            consumer_sync<NT>();
            for (int e = tid; e < 3 * 32 * HD; e += NT) {
                float *x = X[e / (32 * HD)] + (e / HD & 31) * RS + e % HD;
                if (!(fabsf(*x) < INFINITY)) *x = 0.f;
            }
            consumer_sync<NT>();
        }
        // ---- table gradients: lane = row of a 32-row unit ---------------------------------------------------------
        if (dtg < 3 && (dtg < 2 ? do_q : do_k)) {
            const float *hist = dtg == 0 ? s_hq : (dtg == 1 ? s_hv : s_hk);
            const float *X = dtg == 0 ? s_q : (dtg == 1 ? s_do : s_k);
            bool on[NDT], any[NDT];
            const float *hrow[NDT];
#pragma unroll
            for (int u = 0; u < NDT; ++u) {
                const int tile = 2 * (dsub + DTW * u) + (lane >> 4);
                on[u] = tile < n_mt && ((used >> tile) & 1u);
                any[u] = __any_sync(0xffffffffu, on[u]);
                hrow[u] = hist + (on[u] ? (dsub + DTW * u) * 32 + lane : 0) * QT;
            }
            constexpr int STEP = D == 9 && HD == 16 ? 1 : 2;       // two rows of 16 channels ahead spill beside three units
            for (int i = 0; i < QT; i += STEP) {
                uint64_t x[STEP][HP];
#pragma unroll
                for (int j = 0; j < STEP; ++j) load_row<HD>(x[j], X + ((i + j + lane) & 31) * RS);
#pragma unroll
                for (int u = 0; u < NDT; ++u)
                    if (any[u]) {
#pragma unroll
                        for (int j = 0; j < STEP; ++j) {
                            const float h = on[u] ? hrow[u][(i + j + lane) & 31] : 0.f;
                            const uint64_t hh = dup2(h);
#pragma unroll
                            for (int c = 0; c < HP; ++c) dt_acc[u][c] = fma2(hh, x[j][c], dt_acc[u][c]);
                        }
                    }
            }
        }
        // ---- dQ += histQ.Tq, dK += histK.Tk: lane = voxel -----------------------------------------------------------
        if (side < 2 && (side == 0 ? do_q : do_k)) {
            const float *T = side == 0 ? P.tq : P.tk, *hist = side == 0 ? s_hq : s_hk;
            const bool odd_table = s_odd[1 + side];
            uint64_t acc[HP];
#pragma unroll
            for (int i = 0; i < HP; ++i) acc[i] = 0ull;
            TableTile<HD> tile;
            tc::UsedTiles tiles(used, n_mt, ws2, SG);
            int mt = tiles.next();
            if (mt >= 0) tile.fetch(T, HC, co, s_map, mt, lane);
            while (mt >= 0) {
                __syncwarp();
                tile.put(st, lane);
                __syncwarp();
                const int nx = tiles.next();
                if (nx >= 0) tile.fetch(T, HC, co, s_map, nx, lane);
                const float *h = hist + mt * 16 * QT + lane;
                if (__builtin_expect(odd_table, 0)) {
#pragma unroll 1
                    for (int r = 0; r < 16; ++r)
                        if (h[r * QT] != 0.f) axpy_row<HD>(acc, h[r * QT], st + r * HD);
                } else {
#pragma unroll 4
                    for (int r = 0; r < 16; ++r) axpy_row<HD>(acc, h[r * QT], st + r * HD);
                }
                mt = nx;
            }
            store_row<HD>(s_part + ((side * SG + ws2) * 32 + lane) * HD, acc);
        }
        consumer_sync<NT>();
        // ---- reduce and store ---------------------------------------------------------------------------------------
        for (int e = tid; e < 2 * 32 * HP; e += NT) {
            const int sd = e / (32 * HP), xx = e / HP & 31, ch = e % HP * 2;
            if (sd == 0 ? do_q && xx < nq : do_k && xx < nk) {
                const float2 pg = *reinterpret_cast<const float2 *>(s_pg + ((sd == 0 ? 0 : 64) + xx) * HD + ch);
                float a = pg.x, b = pg.y;
                const float *pp = s_part + (sd * SG * 32 + xx) * HD + ch;
#pragma unroll
                for (int ww = 0; ww < SG; ++ww) {
                    const float2 pr = *reinterpret_cast<const float2 *>(pp + ww * 32 * HD);
                    a += pr.x;
                    b += pr.y;
                }
                const bool add = sd == 0 ? add_q : add_k;
                const int64_t o = (int64_t)(sd == 0 ? s_rowq : s_rowk)[xx] * HC + co + ch;
                float2 *dst = reinterpret_cast<float2 *>((sd == 0 ? P.dq : P.dk) + o);
                if (add) {                                     // a later share of a large window
                    const float2 old = *dst;
                    a += old.x;
                    b += old.y;
                }
                *dst = make_float2(a, b);
                if (sd == 1) {
                    float2 dvv = *reinterpret_cast<const float2 *>(s_pg + (32 + xx) * HD + ch);
                    float2 *dst_v = reinterpret_cast<float2 *>(P.dv + o);
                    if (add) {
                        const float2 old = *dst_v;
                        dvv.x += old.x;
                        dvv.y += old.y;
                    }
                    *dst_v = dvv;
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty + s);
    }

    // ---- the table gradients of this block ---------------------------------------------------------------------------
    if (dtg < 3 && it > 0) {
        float *dst = dtg == 0 ? P.dtq : (dtg == 1 ? P.dtv : P.dtk);
#pragma unroll
        for (int u = 0; u < NDT; ++u) {
            const int r = (dsub + DTW * u) * 32 + lane;
            const int row = r < L.R16 ? s_map[r] : 0xffff;      // aliases go to the row they stand for
            if (row != 0xffff) {
                float f[HD];
                store_row<HD>(f, dt_acc[u]);
                float4 *p = reinterpret_cast<float4 *>(dst + (int64_t)row * HC + co);
#pragma unroll
                for (int i = 0; i < HD / 4; ++i) atomicAdd(p + i, make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]));
            }
        }
    }
}

template <int D, int HD>
static int launch(const Params &p, const CrseMeta &meta, const PermMeta &pm, cudaStream_t st)
{
    constexpr int NW = warps_for(D, HD);
    const Smem L = make_smem<D, HD>(pm.R, pm.D * pm.lut_stride);
    auto kern = attn_bwd_f32_kernel<D, HD>;
    int sms = 0;
    const int rc = tc::kernel_setup(reinterpret_cast<const void *>(kern), sms);
    if (rc != S3D_OK) return rc;
    int gx = sms / p.H;
    if (gx < 1) gx = 1;
    kern<<<dim3((unsigned)gx, (unsigned)p.H), (NW + 1) * 32, L.total, st>>>(p, pm, tc::make_pair_consts(meta));
    const cudaError_t le = cudaGetLastError();
    note_cuda_error(le);
    return le == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}

template <int D, int HD>
static bool fits(const PermMeta &pm)
{
    const int n_mt = (pm.R + 15) / 16;                       // the tile mask is one word
    return n_mt <= 32 && (n_mt + 1) / 2 <= Split<D, HD>::NDT * Split<D, HD>::DTW &&
           make_smem<D, HD>(pm.R, pm.D * pm.lut_stride).total <= 227 * 1024;
}

}  // namespace f32

bool attn_f32_bwd_supported(const AttnArgs &a)
{
    if (a.dtype != S3D_F32 || (a.hd != 8 && a.hd != 16)) return false;
    for (int d = 0; d < a.meta.D; ++d)
        if (a.meta.L[d] >= (1 << tc::IDX_BITS)) return false;
    const tc::PermMeta pm = tc::make_perm_meta(a.meta);
    switch (a.meta.D) {
        case 3: return a.hd == 8 ? f32::fits<3, 8>(pm) : f32::fits<3, 16>(pm);
        case 6: return a.hd == 8 ? f32::fits<6, 8>(pm) : f32::fits<6, 16>(pm);
        case 9: return a.hd == 8 ? f32::fits<9, 8>(pm) : f32::fits<9, 16>(pm);
        default: return false;
    }
}

// dtq, dtk, dtv must be zero on entry (accumulated into).
int attn_f32_backward(const AttnArgs &a, cudaStream_t st)
{
    if (a.W == 0) return S3D_OK;
    const tc::PermMeta pm = tc::make_perm_meta(a.meta);
    f32::Params p{};
    p.q = (const float *)a.q; p.k = (const float *)a.k; p.v = (const float *)a.v;
    p.dout = (const float *)a.dout; p.o = (const float *)a.out; p.lse = a.lse;
    p.tq = (const float *)a.tq; p.tk = (const float *)a.tk; p.tv = (const float *)a.tv;
    p.dq = (float *)a.dq; p.dk = (float *)a.dk; p.dv = (float *)a.dv;
    p.dtq = a.dtq; p.dtk = a.dtk; p.dtv = a.dtv;
    p.w_sizes = a.w_sizes; p.w2n = a.w2n; p.n2n = a.n2n; p.n_coords = a.n_coords;
    p.W = a.W; p.H = a.H;
#define S3D_F32_BWD(DD) return a.hd == 8 ? f32::launch<DD, 8>(p, a.meta, pm, st) : f32::launch<DD, 16>(p, a.meta, pm, st)
    switch (a.meta.D) {
        case 3: S3D_F32_BWD(3);
        case 6: S3D_F32_BWD(6);
        case 9: S3D_F32_BWD(9);
        default: return S3D_ERR_UNSUPPORTED;
    }
#undef S3D_F32_BWD
}

cudaError_t attn_f32_bwd_async_error(bool &set) { return take_async_error(set); }

}  // namespace s3d
