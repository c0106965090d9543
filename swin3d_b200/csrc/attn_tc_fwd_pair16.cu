// Forward of the cRSE window attention for head_dim 16 with an even head count (fp16), windows of any size.
//
// A window of n voxels is cut into nt = ceil(n / 32) tiles of equal size.  A block takes query tiles (window, i) and runs
// over the key tiles j of their window: every tile pair is an independent 32 x 32 problem, as in the backward
// (attn_tc_bwd_pair16.cu), with its own row maximum; a thread of the store phase keeps four output channels of one query
// in registers and merges the tile pairs' (maximum, sum, output) as they come.  P_q is projected again for every key
// tile, which lets the histogram reuse its storage.
//
// Per tile pair, phases separated by a barrier of the consumer warps:
//   project    P_q = Tq.Q^T (lane-major), P_k = Tk.K^T (key-major), S0 = K.Q^T                            [tensor cores]
//   scores     lane = query, keys dealt to the warps: D indices, 2*D look-ups; row maxima by shared atomics
//   softmax    p, row sums, pair entries (p, idx 0-4) and (idx 5-8, p); clear the histogram
//   histogram  warp d: hist[row][q] += p for dimension d; warp D: P.V                                      [tensor cores]
//   products   += hist.Tv, row tiles dealt to the warps                                                   [tensor cores]
//   merge      reduce over the warps, merge, store after the last key tile
// Rows are numbered and row tiles skipped as in the backward (PermMeta); the producer lists the used tiles.  The three
// tables of the pair of heads stand in shared memory in the order in which the lanes of an mma take them (71 KB at 23 row
// tiles; fetched from L1/L2 for every item through the row map, a tile ahead, the projections took 4.7 k cycles of an
// item's 18 k and the products 6.8 k).
//
// The blocks take contiguous ranges of (window, query tile) units of equal cost, so that the deep stages -- a handful of
// windows of some hundred voxels -- still spread over the GPU.
// Bound: instruction issue (half of the slots, four warps a scheduler) and the barriers.  A forward call, tiled kernel with an
// online softmax that did the work of a query tile once / this one with tables from L1/L2 / now: 144 k voxels, 10 heads,
// 2.8 key tiles per query tile 3.85 / 3.79 / 3.08 ms; 8 k voxels, 20 heads, 4.5 key tiles 611 / 732 / 588 us, three signal
// dimensions 383 / 516 / 381 us; 4 windows of up to 150 voxels, 24 heads 108 / 62 / 60 us.
#include <climits>

#include "attn_kernels.cuh"
#include "attn_tc.cuh"
#include "attn_tc_pair16.cuh"
#include "attn_tc_small.cuh"
#include "async_stage.cuh"

namespace s3d {
namespace tc {

constexpr int F16_STAGES = 2;
__host__ __device__ constexpr int f16_warps(int D) { return 15; }   // with the producer, four warps per scheduler

// Warps of the hist.Tv products: their partial outputs (4 KB each) go where P_k was.
template <int D>
struct F16Split {
    static constexpr int NW = f16_warps(D);
    static constexpr int NHT = D == 9 ? 12 : (D == 6 ? 9 : 6);
};

struct F16Smem {
    int R16, Rp;
    int off_pq, off_pk, off_e, off_rows, off_c, off_ta, off_tb, off_lut, off_map, off_misc, total;
};

template <int D>
__host__ __device__ inline F16Smem make_f16_layout(int R, int lut_entries)
{
    F16Smem L;
    L.R16 = (R + 15) / 16 * 16;
    L.Rp = (L.R16 + 15) / 16 * 16 + 4;                               // see p16_store_key_major
    int off = 0;
    L.off_pq = off; off += L.R16 * QT * 4 > 8192 ? L.R16 * QT * 4 : 8192;          // P_q, later the histogram
    const int pk = 32 * L.Rp * 4, part = F16Split<D>::NHT * 4096;
    L.off_pk = off; off += pk > part ? pk : part;                    // P_k, later the partial outputs
    L.off_e = off; off += 2 * 32 * ES * 8;                           // pair entries, two planes; S0 before
    L.off_rows = off; off += F16_STAGES * 3 * 32 * P16_RS * 2;       // Q (query tile), K, V (key tile), per stage
    L.off_c = off; off += F16_STAGES * 2 * 32 * 12 * 4;
    L.off_ta = off; off += 2 * (L.R16 / 16) * 1024;                  // Tq and Tk as operands of the projections
    L.off_tb = off; off += (L.R16 / 16) * 1024;                      // Tv as operand of the products
    L.off_lut = off; off += (lut_entries * 2 + 15) / 16 * 16;
    L.off_map = off; off += (L.R16 * 2 + 15) / 16 * 16;
    L.off_misc = off; off += 6144;
    L.total = off;
    return L;
}

struct F16Params {
    const __half *q, *k, *v, *tq, *tk, *tv;
    __half *out;
    float *lse;
    const int32_t *w_sizes, *w2n, *n2n;
    const float *n_coords;
    int64_t W;
    int H;
    Mirrors m_out;
};

template <int D>
__global__ void __launch_bounds__((f16_warps(D) + 1) * 32, 1)
attn_fwd_pair16_kernel(const __grid_constant__ F16Params P, const PermMeta pm, const PairConsts pc)
{
    constexpr int NW = f16_warps(D), NT = NW * 32;
    constexpr int NHT = F16Split<D>::NHT;        // warps of the hist.Tv products; P.V belongs to one of them
    constexpr int PV_WARP = D;
    static_assert(D < NHT && NHT <= NW, "P.V needs a warp of its own");
    constexpr int HALF = NW / 2;                 // warps per projection table
    constexpr int KPW = (QT + NW - 1) / NW;      // keys per warp in the score phase
    constexpr int RS = P16_RS, ROWS = 32 * RS;
    extern __shared__ __align__(16) unsigned char smem[];
    const F16Smem L = make_f16_layout<D>(pm.R, pm.D * pm.lut_stride);
    uint32_t *s_pq = reinterpret_cast<uint32_t *>(smem + L.off_pq), *s_hist = s_pq;
    uint32_t *s_pk = reinterpret_cast<uint32_t *>(smem + L.off_pk);
    uint2 *s_elo = reinterpret_cast<uint2 *>(smem + L.off_e);        // [32][ES] (p, idx 0-4); S0 before
    uint2 *s_ehi = s_elo + 32 * ES;                                  // [32][ES] (idx 5-8, p)
    float *s_part = reinterpret_cast<float *>(smem + L.off_pk);      // [NHT][32][32]
    __half *s_rows = reinterpret_cast<__half *>(smem + L.off_rows);  // [stage][Q,K,V][32][RS]
    float *s_cs = reinterpret_cast<float *>(smem + L.off_c);         // [stage][query tile, key tile][32][12]
    uint4 *s_ta = reinterpret_cast<uint4 *>(smem + L.off_ta);        // [Tq, Tk][row tile][2][lane]
    uint4 *s_tb = reinterpret_cast<uint4 *>(smem + L.off_tb);        // [row tile][2][lane]
    uint16_t *s_lut = reinterpret_cast<uint16_t *>(smem + L.off_lut);
    uint16_t *s_map = reinterpret_cast<uint16_t *>(smem + L.off_map);
    float *s_max = reinterpret_cast<float *>(smem + L.off_misc);     // [32][2]
    float *s_lsum = s_max + 64;                                      // [NW][32][2]
    int *s_rowi = reinterpret_cast<int *>(s_lsum + 16 * 64);         // [stage][32] rows of the query tile
    int *s_n = s_rowi + F16_STAGES * 32;                             // [stage][8]: nq, nk, first key tile, last key tile, used tiles, stop
    int *s_fail = s_n + F16_STAGES * 8;
    uint8_t *s_tiles = reinterpret_cast<uint8_t *>(s_fail + 1);      // [stage][32] the used tiles in order
    uint64_t *s_full = reinterpret_cast<uint64_t *>(smem + L.off_misc + 6144 - 64), *s_empty = s_full + F16_STAGES;

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int hp = blockIdx.y, H = P.H, HC = H * 16, co = hp * 32;

    if (tid == 0) {
        for (int s = 0; s < F16_STAGES; ++s) {
            mbar_init(s_full + s, 64);         // every producer lane: its stores, its copies
            mbar_init(s_empty + s, NW);
        }
        *s_fail = 0;
        mbar_init_fence();
    }
    fill_perm_lut(s_lut, pm, tid, blockDim.x);
    for (int r = tid; r < L.R16; r += blockDim.x) {
        const int row = perm_table_row(pm, r);
        s_map[r] = row < 0 ? (uint16_t)0xffff : (uint16_t)row;
    }
    __syncthreads();
    // the tables of this pair of heads, in the order the lanes of an mma take them
    const int g = lane >> 2, t = lane & 3, n_mt = L.R16 / 16;
    for (int u = wid; u < 3 * n_mt; u += NW + 1) {
        const int tab = u / n_mt, mt = u - tab * n_mt;
        if (tab < 2) {
            P16TileA a;
            a.fetch(tab == 0 ? P.tq : P.tk, HC, co, s_map, mt, g, t);
            uint4 *o = s_ta + u * 64 + lane;
            o[0] = make_uint4(a.f[0][0].x, a.f[0][0].y, a.f[0][1].x, a.f[0][1].y);
            o[32] = make_uint4(a.f[1][0].x, a.f[1][0].y, a.f[1][1].x, a.f[1][1].y);
        } else {
            P16TileB raw;
            raw.fetch(P.tv, HC, co, s_map, mt, g, t);
            const P16FragB f(raw);
            uint4 *o = s_tb + mt * 64 + lane;
            o[0] = make_uint4(f.b[0][0][0], f.b[0][0][1], f.b[0][1][0], f.b[0][1][1]);
            o[32] = make_uint4(f.b[1][0][0], f.b[1][0][1], f.b[1][1][0], f.b[1][1][1]);
        }
    }
    int64_t w_begin, w_end;
    int i_begin, i_end;                          // first query tile of window w_begin, one past the last of window w_end
    balanced_units<(NW + 1) * 32>(P.w_sizes, P.W, smem + L.off_pq, UnitsPerQueryTile{1, INT_MAX}, w_begin, w_end, i_begin, i_end);

    if (wid == NW) {
        // ================================ producer warp ================================================
        int64_t w = w_begin - 1;
        int n = 0, base = 0, nt = 0, ts = 0, ti = 0, tj = 0, ti_end = 0;
        int n_nx = 0, base_nx = 0;
        if (w_begin < P.W) {
            n_nx = __ldg(P.w_sizes + w_begin);
            base_nx = __ldg(P.w2n + w_begin);
        }
        bool have = false;
        int nq = 0, nk = 0, rowq = 0, rowk = 0;
        float cq[D], ck[D];
        auto advance = [&]() {
            if (have && tj + 1 < nt) {
                ++tj;
            } else if (have && ti + 1 < ti_end) {
                ++ti;
                tj = 0;
            } else {
                do {                              // the range may end inside window w_end, and begin inside w_begin
                    ++w;
                    have = w < w_end || (w == w_end && i_end > 0);
                    if (have) {
                        n = n_nx;
                        base = base_nx;
                        if (w + 1 < P.W) {
                            n_nx = __ldg(P.w_sizes + w + 1);
                            base_nx = __ldg(P.w2n + w + 1);
                        }
                        nt = (n + QT - 1) / QT;
                        ts = nt > 0 ? (n + nt - 1) / nt : 0;
                        ti = w == w_begin ? i_begin : 0;
                        ti_end = w == w_end ? i_end : nt;
                        tj = 0;
                    }
                } while (have && ti >= ti_end);
            }
            nq = have ? max(min(ts, n - ti * ts), 0) : 0;
            nk = have ? max(min(ts, n - tj * ts), 0) : 0;
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
            const uint32_t used = item_tile_mask<D>(cq, ck, nq, nk, s_lut, pm, pc, lane) & (n_mt < 32 ? (1u << n_mt) - 1u : 0xffffffffu);
            const int s = it % F16_STAGES;
            bool stop = !have;
            if (it >= F16_STAGES && !mbar_wait(s_empty + s, ((it / F16_STAGES) - 1) & 1)) {
                g_async_error = 1;
                stop = true;                      // tell the consumers to stop
            }
            if (stop) nq = nk = 0;
            __half *rq = s_rows + s * (3 * ROWS);
            float *cs = s_cs + s * 768;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                cs[lane * 12 + d] = cq[d];
                cs[384 + lane * 12 + d] = ck[d];
            }
            s_rowi[s * 32 + lane] = rowq;
            if ((used >> lane) & 1u) s_tiles[s * 32 + __popc(used & ((1u << lane) - 1u))] = (uint8_t)lane;
            if (lane == 0) {
                s_n[s * 8] = nq;
                s_n[s * 8 + 1] = nk;
                s_n[s * 8 + 2] = tj == 0;
                s_n[s * 8 + 3] = tj + 1 == nt;
                s_n[s * 8 + 4] = (int)used;
                s_n[s * 8 + 5] = stop;
            }
            mbar_arrive(s_full + s);
            stage_rows<4>(rq, RS, P.q + co, HC, rowq, nq, lane);
            stage_rows<4>(rq + ROWS, RS, P.k + co, HC, rowk, nk, lane);
            stage_rows<4>(rq + 2 * ROWS, RS, P.v + co, HC, rowk, nk, lane);
            mbar_arrive_cp_async(s_full + s);
            if (stop) break;
            advance();
        }
        return;
    }

    // ==================================== consumer warps ===============================================
    const int Rp = L.Rp;
    const int mypos = qpos(lane);
    constexpr float LOG2E = 1.4426950408889634f;
    const int pside = wid / HALF, wsub = wid - pside * HALF;         // projections: 0 = Tq with Q, 1 = Tk with K
    // the store phase: this thread's query and four channels, merged over the key tiles
    const int xx = tid >> 3, ch = (tid & 7) * 4, hh = ch >> 4;
    float4 o_run = make_float4(0.f, 0.f, 0.f, 0.f);
    float m_run = 0.f, l_run = 0.f;

    for (int it = 0;; ++it) {
        const int s = it % F16_STAGES;
        if (!mbar_wait(s_full + s, (it / F16_STAGES) & 1)) {
            *s_fail = 1;
            g_async_error = 2;
        }
        consumer_sync<NT>();          // the previous item's merge is over; the flag is settled
        const int nq = s_n[s * 8], nk = s_n[s * 8 + 1];
        const bool first = s_n[s * 8 + 2] != 0, last = s_n[s * 8 + 3] != 0;
        const uint32_t used = (uint32_t)s_n[s * 8 + 4];
        const int n_used = __popc(used);
        const uint8_t *tiles = s_tiles + s * 32;
        if (s_n[s * 8 + 5] || *s_fail) break;
        const __half *s_q = s_rows + s * (3 * ROWS), *s_k = s_q + ROWS, *s_v = s_k + ROWS;
        const float *s_c = s_cs + s * 768, *s_ck = s_c + 384;
        if (tid < 64) s_max[tid] = -INFINITY;
        // ---- projections, S0 ------------------------------------------------------------------------------------
        if (pside < 2) {
            const int nv = pside == 0 ? nq : nk;
            uint2 bf[4][2];
            p16_feat_frag(bf, pside == 0 ? s_q : s_k, nv, g, t);
#pragma unroll 1
            for (int i = wsub; i < n_used; i += HALF) {
                const int mt = tiles[i];
                const uint4 *f = s_ta + (pside * n_mt + mt) * 64 + lane;
                const uint4 x = f[0], y = f[32];
                P16TileA cur;
                cur.f[0][0] = make_uint2(x.x, x.y); cur.f[0][1] = make_uint2(x.z, x.w);
                cur.f[1][0] = make_uint2(y.x, y.y); cur.f[1][1] = make_uint2(y.z, y.w);
                uint32_t d[2][2][4];
                p16_project(d, cur, bf, nv);
                if (pside == 0) p16_store_lane_major(s_pq, d, mt, g, t);
                else p16_store_key_major(s_pk, d, mt, Rp, nv, g, t);
            }
        }
        for (int u = NW - 1 - wid; u < 8; u += NW) {
            const int mt = u >> 2, j = u & 3;       // key rows 16mt.., query columns 8j..
            if (16 * mt < nk && 8 * j < nq) {
                float c[2][2][2];
                p16_dot_block(c, s_k, 16 * mt, s_q, 8 * j, g, t);
#pragma unroll
                for (int rr = 0; rr < 2; ++rr)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        *reinterpret_cast<float2 *>(s_elo + (16 * mt + g + 8 * rr) * ES + 8 * j + 2 * t + e) = make_float2(c[rr][e][0], c[rr][e][1]);
            }
        }
        consumer_sync<NT>();
        // ---- scores: keys wid, wid + NW, ... ; lane = query -----------------------------------------------------
        float cx[D];
        load_coords12<D>(s_c + lane * 12, cx);
        float sreg[KPW][2];
        uint32_t wreg[KPW][2];
        float mloc0 = -INFINITY, mloc1 = -INFINITY;
        const uint32_t *pq_lane = s_pq + mypos;
#pragma unroll
        for (int j = 0; j < KPW; ++j) {
            const int kk = wid + NW * j;
            sreg[j][0] = sreg[j][1] = 0.f;
            wreg[j][0] = wreg[j][1] = 0u;
            if (kk < nk) {
                float ck[D];
                load_coords12<D>(s_ck + kk * 12, ck);
                const uint32_t *pk_row = s_pk + kk * Rp;
                __half2 bq = __float2half2_rn(0.f), bk = bq;
                uint32_t w0 = 0, w1 = 0;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const uint32_t idx = crse_index_pc(cx[d], ck[d], pc.half[d], pc.clamp[d]);
                    const uint32_t row = s_lut[d * pm.lut_stride + idx];
                    bq = __hadd2(bq, u32_as_h2(pq_lane[row * QT]));
                    bk = __hadd2(bk, u32_as_h2(pk_row[row]));
                    if (d < 5) w0 |= idx << (IDX_BITS * d);
                    else w1 |= idx << (IDX_BITS * (d - 5));
                }
                const float2 s0 = *reinterpret_cast<const float2 *>(s_elo + kk * ES + lane);
                const float2 b = __half22float2(__hadd2(bq, bk));
                sreg[j][0] = s0.x + b.x;
                sreg[j][1] = s0.y + b.y;
                wreg[j][0] = w0;
                wreg[j][1] = w1;
                mloc0 = fmaxf(mloc0, sreg[j][0]);
                mloc1 = fmaxf(mloc1, sreg[j][1]);
            }
        }
        if (wid < nk) {
            atomic_max_float(s_max + lane * 2, mloc0);
            atomic_max_float(s_max + lane * 2 + 1, mloc1);
        }
        consumer_sync<NT>();
        // ---- probabilities, pair entries; clear the histogram (P_q is dead) -----------------------------------------
        {
            const float m0 = s_max[lane * 2] * LOG2E, m1 = s_max[lane * 2 + 1] * LOG2E;
            float l0 = 0.f, l1 = 0.f;
#pragma unroll
            for (int j = 0; j < KPW; ++j) {
                const int kk = wid + NW * j;
                if (kk < QT) {
                    uint32_t ph = 0u;                         // zero for keys beyond the tile: P.V reads whole 16-key steps
                    if (kk < nk && lane < nq) {
                        const float p0 = ex2_approx(fmaf(sreg[j][0], LOG2E, -m0));
                        const float p1 = ex2_approx(fmaf(sreg[j][1], LOG2E, -m1));
                        l0 += p0;
                        l1 += p1;
                        ph = h2_as_u32(__floats2half2_rn(p0, p1));
                    }
                    s_elo[kk * ES + lane] = make_uint2(ph, wreg[j][0]);
                    s_ehi[kk * ES + lane] = make_uint2(wreg[j][1], ph);
                }
            }
            s_lsum[(wid * QT + lane) * 2] = l0;
            s_lsum[(wid * QT + lane) * 2 + 1] = l1;
        }
        for (int i = tid; i < L.R16 * QT / 4; i += NT)
            if ((used >> (i >> 7)) & 1u) reinterpret_cast<uint4 *>(s_hist)[i] = make_uint4(0, 0, 0, 0);
        consumer_sync<NT>();
        // ---- histogram (warp d: signal dimension d) | P.V -----------------------------------------------------------
        float acc[2][2][2][4];
        p16_zero(acc);
        if (wid < D) {
            const int d = wid;
            const bool lo = d < 5;
            const int sh = IDX_BITS * (lo ? d : d - 5);
            // the half of a pair entry this dimension needs: (p, idx 0-4) or (idx 5-8, p)
            const uint2 *ecol = (lo ? s_elo : s_ehi) + lane;
            const uint16_t *lut = s_lut + d * pm.lut_stride;
            uint32_t *cell = s_hist + mypos;
            auto row_of = [&](uint2 e) { return (uint32_t)lut[((lo ? e.y : e.x) >> sh) & ((1u << IDX_BITS) - 1u)] * QT; };
            // the rows of this step are known; its cells, the rows of the next step and the entries after that are
            // fetched together (keys beyond the tile hold zero entries)
            uint2 e0 = ecol[0], e1 = ecol[ES];
            uint32_t r0 = row_of(e0), r1 = row_of(e1);
            uint32_t p0 = lo ? e0.x : e0.y, p1 = lo ? e1.x : e1.y;
            e0 = ecol[2 * ES];
            e1 = ecol[3 * ES];
            for (int kk = 0; kk < nk; kk += 2) {
                uint32_t *a0 = cell + r0, *a1 = cell + r1;
                const uint32_t c0 = *a0, c1 = *a1;
                const bool same = r1 == r0, second = kk + 1 < nk;
                const __half2 h0 = u32_as_h2(p0), h1 = u32_as_h2(p1);
                r0 = row_of(e0);
                r1 = row_of(e1);
                p0 = lo ? e0.x : e0.y;
                p1 = lo ? e1.x : e1.y;
                e0 = ecol[min(kk + 4, QT - 1) * ES];
                e1 = ecol[min(kk + 5, QT - 1) * ES];
                const __half2 s0 = __hadd2(u32_as_h2(c0), h0), s1 = __hadd2(same ? s0 : u32_as_h2(c1), h1);
                *a0 = h2_as_u32(s0);
                if (second) *a1 = h2_as_u32(s1);
            }
        }
        if (wid == PV_WARP) p16_pair_gemm<false, 2>(acc, reinterpret_cast<const uint32_t *>(s_elo), s_v, nk, g, t);   // O[q] = sum_k p V[k]
        consumer_sync<NT>();
        // ---- O += hist . Tv ---------------------------------------------------------------------------------------
        if (wid < NHT) {
#pragma unroll 1
            for (int i = wid; i < n_used; i += NHT) {
                const int ks = tiles[i];
                const uint4 *f = s_tb + ks * 64 + lane;
                p16_hist_t(acc, s_hist, P16FragB(f[0], f[32]), ks, lane, g, t);
            }
            p16_store(s_part + wid * 1024, acc, g, t);       // P_k is dead since the scores
        }
        consumer_sync<NT>();
        // ---- reduce, merge with the earlier key tiles, store after the last -------------------------------------------
        if (tid < 256 && xx < nq) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            float ls = 0.f;
#pragma unroll
            for (int ww = 0; ww < NHT; ++ww) {
                const float4 pr = *reinterpret_cast<const float4 *>(s_part + ww * 1024 + xx * 32 + ch);
                a.x += pr.x; a.y += pr.y; a.z += pr.z; a.w += pr.w;
            }
#pragma unroll
            for (int ww = 0; ww < NW; ++ww) ls += s_lsum[(ww * QT + xx) * 2 + hh];
            const float mt = s_max[xx * 2 + hh];
            float m = mt;
            if (!first) {
                m = fmaxf(m_run, mt);
                const float f0 = ex2_approx((m_run - m) * LOG2E), f1 = ex2_approx((mt - m) * LOG2E);
                a.x = o_run.x * f0 + a.x * f1; a.y = o_run.y * f0 + a.y * f1;
                a.z = o_run.z * f0 + a.z * f1; a.w = o_run.w * f0 + a.w * f1;
                ls = l_run * f0 + ls * f1;
            }
            if (last) {
                const float inv = 1.f / ls;
                const int64_t row = s_rowi[s * 32 + xx];
                const int64_t off = row * HC + co + ch;
                const uint2 r = make_uint2(h2_as_u32(__floats2half2_rn(a.x * inv, a.y * inv)), h2_as_u32(__floats2half2_rn(a.z * inv, a.w * inv)));
                *reinterpret_cast<uint2 *>(P.out + off) = r;
                for (int i = 0; i < P.m_out.n; ++i) *reinterpret_cast<uint2 *>(static_cast<__half *>(P.m_out.p[i]) + off) = r;
                if ((ch & 15) == 0) P.lse[row * H + 2 * hp + hh] = m + __logf(ls);
            } else {
                o_run = a;
                m_run = m;
                l_run = ls;
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty + s);
    }
}

template <int D>
static int launch_fwd_pair16(const F16Params &p, const CrseMeta &meta, const PermMeta &pm, cudaStream_t st)
{
    static_assert(f16_warps(D) * 32 >= 256, "the merge keeps one entry per thread");
    const F16Smem L = make_f16_layout<D>(pm.R, pm.D * pm.lut_stride);
    auto kern = attn_fwd_pair16_kernel<D>;
    int sms = 0;
    const int rc = kernel_setup(reinterpret_cast<const void *>(kern), sms);
    if (rc != S3D_OK) return rc;
    const int hp = p.H / 2;
    int gx = sms / hp;
    if (gx < 1) gx = 1;
    kern<<<dim3((unsigned)gx, (unsigned)hp), (f16_warps(D) + 1) * 32, L.total, st>>>(p, pm, make_pair_consts(meta));
    const cudaError_t le = cudaGetLastError();
    note_cuda_error(le);
    return le == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}

}  // namespace tc

bool attn_tc_fwd_pair16_supported(const AttnArgs &a)
{
    if (a.dtype != S3D_F16 || a.hd != 16 || (a.H & 1)) return false;
    for (int d = 0; d < a.meta.D; ++d)
        if (a.meta.L[d] >= (1 << tc::IDX_BITS)) return false;
    const tc::PermMeta pm = tc::make_perm_meta(a.meta);
    if ((pm.R + 15) / 16 > 32) return false;                 // the tile mask is one word
    const int lut = pm.D * pm.lut_stride;
    const int total = a.meta.D == 3 ? tc::make_f16_layout<3>(pm.R, lut).total
                                    : (a.meta.D == 6 ? tc::make_f16_layout<6>(pm.R, lut).total : tc::make_f16_layout<9>(pm.R, lut).total);
    return total <= 227 * 1024;
}

int attn_tc_forward_pair16(const AttnArgs &a, cudaStream_t st)
{
    if (a.W == 0) return S3D_OK;
    const tc::PermMeta pm = tc::make_perm_meta(a.meta);
    tc::F16Params p{};
    p.q = (const __half *)a.q; p.k = (const __half *)a.k; p.v = (const __half *)a.v;
    p.tq = (const __half *)a.tq; p.tk = (const __half *)a.tk; p.tv = (const __half *)a.tv;
    p.out = (__half *)a.out; p.lse = a.lse;
    p.w_sizes = a.w_sizes; p.w2n = a.w2n; p.n2n = a.n2n; p.n_coords = a.n_coords;
    p.W = a.W; p.H = a.H;
    p.m_out = a.m_out;
    switch (a.meta.D) {
        case 3: return tc::launch_fwd_pair16<3>(p, a.meta, pm, st);
        case 6: return tc::launch_fwd_pair16<6>(p, a.meta, pm, st);
        case 9: return tc::launch_fwd_pair16<9>(p, a.meta, pm, st);
        default: return S3D_ERR_UNSUPPORTED;
    }
}

cudaError_t attn_tc_fwd_pair16_async_error(bool &set) { return take_async_error(set); }

}  // namespace s3d
