// Backward of the cRSE window attention for head_dim 16 with an even head count (fp16), windows of any
// size: the single-sweep tile-pair scheme of attn_tc_bwd_small.cu with two heads of 16 channels per block.
//
// The look-ups, histograms and pair planes are those of a head_dim-8 pair (half2 = two heads); only the
// products see the 16 channels (attn_tc_pair16.cuh).
//
// What does not fit beside 24 row tiles of projections (148 KB) stays outside shared memory: the table
// operands are fetched per tile from L1/L2, one tile ahead, and the table gradients of a block (24 tiles x
// 3 tables x 32 channels in fp32 = 147 KB, more than the registers left) live in local memory, which
// L2 holds; a warp touches the tiles an item uses, 16 bytes per lane and access.  The gradients run on
// 3 warps per table, the hist.T products on the others at the same time.
//
// Bound: instruction issue and shared-memory wavefronts of the look-ups and histograms (half of the slots, three quarters of
// the L1 pipe), then latency between the barriers.  Against the two-sweep kernels of attn_tc_bwd.cu (scores twice, no tile
// skipping), forward and backward of 144 k voxels, 10 heads: 16.8 -> 9.4 ms; 8 k voxels, 20 heads, 4.5 key tiles per query
// tile: 2.63 -> 2.15 ms.
#include "attn_kernels.cuh"
#include "attn_tc.cuh"
#include "attn_tc_pair16.cuh"
#include "attn_tc_small.cuh"
#include "async_stage.cuh"

namespace s3d {
namespace tc {

constexpr int P16_STAGES = 2;

// Windows of up to P16_SLOTS tiles (7^3 cells are 11) run over their tile pairs (i, j) once, j innermost: dQ of a query
// tile is complete after its last key tile, dK and dV of every key tile with the last query tile.  Until then the thread
// that stores a row piece keeps its sum in fp32, for dK and dV one per key tile (local memory: 0.7 KB a thread, L1 and L2
// hold it; rows in fp16 that every pair adds to were as fast and cost half the precision: 6.0 against 3.8e-4 of the norm
// for windows of 343 voxels).  Larger windows run over their pairs twice, for dQ (and dTq, dTv) with j innermost and
// for dK, dV (and dTk) with i innermost, so that one sum suffices.
constexpr int P16_SLOTS = 11;
//
// The same two halves serve calls of few windows (split_windows).
struct P16UnitsWhole {
    __device__ __forceinline__ Units operator()(int n) const
    {
        const int64_t nt = (n + QT - 1) / QT;
        return {nt > 0 ? 1 : 0, (nt > P16_SLOTS ? 4 : 3) * nt * nt};
    }
};
enum { ROLE_Q = 1, ROLE_K = 2, Q_FIRST = 4, Q_LAST = 8, K_FIRST = 16, K_LAST = 32 };

template <int D>
struct P16Split {
    static constexpr int NW = p16_warps(D);
    static constexpr int DTW = D == 3 ? 2 : 3;                       // gradient warps per table
    static constexpr int NU = D == 9 ? 8 : (D == 6 ? 7 : 6);        // row tiles per gradient warp, at most
    static constexpr int HT0 = 3 * DTW;                              // first warp of the hist.T products
    static constexpr int SG = (NW - HT0) / 2;                        // warps per side of them
};

struct P16Smem {
    int R16, Rp;
    int off_pq, off_db, off_pk, off_s0, off_pl, off_rows, off_c, off_pg, off_lut, off_map, off_misc, total;
};

template <int D>
__host__ __device__ inline P16Smem make_p16_layout(int R, int lut_entries)
{
    P16Smem L;
    L.R16 = (R + 15) / 16 * 16;
    L.Rp = (L.R16 + 15) / 16 * 16 + 4;                             // see p16_store_key_major
    const int lane_arr = L.R16 * QT * 4, pk = 32 * L.Rp * 4;
    int off = 0;
    L.off_pq = off; off += lane_arr;                               // P_q, later histQ
    L.off_db = off; off += lane_arr;                               // dB, later histV
    L.off_pk = off; off += pk > lane_arr ? pk : lane_arr;          // P_k, later histK
    // S0 and dPV0 of every pair, then the pair planes; over both, once the histograms exist, partial dQ and dK
    const int part = 2 * P16Split<D>::SG * 32 * 32 * 4, s0pl = 32 * ES * 16 + 4 * 32 * ES * 4;
    L.off_s0 = off; off += 32 * ES * 16;
    L.off_pl = off; off += 4 * 32 * ES * 4;
    if (part > s0pl) off += part - s0pl;
    L.off_rows = off; off += P16_STAGES * 4 * 32 * P16_RS * 2;     // Q, dO (query tile), K, V (key tile), per stage
    L.off_c = off; off += P16_STAGES * 2 * 32 * 12 * 4;            // coordinates of both tiles, per stage
    L.off_pg = off; off += 3 * 32 * 32 * 4;                        // dQ, dV, dK of the pair products
    L.off_lut = off; off += (lut_entries * 2 + 15) / 16 * 16;
    L.off_map = off; off += (L.R16 * 2 + 15) / 16 * 16;            // internal row -> table row, 0xffff: none
    L.off_misc = off; off += 2048;
    L.total = off;
    return L;
}

struct P16Params {
    const __half *q, *k, *v, *dout, *o;
    const float *lse;
    const __half *tq, *tk, *tv;
    __half *dq, *dk, *dv;
    float *dtq, *dtk, *dtv;
    const int32_t *w_sizes, *w2n, *n2n;
    const float *n_coords;
    int64_t W;
    int H;
};

template <int D>
__global__ void __launch_bounds__((p16_warps(D) + 1) * 32, 1)
attn_bwd_pair16_kernel(const P16Params P, const PermMeta pm, const PairConsts pc)
{
    using SP = P16Split<D>;
    constexpr int NW = SP::NW, NT = NW * 32;
    constexpr int TG = NW / 3;                   // warps per table (projections)
    constexpr int NKW = (D + 1) / 2;             // warps of the key-side histogram, two dimensions each
    constexpr int GEMM_WARP = D + NKW;           // dQ and dK pair products
    constexpr int DV_WARP = (D & 1) ? D + NKW - 1 : D + NKW + 1;
    static_assert(DV_WARP < NW && GEMM_WARP < NW, "not enough warps");
    constexpr int SG = SP::SG, DTW = SP::DTW, NU = SP::NU;
    constexpr int KPW = (QT + NW - 1) / NW;      // keys per warp in the score phase
    constexpr int RS = P16_RS, ROWS = 32 * RS;
    extern __shared__ __align__(16) unsigned char smem[];
    const P16Smem L = make_p16_layout<D>(pm.R, pm.D * pm.lut_stride);
    uint32_t *s_pq = reinterpret_cast<uint32_t *>(smem + L.off_pq);
    uint32_t *s_db = reinterpret_cast<uint32_t *>(smem + L.off_db);
    uint32_t *s_pk = reinterpret_cast<uint32_t *>(smem + L.off_pk);
    uint32_t *s_hq = s_pq, *s_hv = s_db, *s_hk = s_pk;
    float4 *s_s0 = reinterpret_cast<float4 *>(smem + L.off_s0);         // [32][ES] (S0 h0, S0 h1, dPV0 h0, dPV0 h1)
    uint32_t *s_P = reinterpret_cast<uint32_t *>(smem + L.off_pl);      // [32][ES] half2 p
    uint32_t *s_DS = s_P + 32 * ES, *s_W0 = s_DS + 32 * ES, *s_W1 = s_W0 + 32 * ES;
    float *s_part = reinterpret_cast<float *>(smem + L.off_s0);         // [2][SG][32][32]
    __half *s_rows = reinterpret_cast<__half *>(smem + L.off_rows);     // [stage][Q,dO,K,V][32][RS]
    float *s_cs = reinterpret_cast<float *>(smem + L.off_c);            // [stage][query tile, key tile][32][12]
    float *s_pg = reinterpret_cast<float *>(smem + L.off_pg);           // [3][32][32]
    uint16_t *s_lut = reinterpret_cast<uint16_t *>(smem + L.off_lut);
    uint16_t *s_map = reinterpret_cast<uint16_t *>(smem + L.off_map);
    float *s_lses = reinterpret_cast<float *>(smem + L.off_misc);       // [stage][32][2]
    float *s_dels = s_lses + P16_STAGES * 64;                           // [stage][32][2]
    int *s_rowi = reinterpret_cast<int *>(s_dels + P16_STAGES * 64);    // [stage][query tile, key tile][32]
    int *s_n = s_rowi + P16_STAGES * 64;                                // [stage][8]: nq, nk, roles, slot, used tiles; nq = 0: no more items
    int *s_fail = s_n + P16_STAGES * 8;
    uint64_t *s_full = reinterpret_cast<uint64_t *>(smem + L.off_misc + 1792), *s_empty = s_full + P16_STAGES;

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int hp = blockIdx.y, H = P.H, HC = H * 16, co = hp * 32;

    if (tid == 0) {
        for (int s = 0; s < P16_STAGES; ++s) {
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
    // this block's share: a contiguous range of equal cost
    const bool split = split_windows<(NW + 1) * 32, 2, 3>(P.w_sizes, P.W, smem + L.off_pq);
    int64_t w_begin, w_end;
    int u_begin, u_end;                          // first unit of window w_begin, one past the last of window w_end
    if (split) balanced_units<(NW + 1) * 32>(P.w_sizes, P.W, smem + L.off_pq, UnitsSplit<2, 3>{}, w_begin, w_end, u_begin, u_end);
    else balanced_units<(NW + 1) * 32>(P.w_sizes, P.W, smem + L.off_pq, P16UnitsWhole{}, w_begin, w_end, u_begin, u_end);

    if (wid == NW) {
        // ================================ producer warp ================================================
        // Software-pipelined so that no load is consumed right after it is issued: the sizes of the next
        // window are fetched when a window is opened, the row numbers and coordinates of the next item
        // (indexed by sorted position) at the end of the current iteration, and only lse / dO / O (indexed
        // by the row number) inside the iteration, under the tile-mask arithmetic.
        int64_t w = w_begin - 1;
        int n = 0, base = 0, nt = 0, ts = 0, ti = 0, tj = 0;
        int unit = 0, unit_end = 0, role = 0;              // a window is one unit of both roles, or (halves) 2 nt of one
        bool halves = false;
        int n_nx = 0, base_nx = 0;                         // sizes of window w + 1
        if (w_begin < P.W) {
            n_nx = __ldg(P.w_sizes + w_begin);
            base_nx = __ldg(P.w2n + w_begin);
        }
        bool have = false;
        int nq = 0, nk = 0, rowq = 0, rowk = 0;
        float cq[D], ck[D];
        // descriptor of the next item and the loads that depend on the sorted position only
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
                    ts = nt > 0 ? (n + nt - 1) / nt : 0;   // equal tiles of at most QT voxels
                    halves = nt > P16_SLOTS || (split && nt > 1);
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
            float ls0 = 0.f, ls1 = 0.f, de0 = 0.f, de1 = 0.f;
            uint4 gdo[4], go[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) gdo[i] = go[i] = make_uint4(0, 0, 0, 0);
            if (lane < nq) {
                ls0 = __ldg(P.lse + (int64_t)rowq * H + 2 * hp);
                ls1 = __ldg(P.lse + (int64_t)rowq * H + 2 * hp + 1);
                const uint4 *gd = reinterpret_cast<const uint4 *>(P.dout + (int64_t)rowq * HC + co);
                const uint4 *gg = reinterpret_cast<const uint4 *>(P.o + (int64_t)rowq * HC + co);
#pragma unroll
                for (int i = 0; i < 4; ++i) { gdo[i] = __ldg(gd + i); go[i] = __ldg(gg + i); }
            }
            const uint32_t used = item_tile_mask<D>(cq, ck, nq, nk, s_lut, pm, pc, lane);
            // delta[slot] = sum_c dO . O over the sixteen channels of the head
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __half2 *a2 = reinterpret_cast<const __half2 *>(&gdo[i]), *b2 = reinterpret_cast<const __half2 *>(&go[i]);
                float acc = 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float2 fa = __half22float2(a2[c]), fb = __half22float2(b2[c]);
                    acc += fa.x * fb.x + fa.y * fb.y;
                }
                if (i < 2) de0 += acc; else de1 += acc;
            }
            const int s = it % P16_STAGES;
            if (it >= P16_STAGES && !mbar_wait(s_empty + s, ((it / P16_STAGES) - 1) & 1)) {
                g_async_error = 1;
                nq = nk = 0;                              // tell the consumers to stop
            }
            __half *rq = s_rows + s * (4 * ROWS);
            float *cs = s_cs + s * 768;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                cs[lane * 12 + d] = cq[d];
                cs[384 + lane * 12 + d] = ck[d];
            }
            s_rowi[s * 64 + lane] = rowq;
            s_rowi[s * 64 + 32 + lane] = rowk;
            s_lses[s * 64 + lane * 2] = ls0;
            s_lses[s * 64 + lane * 2 + 1] = ls1;
            s_dels[s * 64 + lane * 2] = de0;
            s_dels[s * 64 + lane * 2 + 1] = de1;
            if (lane == 0) {
                s_n[s * 8] = nq;
                s_n[s * 8 + 1] = nk;
                s_n[s * 8 + 2] = role | (tj == 0 ? Q_FIRST : 0) | (tj + 1 == nt ? Q_LAST : 0) | (ti == 0 ? K_FIRST : 0) | (ti + 1 == nt ? K_LAST : 0);
                s_n[s * 8 + 3] = role & ROLE_Q ? tj : 0;      // sums of dK and dV: slot
                s_n[s * 8 + 4] = (int)used;
            }
            mbar_arrive(s_full + s);
            stage_rows<4>(rq, RS, P.q + co, HC, rowq, nq, lane);
            stage_rows<4>(rq + ROWS, RS, P.dout + co, HC, rowq, nq, lane);
            stage_rows<4>(rq + 2 * ROWS, RS, P.k + co, HC, rowk, nk, lane);
            stage_rows<4>(rq + 3 * ROWS, RS, P.v + co, HC, rowk, nk, lane);
            mbar_arrive_cp_async(s_full + s);
            if (nq == 0) break;
            advance();                                    // the next item's position-indexed loads fly during the wait above
        }
        return;
    }

    // ==================================== consumer warps ===============================================
    const int g = lane >> 2, t = lane & 3;
    const int n_mt = L.R16 / 16, Rp = L.Rp;
    const int mypos = qpos(lane);
    const bool od = g & 1;
    constexpr float LOG2E = 1.4426950408889634f;
    // projections: warps [0, TG) serve Tq with Q, [TG, 2 TG) Tv with dO, [2 TG, 3 TG) Tk with K
    const int tg = wid / TG, wsub = wid - tg * TG;
    const __half *Tproj = tg == 0 ? P.tq : (tg == 1 ? P.tv : P.tk);
    // table gradients: the same order of tables, DTW warps each, row tiles dsub + DTW i; hist.T: 0 = histQ.Tq, 1 = histK.Tk
    const int dtg = wid / DTW, dsub = wid - dtg * DTW;
    const int side = wid < SP::HT0 ? 2 : (wid - SP::HT0) / SG, ws2 = (wid - SP::HT0) - side * SG;
    // [tile][slot, even / odd channels]: rows g (x, y), g + 8 (z, w); indexed at run time, hence in local memory
    float4 dt_acc[NU][4];
    if (dtg < 3)
#pragma unroll 1
        for (int i = 0; i < NU; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dt_acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);

    // sums of the store phase: this thread's entries, dQ (slot 0) or dK and dV of a key tile
    constexpr int EPT = (512 + NT - 1) / NT;
    float4 run[P16_SLOTS][EPT][2];

    int it = 0;
    for (;; ++it) {
        const int s = it % P16_STAGES;
        if (!mbar_wait(s_full + s, (it / P16_STAGES) & 1)) {
            *s_fail = 1;
            g_async_error = 2;
        }
        consumer_sync<NT>();          // the previous item's stores are over; the flag is settled
        const int nq = s_n[s * 8], nk = s_n[s * 8 + 1];
        const int roles = s_n[s * 8 + 2], slot = s_n[s * 8 + 3];
        const bool do_q = roles & ROLE_Q, do_k = roles & ROLE_K;
        const uint32_t used = (uint32_t)s_n[s * 8 + 4];
        if (nq == 0 || *s_fail) break;
        const __half *s_q = s_rows + s * (4 * ROWS), *s_do = s_q + ROWS, *s_k = s_do + ROWS, *s_v = s_k + ROWS;
        const float *s_c = s_cs + s * 768, *s_ck = s_c + 384;
        const int *s_rowq = s_rowi + s * 64, *s_rowk = s_rowq + 32;
        const float *s_lse = s_lses + s * 64, *s_del = s_dels + s * 64;
        // ---- projections P_q, dB (lane-major), P_k (key-major); S0 = K.Q^T and dPV0 = V.dO^T -----------------
        if (tg < 3) {
            UsedTiles tiles(used, n_mt, wsub, TG);
            int mt = tiles.next();
            P16TileA tile;
            if (mt >= 0) tile.fetch(Tproj, HC, co, s_map, mt, g, t);
            const int nv = tg == 2 ? nk : nq;
            uint2 bf[4][2];
            p16_feat_frag(bf, tg == 0 ? s_q : (tg == 1 ? s_do : s_k), nv, g, t);
#pragma unroll 1
            while (mt >= 0) {
                const P16TileA cur = tile;
                const int nx = tiles.next();
                if (nx >= 0) tile.fetch(Tproj, HC, co, s_map, nx, g, t);
                uint32_t d[2][2][4];
                p16_project(d, cur, bf, nv);
                if (tg < 2) p16_store_lane_major(tg == 0 ? s_pq : s_db, d, mt, g, t);
                else p16_store_key_major(s_pk, d, mt, Rp, nv, g, t);
                mt = nx;
            }
        }
        for (int u = NW - 1 - wid; u < 16; u += NW) {
            const int a = u >> 3, mt = (u >> 2) & 1, j = u & 3;     // key rows 16mt.., query columns 8j..
            if (16 * mt < nk && 8 * j < nq) {
                float c[2][2][2];
                p16_dot_block(c, a == 0 ? s_k : s_v, 16 * mt, a == 0 ? s_q : s_do, 8 * j, g, t);
#pragma unroll
                for (int rr = 0; rr < 2; ++rr)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        *reinterpret_cast<float2 *>(reinterpret_cast<float *>(s_s0 + (16 * mt + g + 8 * rr) * ES + 8 * j + 2 * t + e) + 2 * a) = make_float2(c[rr][e][0], c[rr][e][1]);
            }
        }
        consumer_sync<NT>();
        // ---- scores: keys wid, wid + NW, ... ; lane = query ----------------------------------------------------
        {
            float cx[D];
            load_coords12<D>(s_c + lane * 12, cx);
            const float xlse0 = s_lse[lane * 2] * LOG2E, xlse1 = s_lse[lane * 2 + 1] * LOG2E;
            const float xdel0 = s_del[lane * 2], xdel1 = s_del[lane * 2 + 1];
            const uint32_t *pq_lane = s_pq + mypos, *db_lane = s_db + mypos;
#pragma unroll
            for (int j = 0; j < KPW; ++j) {
                const int kk = wid + NW * j;
                if (kk < QT) {
                    uint32_t pw = 0u, dsw = 0u, w0 = 0u, w1 = 0u;     // zero for keys beyond the tile
                    if (kk < nk) {
                        float ck[D];
                        load_coords12<D>(s_ck + kk * 12, ck);
                        const uint32_t *pk_row = s_pk + kk * Rp;
                        __half2 b0 = __float2half2_rn(0.f), b1 = b0, b2 = b0;
#pragma unroll
                        for (int d = 0; d < D; ++d) {
                            const uint32_t idx = crse_index_pc(cx[d], ck[d], pc.half[d], pc.clamp[d]);
                            const uint32_t row = s_lut[d * pm.lut_stride + idx];
                            b0 = __hadd2(b0, u32_as_h2(pq_lane[row * QT]));
                            b1 = __hadd2(b1, u32_as_h2(pk_row[row]));
                            b2 = __hadd2(b2, u32_as_h2(db_lane[row * QT]));
                            if (d < 5) w0 |= idx << (IDX_BITS * d);
                            else w1 |= idx << (IDX_BITS * (d - 5));
                        }
                        const float4 in = s_s0[kk * ES + lane];          // S0 (h0,h1), dPV0 (h0,h1)
                        const float2 bs = __half22float2(__hadd2(b0, b1)), bd = __half22float2(b2);
                        float p0 = ex2_approx(fmaf(in.x + bs.x, LOG2E, -xlse0));
                        float p1 = ex2_approx(fmaf(in.y + bs.y, LOG2E, -xlse1));
                        float ds0 = p0 * (in.z + bd.x - xdel0);
                        float ds1 = p1 * (in.w + bd.y - xdel1);
                        if (lane >= nq) { p0 = 0.f; p1 = 0.f; ds0 = 0.f; ds1 = 0.f; }
                        pw = h2_as_u32(__floats2half2_rn(p0, p1));
                        dsw = h2_as_u32(__floats2half2_rn(ds0, ds1));
                    }
                    s_P[kk * ES + lane] = pw;
                    s_DS[kk * ES + lane] = dsw;
                    s_W0[kk * ES + lane] = w0;
                    s_W1[kk * ES + lane] = w1;
                }
            }
        }
        consumer_sync<NT>();
        // ---- clear the three histograms (P_q, dB, P_k are dead) ------------------------------------------------
        for (int i = tid; i < L.R16 * QT / 4; i += NT)                       // 128 16-byte pieces per 16-row tile
            if ((used >> (i >> 7)) & 1u) {
                const uint4 z = make_uint4(0, 0, 0, 0);
                if (do_q) {
                    reinterpret_cast<uint4 *>(s_hq)[i] = z;
                    reinterpret_cast<uint4 *>(s_hv)[i] = z;
                }
                if (do_k) reinterpret_cast<uint4 *>(s_hk)[i] = z;
            }
        consumer_sync<NT>();
        // ---- histograms and pair products -----------------------------------------------------------------------
        if (wid < D) {
            if (do_q) hist_query_side(s_hq + mypos, L.R16 * QT, s_P, s_DS, s_W0, s_W1, s_lut, pm.lut_stride, wid, nk, lane);
        } else if (wid < D + NKW && do_k) {
            for (int d = 2 * (wid - D); d < 2 * (wid - D) + 2 && d < D; ++d)
                hist_key_side(s_hk + mypos, s_DS, s_W0, s_W1, s_lut, pm.lut_stride, d, nq, lane);
        }
        if (wid == GEMM_WARP) {
            float acc[2][2][2][4];
            if (do_q) {
                p16_zero(acc);
                p16_pair_gemm<false>(acc, s_DS, s_k, nk, g, t);                 // dQ[q] = sum_k ds K[k]
                p16_store(s_pg, acc, g, t);
            }
            if (do_k) {
                p16_zero(acc);
                p16_pair_gemm<true>(acc, s_DS, s_q, nq, g, t);                  // dK[k] = sum_q ds Q[q]
                p16_store(s_pg + 2048, acc, g, t);
            }
        } else if (wid == DV_WARP && do_k) {
            float acc[2][2][2][4];
            p16_zero(acc);
            p16_pair_gemm<true>(acc, s_P, s_do, nq, g, t);                      // dV[k] = sum_q p dO[q]
            p16_store(s_pg + 1024, acc, g, t);
        }
        consumer_sync<NT>();
        // ---- dTq, dTv, dTk | dQ += histQ.Tq, dK += histK.Tk --------------------------------------------------------
        if (dtg < 3 && (dtg < 2 ? do_q : do_k)) {
            const __half *X = dtg == 0 ? s_q : (dtg == 1 ? s_do : s_k);
            const uint32_t *hist = dtg == 0 ? s_hq : (dtg == 1 ? s_hv : s_hk);
            uint32_t b[2][2][2][2];                            // [k-step][slot][parity][half]
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int p0 = 16 * ks + 4 * t + 2 * half, p1 = p0 + 1;   // column -> voxel: (p >> 2) + 8 (p & 3)
                        const int xa = (p0 >> 2) + 8 * (p0 & 3), xb = (p1 >> 2) + 8 * (p1 & 3);
                        const uint32_t u = *reinterpret_cast<const uint32_t *>(X + xa * RS + h * 16 + 2 * g);
                        const uint32_t w = *reinterpret_cast<const uint32_t *>(X + xb * RS + h * 16 + 2 * g);
                        b[ks][h][0][half] = pack_lo(u, w);
                        b[ks][h][1][half] = pack_hi(u, w);
                    }
#pragma unroll 1
            for (int i = 0; i < NU; ++i) {
                const int mt = dsub + DTW * i;
                if (mt >= n_mt) break;
                if (!((used >> mt) & 1u)) continue;
                float4 c[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) c[j] = dt_acc[i][j];
                const uint32_t *hu = hist + (mt * 16 + g) * QT + 4 * t, *hw = hu + 8 * QT;
                const uint4 ua = *reinterpret_cast<const uint4 *>(hu + (od ? 16 : 0)), ub = *reinterpret_cast<const uint4 *>(hu + (od ? 0 : 16));
                const uint4 wa = *reinterpret_cast<const uint4 *>(hw + (od ? 16 : 0)), wb = *reinterpret_cast<const uint4 *>(hw + (od ? 0 : 16));
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const bool first = (ks == 0) != od;
                    const uint4 u = first ? ua : ub, w = first ? wa : wb;
                    const uint32_t a[2][4] = {{pack_lo(u.x, u.y), pack_lo(w.x, w.y), pack_lo(u.z, u.w), pack_lo(w.z, w.w)},
                                              {pack_hi(u.x, u.y), pack_hi(w.x, w.y), pack_hi(u.z, u.w), pack_hi(w.z, w.w)}};
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            float4 &x = c[2 * h + p];
                            float d[4] = {x.x, x.y, x.z, x.w};
                            mma_f32(d, a[h], b[ks][h][p][0], b[ks][h][p][1]);
                            x = make_float4(d[0], d[1], d[2], d[3]);
                        }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) dt_acc[i][j] = c[j];
            }
        } else if (side < 2 && (side == 0 ? do_q : do_k)) {
            const __half *T = side == 0 ? P.tq : P.tk;
            const uint32_t *hist = side == 0 ? s_hq : s_hk;
            float acc[2][2][2][4];
            p16_zero(acc);
            UsedTiles tiles(used, n_mt, ws2, SG);
            int ks = tiles.next();
            P16TileB tile;
            if (ks >= 0) tile.fetch(T, HC, co, s_map, ks, g, t);
#pragma unroll 1
            while (ks >= 0) {
                const P16TileB cur = tile;
                const int nx = tiles.next();
                if (nx >= 0) tile.fetch(T, HC, co, s_map, nx, g, t);
                p16_hist_t(acc, hist, P16FragB(cur), ks, lane, g, t);
                ks = nx;
            }
            p16_store(s_part + (side * SG + ws2) * 1024, acc, g, t);
        }
        consumer_sync<NT>();
        // ---- reduce dQ (first half of the entries), dK and dV (second half), four channels each; sum over the tile pairs
        // of a row, store after the last ---------------------------------------------------------------------------
#pragma unroll
        for (int k = 0; k < EPT; ++k) {
            const int e = tid + NT * k, sd = e >> 8, xx = (e >> 3) & 31, ch = (e & 7) * 4;
            if (e < 512 && (sd == 0 ? do_q && xx < nq : do_k && xx < nk)) {
                float4 a = *reinterpret_cast<const float4 *>(s_pg + (sd == 0 ? 0 : 2048) + xx * 32 + ch), v = make_float4(0.f, 0.f, 0.f, 0.f);
                const float *pp = s_part + sd * SG * 1024 + xx * 32 + ch;
#pragma unroll
                for (int ww = 0; ww < SG; ++ww) {
                    const float4 pr = *reinterpret_cast<const float4 *>(pp + ww * 1024);
                    a.x += pr.x; a.y += pr.y; a.z += pr.z; a.w += pr.w;
                }
                if (sd == 1) v = *reinterpret_cast<const float4 *>(s_pg + 1024 + xx * 32 + ch);
                const int at = sd == 0 ? 0 : slot;
                if (!(roles & (sd == 0 ? Q_FIRST : K_FIRST))) {
                    const float4 b = run[at][k][0];
                    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
                    if (sd == 1) {
                        const float4 c = run[at][k][1];
                        v.x += c.x; v.y += c.y; v.z += c.z; v.w += c.w;
                    }
                }
                if (roles & (sd == 0 ? Q_LAST : K_LAST)) {
                    const int64_t o = (int64_t)(sd == 0 ? s_rowq : s_rowk)[xx] * HC + co + ch;
                    store_h4((sd == 0 ? P.dq : P.dk) + o, a);
                    if (sd == 1) store_h4(P.dv + o, v);
                } else {
                    run[at][k][0] = a;
                    if (sd == 1) run[at][k][1] = v;
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty + s);
    }

    // ---- the table gradients of this block -----------------------------------------------------------------------------
    if (dtg < 3 && it > 0) {
        float *dst = dtg == 0 ? P.dtq : (dtg == 1 ? P.dtv : P.dtk);
#pragma unroll 1
        for (int i = 0; i < NU; ++i) {
            const int mt = dsub + DTW * i;
            if (mt >= n_mt) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 ev = dt_acc[i][2 * h], ov = dt_acc[i][2 * h + 1];
                const int r0 = s_map[mt * 16 + g], r1 = s_map[mt * 16 + g + 8];      // aliases go to the row they stand for
                if (r0 != 0xffff) atomicAdd(reinterpret_cast<float4 *>(dst + (int64_t)r0 * HC + co + h * 16 + 4 * t), make_float4(ev.x, ov.x, ev.y, ov.y));
                if (r1 != 0xffff) atomicAdd(reinterpret_cast<float4 *>(dst + (int64_t)r1 * HC + co + h * 16 + 4 * t), make_float4(ev.z, ov.z, ev.w, ov.w));
            }
        }
    }
}

template <int D>
static int launch_pair16(const P16Params &p, const CrseMeta &meta, const PermMeta &pm, cudaStream_t st)
{
    const P16Smem L = make_p16_layout<D>(pm.R, pm.D * pm.lut_stride);
    auto kern = attn_bwd_pair16_kernel<D>;
    int sms = 0;
    const int rc = kernel_setup(reinterpret_cast<const void *>(kern), sms);
    if (rc != S3D_OK) return rc;
    const int hp = p.H / 2;
    int gx = sms / hp;
    if (gx < 1) gx = 1;
    kern<<<dim3((unsigned)gx, (unsigned)hp), (p16_warps(D) + 1) * 32, L.total, st>>>(p, pm, make_pair_consts(meta));
    const cudaError_t le = cudaGetLastError();
    note_cuda_error(le);
    return le == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}

template <int D>
static bool pair16_fits(const PermMeta &pm)
{
    const int n_mt = (pm.R + 15) / 16;                       // the tile mask is one word
    return n_mt <= 32 && n_mt <= P16Split<D>::NU * P16Split<D>::DTW && make_p16_layout<D>(pm.R, pm.D * pm.lut_stride).total <= 227 * 1024;
}

}  // namespace tc

bool attn_tc_bwd_pair16_supported(const AttnArgs &a)
{
    if (a.dtype != S3D_F16 || a.hd != 16 || (a.H & 1) || a.m_dq.n) return false;
    for (int d = 0; d < a.meta.D; ++d)
        if (a.meta.L[d] >= (1 << tc::IDX_BITS)) return false;
    const tc::PermMeta pm = tc::make_perm_meta(a.meta);
    return a.meta.D == 3 ? tc::pair16_fits<3>(pm) : (a.meta.D == 6 ? tc::pair16_fits<6>(pm) : tc::pair16_fits<9>(pm));
}

// dtq, dtk, dtv must be zero on entry (accumulated into).
int attn_tc_backward_pair16(const AttnArgs &a, cudaStream_t st)
{
    if (a.W == 0) return S3D_OK;
    const tc::PermMeta pm = tc::make_perm_meta(a.meta);
    tc::P16Params p{};
    p.q = (const __half *)a.q; p.k = (const __half *)a.k; p.v = (const __half *)a.v;
    p.dout = (const __half *)a.dout; p.o = (const __half *)a.out; p.lse = a.lse;
    p.tq = (const __half *)a.tq; p.tk = (const __half *)a.tk; p.tv = (const __half *)a.tv;
    p.dq = (__half *)a.dq; p.dk = (__half *)a.dk; p.dv = (__half *)a.dv;
    p.dtq = a.dtq; p.dtk = a.dtk; p.dtv = a.dtv;
    p.w_sizes = a.w_sizes; p.w2n = a.w2n; p.n2n = a.n2n; p.n_coords = a.n_coords;
    p.W = a.W; p.H = a.H;
    switch (a.meta.D) {
        case 3: return tc::launch_pair16<3>(p, a.meta, pm, st);
        case 6: return tc::launch_pair16<6>(p, a.meta, pm, st);
        case 9: return tc::launch_pair16<9>(p, a.meta, pm, st);
        default: return S3D_ERR_UNSUPPORTED;
    }
}

cudaError_t attn_tc_bwd_pair16_async_error(bool &set) { return take_async_error(set); }

}  // namespace s3d
