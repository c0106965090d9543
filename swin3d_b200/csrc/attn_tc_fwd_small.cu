// Forward of the cRSE window attention, tensor-core path (fp16), windows of any size: two heads of 8 channels
// per block, or one of 16 (an odd head count).  Even head counts of 16 channels: attn_tc_fwd_pair16.cu.
//
// A window of n voxels is cut into nt = ceil(n / 32) tiles of equal size.  A block of D+1 warps (at least 8) takes
// query tiles (window, i) and runs over the key tiles j of their window: every tile pair is an independent
// 32 x 32 problem with its own row maximum; a thread of the store phase keeps two output channels of one
// query and merges the tile pairs' (maximum, sum, output) as they come.  Most windows of the first
// stage have at most 32 voxels and are a single item, where nothing is merged.  Per item:
//   stage      Q rows (query tile), K, V rows (key tile) of the head pair, the signal coordinates of both
//   GEMM       P_q = Tq.Q^T (lane-major), P_k = Tk.K^T (key-major), S0 = K.Q^T     [tensor cores]
//              the first half of the warps owns the Tq tiles, the second half the Tk tiles, so a
//              warp builds the block-diagonal B fragments of its feature array once per item
//   scores     lane = query, the keys dealt to the warps: D indices, 2*D look-ups, score; the
//              scores and the packed indices of a thread's (at most four) pairs stay in registers;
//              exact row maxima through shared-memory atomics
//   softmax    probabilities, row sums, pair entries written once: two [key][query] planes of
//              8-byte entries, (p, idx 0-4) and (idx 5-8, p), row stride 33 entries
//   histogram  warp d owns signal dimension d (rows of different dimensions are disjoint):
//              hist[row][q] += p, two keys per step, the next step's entries fetched before the
//              stores of this one; warp D: O = P.V                                    [tensor cores]
//   epilogue   O += hist.Tv (k-steps dealt to the warps) [tensor cores], reduce, merge, store
// The histogram reuses the shared memory of P_q, which is dead once the scores exist, and P_q is projected
// again for every key tile; about 110 KB of shared memory per block, two blocks per SM.
// The blocks take contiguous ranges of (window, query tile) units of equal cost (tile pairs).
// grid = (x, H/2) (head_dim 8) or (x, H) (head_dim 16).
//
// Bound: shared-memory wavefronts (66 % of the pipe's peak), instruction issue (55 %), barriers and staged rows (1.8 and 1.6
// stall cycles per instruction); 241 k voxels, 10 heads.
// Measured against the version for windows of at most 32 voxels (blocks took every gridDim.x-th window) plus a kernel of
// one block per SM with an online softmax for the larger ones: 964 k voxels, 10 heads 8.38 -> 7.69 ms; 115 k
// voxels, 6 heads 680 -> 559 us.
#include "attn_kernels.cuh"
#include "attn_tc.cuh"
#include "attn_tc_small.cuh"
#include "async_stage.cuh"

namespace s3d {
namespace tc {

// Debug build only (-DS3D_PHASE_CLOCK): cycles spent between the block-wide barriers of a window,
// summed over all windows and blocks by thread 0 of every block; read back with
// s3d_debug_phase_cycles().  Compiled out otherwise.
#ifdef S3D_PHASE_CLOCK
__device__ unsigned long long g_phase_cycles[16];
__device__ unsigned int g_ablate;      // bit i set: piece i of the kernel is skipped (results are then wrong)
#define S3D_KEEP(i) (!(ablate & (1u << (i))))
#define S3D_PHASE_DECL long long ph_t = clock64(); unsigned long long ph_acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#define S3D_PHASE_MARK(i) if (threadIdx.x == 0) { const long long now = clock64(); ph_acc[i] += (unsigned long long)(now - ph_t); ph_t = now; }
#define S3D_PHASE_FLUSH(base) if (threadIdx.x == 0) { for (int i = 0; i < 8; ++i) atomicAdd(&g_phase_cycles[(base) + i], ph_acc[i]); }
#else
#define S3D_KEEP(i) true
#define S3D_PHASE_DECL
#define S3D_PHASE_MARK(i)
#define S3D_PHASE_FLUSH(base)
#endif

constexpr int FS_STAGES = 2;      // items staged ahead of the one being computed

struct FwdSmallSmem {
    int R16, Rp;
    int off_pq, off_pk, off_e, off_rows, off_c, off_misc, total;
};

__host__ __device__ inline FwdSmallSmem make_fwd_small_layout(int R, int nw)
{
    FwdSmallSmem L;
    L.R16 = (R + 15) / 16 * 16;
    L.Rp = (L.R16 + 31) / 32 * 32 + 8;
    int off = 0;
    L.off_pq = off; off += L.R16 * QT * 4;                                   // P_q, later the histogram
    const int pk = 32 * L.Rp * 4, red = nw * (QT * 16 + QT * 2) * 4;
    L.off_pk = off; off += pk > red ? pk : red;                              // P_k, later the reduction buffer
    L.off_e = off; off += 2 * 32 * ES * 8;                                   // pair entries, two planes
    L.off_rows = off; off += FS_STAGES * 3 * 32 * 16 * 2;                    // Q, K, V rows, per stage
    L.off_c = off; off += FS_STAGES * 2 * 32 * 12 * 4;                       // signal coordinates of both tiles, per stage
    L.off_misc = off; off += 1024;
    L.total = off;
    return L;
}

struct FwdSmallParams {
    const __half *q, *k, *v, *tq, *tk, *tv;
    __half *out;
    float *lse;
    const int32_t *w_sizes, *w2n, *n2n;
    const float *n_coords;
    int64_t W;
    int H;
    int n_min, n_max;      // the window sizes of this call
    Mirrors m_out;
};

// Block = NW consumer warps + one producer warp.  The producer walks the block's tile pairs ahead of the
// consumers: it reads row numbers and coordinates and copies the 32-byte Q, K, V pieces of the voxels
// into the next stage of shared memory (cp.async, completion on the stage's "full" mbarrier); the
// consumers hand a stage back through its "empty" mbarrier.
template <int D, int NW, int NPU /*projection units per warp*/, int NHU /*hist.T units per warp*/, bool HD16>
__global__ void __launch_bounds__((NW + 1) * 32, 2)
attn_fwd_small_kernel(const __grid_constant__ FwdSmallParams P, const CrseMeta meta, const PairConsts pc)
{
    constexpr int NT = NW * 32;                  // consumer threads
    constexpr int HALF = NW / 2;                 // warps per projection table
    constexpr int KPW = (QT + NW - 1) / NW;      // keys per warp in the score phase
    static_assert(D < NW, "one warp per signal dimension plus one for P.V");
    extern __shared__ __align__(16) unsigned char smem[];
    const FwdSmallSmem L = make_fwd_small_layout(meta.R, NW);
    uint32_t *s_pq = reinterpret_cast<uint32_t *>(smem + L.off_pq);
    uint32_t *s_hist = s_pq;
    uint32_t *s_pk = reinterpret_cast<uint32_t *>(smem + L.off_pk);
    uint2 *s_elo = reinterpret_cast<uint2 *>(smem + L.off_e);        // [32][ES] (p, idx 0-4); S0 before
    uint2 *s_ehi = s_elo + 32 * ES;                                  // [32][ES] (idx 5-8, p)
    __half *s_rows = reinterpret_cast<__half *>(smem + L.off_rows);  // [stage][Q,K,V][32][16]
    float *s_cs = reinterpret_cast<float *>(smem + L.off_c);         // [stage][query tile, key tile][32][12]
    float *s_max = reinterpret_cast<float *>(smem + L.off_misc);     // [32][2]
    int *s_rowi = reinterpret_cast<int *>(s_max + 64);               // [stage][32] rows of the query tile
    int *s_n = s_rowi + FS_STAGES * 32;                              // [stage][4]: nq, nk, first key tile, last key tile; nq = 0: no more items
    int *s_fail = s_n + FS_STAGES * 4;
    uint64_t *s_full = reinterpret_cast<uint64_t *>(smem + L.off_misc + 768);   // [stage]
    uint64_t *s_empty = s_full + FS_STAGES;                                      // [stage]
    float *s_red = reinterpret_cast<float *>(smem + L.off_pk);       // [NW][32][16], P_k is dead by then
    float *s_lsum = s_red + NW * 512;                                // [NW][32][2]

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int hp = blockIdx.y, H = P.H;
    const int HC = H * (HD16 ? 16 : 8), co = hp * 16;

    if (tid == 0) {
        for (int s = 0; s < FS_STAGES; ++s) {
            mbar_init(s_full + s, 64);         // every producer lane: its stores, its copies
            mbar_init(s_empty + s, NW);
        }
        *s_fail = 0;
        mbar_init_fence();
    }
    int64_t w_begin, w_end;
    int i_begin, i_end;                          // first query tile of window w_begin, one past the last of window w_end
    balanced_units<(NW + 1) * 32>(P.w_sizes, P.W, smem + L.off_pq, UnitsPerQueryTile{P.n_min, P.n_max}, w_begin, w_end, i_begin, i_end);

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
                        nt = n >= P.n_min && n <= P.n_max ? (n + QT - 1) / QT : 0;
                        ts = nt > 0 ? (n + nt - 1) / nt : 0;
                        ti = w == w_begin ? i_begin : 0;
                        ti_end = w == w_end ? i_end : nt;
                        tj = 0;
                    }
                } while (have && ti >= ti_end);
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
            if (ti == tj) {                       // the only case of a window of one tile
                rowk = rowq;
#pragma unroll
                for (int d = 0; d < D; ++d) ck[d] = cq[d];
            } else if (lane < nk) {
                const int pos = base + tj * ts + lane;
                rowk = __ldg(P.n2n + pos);
#pragma unroll
                for (int d = 0; d < D; ++d) ck[d] = __ldg(P.n_coords + (int64_t)pos * D + d);
            }
        };
        advance();
        for (int it = 0;; ++it) {
            const int s = it % FS_STAGES;
            if (it >= FS_STAGES && !mbar_wait(s_empty + s, ((it / FS_STAGES) - 1) & 1)) {
                g_async_error = 1;
                have = false;                             // tell the consumers to stop
            }
            if (!have) nq = nk = 0;
            __half *rq = s_rows + s * 1536;
            float *cs = s_cs + s * 768;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                cs[lane * 12 + d] = cq[d];
                cs[384 + lane * 12 + d] = ck[d];
            }
            s_rowi[s * 32 + lane] = rowq;
            if (lane == 0) {
                s_n[s * 4] = nq;
                s_n[s * 4 + 1] = nk;
                s_n[s * 4 + 2] = tj == 0;
                s_n[s * 4 + 3] = tj + 1 == nt;
            }
            mbar_arrive(s_full + s);
            stage_rows<2>(rq, 16, P.q + co, HC, rowq, nq, lane);
            stage_rows<2>(rq + 512, 16, P.k + co, HC, rowk, nk, lane);
            stage_rows<2>(rq + 1024, 16, P.v + co, HC, rowk, nk, lane);
            mbar_arrive_cp_async(s_full + s);
            if (!have) break;
            advance();
        }
        return;
    }

    // ==================================== consumer warps ===============================================
    const int g = lane >> 2, t = lane & 3;
    const int n_mt = L.R16 / 16, Rp = L.Rp;
    const int mypos = qpos(lane);
    constexpr float LOG2E = 1.4426950408889634f;

    // projection units: warps [0, HALF) own the Tq tiles wsub + HALF i, warps [HALF, 2 HALF) the Tk tiles
    const bool q_side = wid < HALF;
    const bool p_side = wid < 2 * HALF;
    const int wsub = q_side ? wid : wid - HALF;
    uint32_t ta[NPU][2][2];
#pragma unroll
    for (int i = 0; i < NPU; ++i) {
        const int mt = wsub + HALF * i;
        const __half *T = q_side ? P.tq : P.tk;
        const bool ok = p_side && mt < n_mt;
        const int r0 = ok ? table_row(meta, mt * 16 + g) : -1, r1 = ok ? table_row(meta, mt * 16 + g + 8) : -1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            ta[i][h][0] = r0 >= 0 ? *reinterpret_cast<const uint32_t *>(T + (int64_t)r0 * HC + co + h * 8 + 2 * t) : 0u;
            ta[i][h][1] = r1 >= 0 ? *reinterpret_cast<const uint32_t *>(T + (int64_t)r1 * HC + co + h * 8 + 2 * t) : 0u;
        }
    }
    // hist.Tv units: k-step = wid + NW i
    uint32_t tb[NHU][2][2];
#pragma unroll
    for (int i = 0; i < NHU; ++i) {
        const int ks = wid + NW * i;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int ra = ks < n_mt ? table_row(meta, ks * 16 + ht_krow(t, half, 0)) : -1;
                const int rb = ks < n_mt ? table_row(meta, ks * 16 + ht_krow(t, half, 1)) : -1;
                const __half lo = ra >= 0 ? P.tv[(int64_t)ra * HC + co + h * 8 + g] : __float2half(0.f);
                const __half hi = rb >= 0 ? P.tv[(int64_t)rb * HC + co + h * 8 + g] : __float2half(0.f);
                tb[i][h][half] = h2_as_u32(__halves2half2(lo, hi));
            }
    }
    // the store phase: this thread's query and two channels, merged over the key tiles
    float2 o_run = make_float2(0.f, 0.f);
    float m_run = 0.f, l_run = 0.f;
    S3D_PHASE_DECL
#ifdef S3D_PHASE_CLOCK
    const unsigned ablate = g_ablate;
#endif
    for (int it = 0;; ++it) {
        const int s = it % FS_STAGES;
        if (!mbar_wait(s_full + s, (it / FS_STAGES) & 1)) {
            *s_fail = 1;
            g_async_error = 2;
        }
        consumer_sync<NT>();          // the previous item's epilogue is over; the flag is settled
        S3D_PHASE_MARK(0)
        const int nq = s_n[s * 4], nk = s_n[s * 4 + 1];
        if (nq == 0 || *s_fail) break;
        const __half *s_q = s_rows + s * 1536, *s_k = s_q + 512, *s_v = s_q + 1024;
        const float *s_c = s_cs + s * 768, *s_ck = s_c + 384;
        float cx[D];
        load_coords12<D>(s_c + lane * 12, cx);
        if (tid < 64) s_max[tid] = -INFINITY;
        // ---- projections P_q (lane-major), P_k (key-major); S0 = K.Q^T ------------------------------
        if (p_side && S3D_KEEP(0)) {
            uint32_t bf[8][2];
            load_feat_bfrag(bf, q_side ? s_q : s_k, q_side ? nq : nk, g, t);
#pragma unroll
            for (int i = 0; i < NPU; ++i) {
                const int mt = wsub + HALF * i;
                if (mt < n_mt) {
                    if (q_side) project_unit_b<true>(ta[i], bf, s_pq, mt, Rp, nq, g, t);
                    else project_unit_b<false>(ta[i], bf, s_pk, mt, Rp, nk, g, t);
                }
            }
        }
        for (int u = wid; u < 16 && S3D_KEEP(1); u += NW) {
            const int mt = u >> 3, j = u & 7;       // key rows 16mt.., query columns 4j..
            if (16 * mt < nk && 4 * j < nq) {
                const __half *ysrc = s_k + mt * 256;
                const uint32_t wv = *reinterpret_cast<const uint32_t *>(s_q + (4 * j + (g >> 1)) * 16 + (g & 1) * 8 + 2 * t);
                const uint32_t a0 = *reinterpret_cast<const uint32_t *>(ysrc + g * 16 + 2 * t);
                const uint32_t a1 = *reinterpret_cast<const uint32_t *>(ysrc + (g + 8) * 16 + 2 * t);
                const uint32_t a2 = *reinterpret_cast<const uint32_t *>(ysrc + g * 16 + 8 + 2 * t);
                const uint32_t a3 = *reinterpret_cast<const uint32_t *>(ysrc + (g + 8) * 16 + 8 + 2 * t);
                float c[4];
                mma_k16_z(c, a0, a1, a2, a3, (g & 1) ? 0u : wv, (g & 1) ? wv : 0u);
                *reinterpret_cast<float2 *>(s_elo + (16 * mt + g) * ES + 4 * j + t) = make_float2(c[0], c[1]);
                *reinterpret_cast<float2 *>(s_elo + (16 * mt + g + 8) * ES + 4 * j + t) = make_float2(c[2], c[3]);
            }
        }
        consumer_sync<NT>();
        S3D_PHASE_MARK(2)
        // ---- scores: keys wid, wid + NW, ... ; lane = query: indices, 2*D look-ups, score -------------
        float sreg[KPW][2];
        uint32_t wreg[KPW][2];
        float mloc0 = -INFINITY, mloc1 = -INFINITY;
        const uint32_t *pq_lane = s_pq + mypos;
#pragma unroll
        for (int j = 0; j < KPW; ++j) {
            const int kk = wid + NW * j;
            sreg[j][0] = sreg[j][1] = 0.f;
            wreg[j][0] = wreg[j][1] = 0u;
            if (kk < nk && S3D_KEEP(2)) {
                float ck[D];
                load_coords12<D>(s_ck + kk * 12, ck);
                const uint32_t *pk_row = s_pk + kk * Rp;
                __half2 bq = __float2half2_rn(0.f), bk = bq;
                uint32_t w0 = 0, w1 = 0;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const uint32_t idx = crse_index_pc(cx[d], ck[d], pc.half[d], pc.clamp[d]);
                    const uint32_t row = meta.rowbase[d] + idx;
                    bq = __hadd2(bq, u32_as_h2(pq_lane[row * QT]));
                    bk = __hadd2(bk, u32_as_h2(pk_row[row]));
                    if (d < 5) w0 |= idx << (IDX_BITS * d);
                    else w1 |= idx << (IDX_BITS * (d - 5));
                }
                const float2 s0 = *reinterpret_cast<const float2 *>(s_elo + kk * ES + lane);
                const float2 b = __half22float2(__hadd2(bq, bk));
                float sx = s0.x + b.x, sy = s0.y + b.y;
                if (HD16) sx = sy = sx + sy;          // one head: both halves carry the full score
                sreg[j][0] = sx;
                sreg[j][1] = sy;
                wreg[j][0] = w0;
                wreg[j][1] = w1;
                mloc0 = fmaxf(mloc0, sx);
                mloc1 = fmaxf(mloc1, sy);
            }
        }
        if (wid < nk) {
            atomic_max_float(s_max + lane * 2, mloc0);
            atomic_max_float(s_max + lane * 2 + 1, mloc1);
        }
        consumer_sync<NT>();
        S3D_PHASE_MARK(3)
        // ---- probabilities, pair entries; clear the histogram (the P_q storage) ---------------------------
        const float m0 = s_max[lane * 2] * LOG2E, m1 = s_max[lane * 2 + 1] * LOG2E;
        float l0 = 0.f, l1 = 0.f;
#pragma unroll
        for (int j = 0; j < KPW; ++j) {
            const int kk = wid + NW * j;
            if (kk < QT && S3D_KEEP(3)) {
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
        for (int i = tid; i < L.R16 * QT / 4 && S3D_KEEP(4); i += NT)
            reinterpret_cast<uint4 *>(s_hist)[i] = make_uint4(0, 0, 0, 0);
        consumer_sync<NT>();
        S3D_PHASE_MARK(4)
        // ---- histogram (warp d: signal dimension d) | warp D: O = P.V -----------------------------------------
        float part[2][2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 2; ++i) part[h][i][0] = part[h][i][1] = part[h][i][2] = part[h][i][3] = 0.f;
        if (wid < D && S3D_KEEP(5)) {
            const int d = wid;
            const bool lo = d < 5;
            const int sh = IDX_BITS * (lo ? d : d - 5);
            // the half of a pair entry this dimension needs: (p, idx 0-4) or (idx 5-8, p)
            const uint2 *ecol = (lo ? s_elo : s_ehi) + lane;
            uint32_t *cell = s_hist + meta.rowbase[d] * QT + mypos;
            uint2 e0 = ecol[0], e1 = ecol[ES];              // keys beyond the tile hold zero entries
            int kk = 0;
            for (; kk + 1 < nk; kk += 2) {
                const uint32_t p0 = lo ? e0.x : e0.y, i0 = ((lo ? e0.y : e0.x) >> sh) & ((1u << IDX_BITS) - 1u);
                const uint32_t p1 = lo ? e1.x : e1.y, i1 = ((lo ? e1.y : e1.x) >> sh) & ((1u << IDX_BITS) - 1u);
                uint32_t *a0 = cell + i0 * QT, *a1 = cell + i1 * QT;
                const uint32_t c0 = *a0, c1 = *a1;
                e0 = ecol[min(kk + 2, QT - 1) * ES];
                e1 = ecol[min(kk + 3, QT - 1) * ES];
                const __half2 s0 = __hadd2(u32_as_h2(c0), u32_as_h2(p0));
                const __half2 s1 = __hadd2(a1 == a0 ? s0 : u32_as_h2(c1), u32_as_h2(p1));
                *a0 = h2_as_u32(s0);
                *a1 = h2_as_u32(s1);
            }
            if (kk < nk) {
                const uint32_t p0 = lo ? e0.x : e0.y, i0 = ((lo ? e0.y : e0.x) >> sh) & ((1u << IDX_BITS) - 1u);
                uint32_t *a0 = cell + i0 * QT;
                *a0 = h2_as_u32(__hadd2(u32_as_h2(*a0), u32_as_h2(p0)));
            }
        } else if (wid == D && S3D_KEEP(6)) {
            pair_gemm2<0, false>(part, s_elo, s_v, nk, g, t);  // O[q] = sum_k p V[k]
        }
        consumer_sync<NT>();
        S3D_PHASE_MARK(5)
        // ---- O += hist . Tv (k-steps split over the warps), reduce, normalise, store --------------------------
#pragma unroll
        for (int i = 0; i < NHU; ++i) {
            const int ks = wid + NW * i;
            if (ks < n_mt && S3D_KEEP(7)) ht_unit(part, s_hist, tb[i], ks, g, t);
        }
        store_part(s_red + wid * 512, part, g, t);       // P_k (aliased by s_red) is dead since the scores
        s_lsum[(wid * QT + lane) * 2] = l0;
        s_lsum[(wid * QT + lane) * 2 + 1] = l1;
        consumer_sync<NT>();
        S3D_PHASE_MARK(6)
        if (tid < 256 && S3D_KEEP(8)) {
            const int qq = tid >> 3, ch = (tid & 7) * 2, h = ch >> 3;
            if (qq < nq) {
                float a = 0.f, b = 0.f, ls = 0.f;
#pragma unroll
                for (int ww = 0; ww < NW; ++ww) {
                    const float2 pr = *reinterpret_cast<const float2 *>(s_red + ww * 512 + qq * 16 + ch);
                    a += pr.x;
                    b += pr.y;
                    ls += s_lsum[(ww * QT + qq) * 2 + h];
                }
                float m = s_max[qq * 2 + h];
                if (!s_n[s * 4 + 2]) {                     // not the first key tile
                    const float mt = m;
                    m = fmaxf(m_run, mt);
                    const float f0 = ex2_approx((m_run - m) * LOG2E), f1 = ex2_approx((mt - m) * LOG2E);
                    a = o_run.x * f0 + a * f1;
                    b = o_run.y * f0 + b * f1;
                    ls = l_run * f0 + ls * f1;
                }
                if (s_n[s * 4 + 3]) {                      // the last one
                    const float inv = 1.f / ls;
                    const int64_t row = s_rowi[s * 32 + qq];
                    store_h2_mirrored(P.out, P.m_out, row * HC + co + ch, __floats2half2_rn(a * inv, b * inv));
                    if (HD16) {
                        if (ch == 0) P.lse[row * H + hp] = m + __logf(ls);
                    } else if ((ch & 7) == 0) {
                        P.lse[row * H + 2 * hp + h] = m + __logf(ls);
                    }
                } else {
                    o_run = make_float2(a, b);
                    m_run = m;
                    l_run = ls;
                }
            }
        }
        // this warp is done with the stage (rows, coordinates, row numbers)
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty + s);
    }  // items
    S3D_PHASE_FLUSH(0)
}

template <int D, int NW, int NPU, int NHU, bool HD16>
static int launch_fwd_small(const FwdSmallParams &p, const CrseMeta &meta, cudaStream_t st)
{
    const FwdSmallSmem L = make_fwd_small_layout(meta.R, NW);
    auto kern = attn_fwd_small_kernel<D, NW, NPU, NHU, HD16>;
    // blocks per SM of this instantiation, found once per device
    static int sms_of[64] = {0};     // 0: this instantiation has not been set up on the device yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return S3D_ERR_LAUNCH;
    if (sms_of[dev] == 0) {
        int sms = 0;
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        note_cuda_error(e);
        if (e != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
            return S3D_ERR_LAUNCH;
        sms_of[dev] = sms;
    }
    const int hp = HD16 ? p.H : p.H / 2;
    // the launch bounds keep two blocks' registers within an SM; shared memory (228 KB per SM, 1 KB
    // reserved per block) decides whether two fit
    const int per_sm = 2 * (L.total + 1024) <= 228 * 1024 ? 2 : 1;
    int gx = sms_of[dev] * per_sm / hp;
    if (gx < 1) gx = 1;
    dim3 grid((unsigned)gx, (unsigned)hp);
    kern<<<grid, (NW + 1) * 32, L.total, st>>>(p, meta, make_pair_consts(meta));
    return cudaGetLastError() == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}

static int fwd_small_warps(int D) { return D + 1 > 8 ? D + 1 : 8; }

}  // namespace tc

#ifdef S3D_PHASE_CLOCK
extern "C" int s3d_debug_set_ablate(unsigned int mask)
{
    return cudaMemcpyToSymbol(tc::g_ablate, &mask, sizeof(mask)) == cudaSuccess ? S3D_OK : S3D_ERR_LAUNCH;
}

extern "C" int s3d_debug_phase_cycles(unsigned long long *out16, int reset)
{
    if (cudaMemcpyFromSymbol(out16, tc::g_phase_cycles, sizeof(unsigned long long) * 16) != cudaSuccess) return S3D_ERR_LAUNCH;
    if (reset) {
        unsigned long long z[16] = {0};
        if (cudaMemcpyToSymbol(tc::g_phase_cycles, z, sizeof(z)) != cudaSuccess) return S3D_ERR_LAUNCH;
    }
    return S3D_OK;
}
#endif

bool attn_tc_fwd_small_supported(const AttnArgs &a)
{
    if (a.dtype != S3D_F16) return false;
    if (!(a.hd == 16 || (a.hd == 8 && !(a.H & 1)))) return false;
    const int Rint = a.meta.R + a.meta.D - 1;
    const int n_mt = (Rint + 15) / 16;
    const int nw = tc::fwd_small_warps(a.meta.D);
    if (n_mt > 6 * (nw / 2) || n_mt > 3 * nw) return false;
    for (int d = 0; d < a.meta.D; ++d)
        if (a.meta.L[d] >= (1 << tc::IDX_BITS)) return false;
    return tc::make_fwd_small_layout(Rint, nw).total <= 227 * 1024;
}

// a.window_class: windows of the other class are left untouched.
int attn_tc_forward_small(const AttnArgs &a0, cudaStream_t st)
{
    if (a0.W == 0) return S3D_OK;
    AttnArgs a = a0;
    a.meta = tc::internal_meta(a0.meta);
    tc::FwdSmallParams p{};
    p.q = (const __half *)a.q; p.k = (const __half *)a.k; p.v = (const __half *)a.v;
    p.tq = (const __half *)a.tq; p.tk = (const __half *)a.tk; p.tv = (const __half *)a.tv;
    p.out = (__half *)a.out; p.lse = a.lse; p.m_out = a.m_out;
    p.w_sizes = a.w_sizes; p.w2n = a.w2n; p.n2n = a.n2n; p.n_coords = a.n_coords;
    p.W = a.W; p.H = a.H;
    p.n_min = a.window_class == 2 ? tc::QT + 1 : 1;
    p.n_max = a.window_class == 1 ? tc::QT : 0x7fffffff;
    const int n_mt = (a.meta.R + 15) / 16;
    const int nw = tc::fwd_small_warps(a.meta.D);
    const int npu = (n_mt + nw / 2 - 1) / (nw / 2);   // <= 6
    const int nhu = (n_mt + nw - 1) / nw;             // <= 3
#define S3D_FS(DD, NWW, HH)                                                                       \
    if (npu <= 2 && nhu <= 1) return tc::launch_fwd_small<DD, NWW, 2, 1, HH>(p, a.meta, st);      \
    if (npu <= 4 && nhu <= 2) return tc::launch_fwd_small<DD, NWW, 4, 2, HH>(p, a.meta, st);      \
    return tc::launch_fwd_small<DD, NWW, 6, 3, HH>(p, a.meta, st);
#define S3D_FS_D(DD, NWW) if (a.hd == 16) { S3D_FS(DD, NWW, true) } else { S3D_FS(DD, NWW, false) }
    switch (a.meta.D) {
        case 3: S3D_FS_D(3, 8)
        case 6: S3D_FS_D(6, 8)
        case 9: S3D_FS_D(9, 10)
        default: return S3D_ERR_UNSUPPORTED;
    }
#undef S3D_FS_D
#undef S3D_FS
}

cudaError_t attn_tc_fwd_small_async_error(bool &set) { return take_async_error(set); }

}  // namespace s3d
