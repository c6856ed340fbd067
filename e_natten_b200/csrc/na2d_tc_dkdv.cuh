// Persistent, warp-specialised tcgen05 dK/dV kernel.  Included by na2d_tc.cuh.
//
// One CTA per SM walks key tiles (TH x TW keys, row r of every MMA = key r = tensor-memory lane
// r).  The queries that can see a tile form a box (the union of the keys' inverse
// neighbourhoods, clipped to the local query band), walked in chunks of RC rows x HW columns
// (at most NMAX queries).  Two forms.  STRIPS (from kernel size 7 on, where strips_pay says so): a chunk is a column strip as
// tall as the box of an inner tile.  A warp's 32 keys (four image rows) are seen from ks + 3 of its rows, the same share of every
// chunk, while of a group of rows some warps see everything and others nothing, and a chunk lasts as long as its busiest warp.
// Otherwise (kernel sizes 3 and 5, and images on which strips would mostly hang over the box): groups of box rows.
//     S^T = K Q_c^T,  dP^T = V dO_c^T                      (tensor memory, fp32)
//     P^T = exp(S^T - lse),  dS^T = scale P^T (dP^T - delta)   (softmax warps, registers; the scale is dK's)
//     dV += P^T dO_c,  dK += dS^T Q_c                      (P^T, dS^T read from tensor memory)
// P^T and dS^T are written back over S^T / dP^T as packed 16-bit pairs; on the bf16 path dS^T
// is written as head + residual (two MMAs), because one bf16 keeps too few bits for dK.
//
// Tensor memory holds two or three chunk stages (S^T, dP^T of NMAX columns each) next to the dV and dK
// accumulators, so the score MMAs of one chunk run while the softmax warps work on the previous
// one.  Sixteen warps: 0-7 softmax (warps w and w + 4 own the same 32 keys of a lane quarter and split
// the 8-column blocks of every chunk between them), 8 producer of the Q / dO chunk ring and of the chunks' lse and
// delta, 11 TMA producer of the K, V tile, 9 issues the score MMAs, 10 the output MMAs, 12-15 epilogue (dV, dK rows ->
// staging -> TMA store), which
// overlaps the next tile.  dK and dV accumulate in tensor memory over all chunks of a tile; no
// atomics.
//
// What bounds it: the chain score MMAs -> softmax warps -> output MMAs -> stage free, of which tensor memory holds two or three; the
// softmax part of it was cut by strips, packed fp32 pairs, and lse and delta handed over by the producer.  Measured on one B200
// against the chunks of box rows before: 32 x 2 x 56 x 56 x 32, window 7, bf16 104 -> 62 us; 16 x 8 x 28 x 28 x 64, window 13, bf16
// 135 -> 91 us (groups of rows, without strips); 16 x 16 x 14 x 14 x 64, window 13, fp16 39 -> 29 us; 8 heads of 1024 x 1024 x 128, window 13, bf16 7.8 -> 6.6 ms;
// 4 x 4 x 256 x 256 x 128, window 5, bf16 (the same chunks as before) 0.39 -> 0.375 ms.
#pragma once

#include <algorithm>

namespace na2d_tc {

// Chunks of an interior tile's query box when the box is cut into `split` column strips.
constexpr int dkv_chunks(int ks, int split) {
    const int bw = TW + ks - 1, hh = TH + ks - 1;
    if (bw % split != 0 || 64 / (bw / split) == 0) return 1 << 20;
    const int rc_max = 64 / (bw / split);
    return (hh + rc_max - 1) / rc_max * split;
}
// Fewest chunks wins; on a tie the narrower strips, which spread the work evenly over the lane
// quarters (a key row group sees the same number of queries in every strip).
constexpr int dkv_w_split(int ks) {
    const int c1 = dkv_chunks(ks, 1), c2 = dkv_chunks(ks, 2), c4 = dkv_chunks(ks, 4);
    return (c4 <= c2 && c4 <= c1) ? 4 : (c2 <= c1 ? 2 : 1);
}

constexpr unsigned long long row_repeat(int hw, int rc) {
    unsigned long long m = 0;
    for (int r = 0; r < rc; ++r) m |= 1ull << (r * hw);
    return m;
}

// Queries per chunk at most: 2 x (S^T + dP^T) + dV + dK in 512 columns.  (Groups of rows are kept to 64.)
constexpr int dkv_nmax(int d, bool strips) { return !strips || d == 128 ? 64 : (512 - 2 * d) / 4 / 16 * 16; }
// Columns of a strip: 4 or 2, so that a column pattern repeats every 8 queries.
constexpr int dkv_strip(int d, int ks) { return (TH + ks - 1) * 4 <= dkv_nmax(d, true) ? 4 : 2; }
// Tensor-memory columns of S^T and of dP^T.
constexpr int dkv_cols(int d, int ks, bool strips) { return strips && dkv_strip(d, ks) == 4 ? dkv_nmax(d, strips) : 64; }

// (Cfg wants strips that tile the box: it is taken as wide as the next multiple of 8.)
constexpr int dkv_box_w(int ks) { return (TW + ks - 1 + 7) / 8 * 8; }
template <int D, int KS, bool STRIPS>
using DkvCfgBase = Cfg<D, KS, dkv_nmax(D, STRIPS), STRIPS ? dkv_box_w(KS) - (TW + KS - 1) : 0, STRIPS ? dkv_box_w(KS) / dkv_strip(D, KS) : dkv_w_split(KS)>;

template <int D, int KS, bool STRIPS>
struct DkvCfg : DkvCfgBase<D, KS, STRIPS> {
    using B = DkvCfgBase<D, KS, STRIPS>;
    // names of the base read as "queries per chunk" here: NK = queries in a chunk, NKP padded
    static constexpr bool PATTERN = STRIPS;                                // masks by pattern (HW divides 8)
    static constexpr int NMAX = dkv_cols(D, KS, STRIPS);
    static constexpr int TMEM_STAGE = 2 * NMAX;                            // columns per chunk stage
    // Chunk stages: a third one where it fits (head dims 32 and 64, chunks of up to 64 queries), which takes a chunk's MMAs out of the
    // softmax warps' way (16 x 8 x 28 x 28 x 64, window 13, bf16, on strips: 101 -> 98 us).
    static constexpr int NSTG = 3 * TMEM_STAGE <= 512 - 2 * D ? 3 : 2;
    static constexpr int TMEM_ST = 0, TMEM_DPT = NMAX, TMEM_DV = 512 - 2 * D, TMEM_DK = TMEM_DV + D;
    static constexpr int TMEM_PT = 0, TMEM_DST = NMAX / 2, TMEM_RES = NMAX;   // 16-bit operands over S^T / dP^T
    static constexpr int STAGE = 2 * B::KV_BYTES;                          // Q chunk then dO chunk
    static constexpr int OUT_BYTES = 4 * 2 * OutStage<32>::BYTES;          // two staging buffers for each of the 4 epilogue warps
    static constexpr int XCHG_BYTES = 4 * 2 * B::NKP * 4;                  // [ring slot]{-lse * log2(e), -delta * scale}[NKP]
    static constexpr int FIXED = 2 * B::Q_BYTES /*K, V tile*/ + OUT_BYTES + XCHG_BYTES + 256 + 1024;
    static constexpr int NSTQ = (FIXED + 4 * STAGE <= kSmemLimit) ? 4 : 3;
    static constexpr int SMEM = FIXED + NSTQ * STAGE;
    static constexpr int NB8 = B::NKP / 8;
    // A warp pair works on blocks b_lo .. b_lo + 2 NOWN - 1 in any case (what an inner tile needs), and on those beyond where a
    // tile at a border needs them: a warp's 32 / TW key rows are seen from at most that many + 2 ks - 2 query rows.
    static constexpr int kInner = (32 / TW - 1 + KS) < B::RC ? (32 / TW - 1 + KS) : B::RC;
    static constexpr int kMost = (32 / TW - 1 + 2 * KS - 1) < B::RC ? (32 / TW - 1 + 2 * KS - 1) : B::RC;
    static constexpr int half_blocks(int rows, bool aligned) {
        const int n = (rows * B::HW + 7) / 8 + (aligned ? 0 : 1);
        return ((n < NB8 ? n : NB8) + 1) / 2;
    }
    static constexpr int NOWN = half_blocks(kInner, PATTERN), NALL = half_blocks(kMost, false);
    static constexpr unsigned long long ROW_REP = PATTERN ? 0ull : row_repeat(B::HW, B::RC);
    static constexpr uint32_t REP8 = B::HW == 4 ? 0x11u : 0x55u;
    static_assert(SMEM <= kSmemLimit, "dK/dV kernel shared memory");
    static_assert(!PATTERN || B::HW == 2 || B::HW == 4, "strips of 2 or 4 columns");
    static_assert(!PATTERN || B::HW <= KS / 2 + 1, "no box is narrower than a strip");
    static_assert(B::NKP <= NMAX && NSTG * TMEM_STAGE <= TMEM_DV && TMEM_DK + D <= 512 && D % 32 == 0, "tensor memory layout");
    static_assert(NMAX % 16 == 0 && NB8 % 2 == 0 && NOWN <= NALL, "blocks in pairs");
};

template <typename DT, int D, int KS, bool STRIPS>
__global__ void __launch_bounds__(512, 1)
dkdv_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
            const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
            const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
            const float* __restrict__ lse, const float* __restrict__ delta, const int f32_out,
            const ErrorState* __restrict__ errors, const Na2dGeom g, const int tiles_r, const int tiles_c,
            const int total_tiles) {
    constexpr bool SPLIT = IsBf16<DT>::value;
    using C = DkvCfg<D, KS, STRIPS>;
    constexpr int NSTQ = C::NSTQ;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sK = smem;                               // key tile   [128 x D]
    uint8_t* sV = sK + C::Q_BYTES;                    // value tile [128 x D]
    uint8_t* sQD = sV + C::Q_BYTES;                   // NSTQ x (query chunk, dO chunk), each [NKP x D]
    uint8_t* sOut = sQD + NSTQ * C::STAGE;            // 4 x output staging (1024-byte aligned)
    float* s_x = reinterpret_cast<float*>(sOut + C::OUT_BYTES);   // [ring slot]{-lse * log2(e), -delta * scale}[NKP]
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_x + C::XCHG_BYTES / 4);
    uint64_t* kv_full = bars + 0;            //       TMA -> MMA
    uint64_t* kv_empty = bars + 1;           //       MMA (commit) -> TMA
    uint64_t* acc_full = bars + 2;           //       MMA (commit) -> epilogue
    uint64_t* acc_free = bars + 3;           //       epilogue -> MMA: dV and dK have been read
    uint64_t* accv_free = bars + 4;          //       epilogue -> MMA: dV has been read (dK follows)
    uint64_t* s_full = bars + 5;             // [3]   MMA (commit) -> softmax warps, per stage
    uint64_t* p_full = bars + 8;             // [3]   softmax warps -> MMA
    uint64_t* st_free = bars + 11;           // [3]   output MMAs (commit) -> score MMAs: the stage is free
    uint64_t* qd_full = bars + 14;           // [4]   TMA -> MMA
    uint64_t* qd_empty = bars + 18;          // [4]   MMA (commit) -> TMA
    uint64_t* x_full = bars + 22;            // [4]   producer -> score MMAs (and through them softmax): lse and delta
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
    const WaitCtx wctx{reinterpret_cast<WaitState*>(bars + 27)};
    constexpr int NSTG = C::NSTG;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_my = total_tiles > (int)blockIdx.x ? (total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;

    if (tid == 0) {
        wait_state_init(wctx.st, errors, kWaitLimitNs);
        mbar_init(kv_full, 1);
        mbar_init(kv_empty, 1);
        mbar_init(acc_full, 1);
        mbar_init(acc_free, 4);
        mbar_init(accv_free, 4);
        for (int i = 0; i < NSTG; ++i) {
            mbar_init(s_full + i, 1);
            mbar_init(p_full + i, 8);
            mbar_init(st_free + i, 1);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(qd_full + i, 1);
            mbar_init(qd_empty + i, 1);
            mbar_init(x_full + i, 1);
        }
        mbar_fence_init();
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_do);
        tma_prefetch_desc(&tm_dk);
        tma_prefetch_desc(&tm_dv);
    }
    // Rows [NK, NKP) of every query / dO chunk buffer are contraction rows of the output MMAs that
    // TMA never writes: zero them once.
    if constexpr (C::NKP > C::NK) {
        constexpr int pad16 = (C::NKP - C::NK) * C::ROWB / 16;
        for (int i = tid; i < NSTQ * 2 * C::NS * pad16; i += 512) {
            const int which = i / pad16, off = i - which * pad16;          // which = (stage * 2 + q/dO) * NS + slab
            const int slab = which % C::NS, buf = which / C::NS;
            uint8_t* base = sQD + (buf >> 1) * C::STAGE + (buf & 1) * C::KV_BYTES + slab * C::KV_SLAB;
            st_shared_v4(smem_u32(base + C::NK * C::ROWB + off * 16), 0u, 0u, 0u, 0u);
        }
        fence_proxy_async();
    }
    after_previous_grid();
    if (warp == 0) {
        __syncwarp();
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    next_grid_may_start();
    const uint32_t tmem_base = *tmem_slot;

    // Geometry of my i-th tile: key tile origin and the query box it is seen from.
    struct TileGeo { int bn, hn, hb, kr0, kc0, qb_r0, q_local_r0, n_rows, qb_c0, n_cols, n_cc, n_ch; };
    // (each role steps through the tiles by itself)
    TileWalk walk((int)blockIdx.x, (int)gridDim.x, tiles_r, tiles_c);
    auto tile_geo = [&](const TileWalk& at) {
        TileGeo t;
        t.kr0 = at.row();
        t.kc0 = at.col();
        t.bn = at.bn;
        split_unit(t.bn, g, t.hn, t.hb);
        const int kg_first = g.kv_row0 + t.kr0;
        const int kg_last = g.kv_row0 + min(t.kr0 + TH, g.Hkv) - 1;
        t.qb_r0 = max(na2d_bws(kg_first, KS), g.q_row0);                           // global row
        const int qb_r1 = min(na2d_bwe(kg_last, g.Hg, KS), g.q_row0 + g.Hq);
        t.n_rows = max(qb_r1 - t.qb_r0, 0);
        t.q_local_r0 = t.qb_r0 - g.q_row0;
        t.qb_c0 = na2d_bws(t.kc0, KS);
        t.n_cols = na2d_bwe(min(t.kc0 + TW, g.W) - 1, g.W, KS) - t.qb_c0;
        t.n_cc = (t.n_cols + C::HW - 1) / C::HW;         // strips; more where both borders stretch the box
        t.n_ch = ((t.n_rows + C::RC - 1) / C::RC) * t.n_cc;       // (divisions by constants)
        return t;
    };

    // First box column of strip cc.  The last one starts earlier where it would reach past the box, and takes no part of the columns
    // it shares with the one before: weights of zero meet no query outside the box, whose dO or q need not be finite.  (A box
    // is at least ks / 2 + 1 columns wide.)
    auto first_col = [](const TileGeo& t, int cc) { return C::PATTERN ? min(cc * C::HW, t.n_cols - C::HW) : cc * C::HW; };

    if (warp == 8) {
        // ------------------------------------------------------------------ producer of the Q / dO chunk ring
        // (the K, V tile has a producer of its own, warp 11: a chunk of the next tile can be
        // fetched as soon as a ring slot is free, long before the K, V buffers are)
        // The chunk's lse and delta go with it, as the softmax warps use them: lane l has queries l, l + 32, ...; they are read
        // one chunk ahead, so that their latency runs under the wait for a ring slot, and first touched when the chunk's loads are on
        // their way, which a tile's first chunk would wait for otherwise (a call of few tiles, 4 x 4 x 32 x 32 x 128, window 5, bf16:
        // 12.4 -> 11.8 us).
        reg_dec<kDkvRegsCtl>();
        constexpr int kPer = (C::NKP + 31) / 32;
        float pre_lse[kPer], pre_delta[kPer];
        auto fetch = [&](const TileGeo& t, int rc, int cc) {
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int j = lane + 32 * u, br = rc * C::RC + j / C::HW, qc = t.qb_c0 + first_col(t, cc) + j % C::HW;
                pre_lse[u] = pre_delta[u] = 0.f;                 // zero outside the band
                if (j < C::NK && br < t.n_rows && qc < g.W) {
                    const size_t qi = (static_cast<size_t>(t.bn) * g.Hq + (t.q_local_r0 + br)) * g.W + qc;
                    pre_lse[u] = lse[qi];
                    pre_delta[u] = delta[qi];
                }
            }
        };
        uint32_t n = 0;
        LoadTracker lt(bars);
        for (int i = 0; i < n_my && lt.ok; ++i, walk.next()) {
            const TileGeo t = tile_geo(walk);
            if (t.n_ch == 0) continue;
            fetch(t, 0, 0);
            for (int ch = 0, rc = 0, cc = 0; ch < t.n_ch; ++ch, ++n) {
                const uint32_t st = n % NSTQ;
                if (!lt.acquire_warp(qd_empty + st, ((n / NSTQ) & 1) ^ 1, wctx)) break;
                if (lane == 0) {
                    NA2D_TR(2, 7, n);
                    lt.arm(qd_full + st, (n / NSTQ) & 1, 2u * C::NS * C::NK * C::ROWB);
                    uint8_t* dst = sQD + st * C::STAGE;
                    const int col = t.qb_c0 + first_col(t, cc);
#pragma unroll
                    for (int s = 0; s < C::NS; ++s) {
                        tma_load_5d(dst + s * C::KV_SLAB, &tm_q, qd_full + st, s * 64, col, t.q_local_r0 + rc * C::RC, t.hn, t.hb);
                        tma_load_5d(dst + C::KV_BYTES + s * C::KV_SLAB, &tm_do, qd_full + st, s * 64, col,
                                    t.q_local_r0 + rc * C::RC, t.hn, t.hb);
                    }
                }
                float* x = s_x + st * 2 * C::NKP;
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const int j = lane + 32 * u;
                    if (j < C::NKP) {
                        x[j] = -(pre_lse[u] * kLog2e);
                        x[C::NKP + j] = -(pre_delta[u] * g.scale);      // dS^T carries the softmax scale of dK: scale p (dP - delta)
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(x_full + st);
                if (++cc == t.n_cc) {
                    cc = 0;
                    ++rc;
                }
                if (ch + 1 < t.n_ch) fetch(t, rc, cc);
            }
        }
        if (lane == 0) lt.drain(wctx);
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issue: scores
        // Two warps issue MMAs, so that the bookkeeping of one runs under the MMAs of the other:
        // this one the score MMAs of chunk n into stage n % NSTG, as soon as the chunk's Q / dO have
        // landed and the output MMAs of chunk n - NSTG (warp 10) have left the stage.  The whole warp
        // walks the loop with uniform control flow; one elected lane issues.
        reg_dec<kDkvRegsCtl>();
        constexpr uint32_t idesc_s = umma_idesc(TM, C::NKP, IsBf16<DT>::value, IsBf16<DT>::value, false, false);
        constexpr uint32_t hi = smem_desc_hi(C::ATOM, C::SWZ);
        const uint32_t k_lo = smem_desc_lo(smem_u32(sK), 16), v_lo = smem_desc_lo(smem_u32(sV), 16);
        const uint32_t qd_base = smem_u32(sQD);
        uint32_t n = 0, it = 0;
        for (int i = 0; i < n_my; ++i, walk.next()) {
            const TileGeo t = tile_geo(walk);
            if (t.n_ch == 0) continue;
            for (int ch = 0; ch < t.n_ch; ++ch, ++n) {
                const uint32_t q_addr = qd_base + (n % NSTQ) * C::STAGE, g_addr = q_addr + C::KV_BYTES;
                const uint32_t q_lo = smem_desc_lo(q_addr, 16), g_lo = smem_desc_lo(g_addr, 16);
                const uint32_t tm = tmem_base + (n % NSTG) * C::TMEM_STAGE;
                if (lane == 0) NA2D_TR(2, 0, n);
                if (ch == 0) mbar_wait(kv_full, it & 1, wctx, kErrLoadWait);
                if (lane == 0) NA2D_TR(2, 1, n);
                mbar_wait(qd_full + n % NSTQ, (n / NSTQ) & 1, wctx, kErrLoadWait);
                mbar_wait(x_full + n % NSTQ, (n / NSTQ) & 1, wctx, kErrLoadWait);
                if (lane == 0) NA2D_TR(2, 3, n);
                mbar_wait(st_free + n % NSTG, ((n / NSTG) & 1) ^ 1, wctx, kErrMmaWait);
                if (lane == 0) NA2D_TR(2, 5, n);
                tc_fence_after();
                if (elect_one()) {
                    // the S^T and dP^T chains alternate
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        constexpr int kPerSlab = C::SLAB_C / 16;
                        const int slab = kk / kPerSlab, in_slab = kk % kPerSlab;
                        umma_ss(tm + C::TMEM_ST, desc64(hi, k_lo + ((slab * C::Q_SLAB) >> 4) + 2 * in_slab),
                                desc64(hi, q_lo + ((slab * C::KV_SLAB) >> 4) + 2 * in_slab), idesc_s, kk > 0);
                        umma_ss(tm + C::TMEM_DPT, desc64(hi, v_lo + ((slab * C::Q_SLAB) >> 4) + 2 * in_slab),
                                desc64(hi, g_lo + ((slab * C::KV_SLAB) >> 4) + 2 * in_slab), idesc_s, kk > 0);
                    }
                    umma_commit(s_full + n % NSTG);
                    if (ch == t.n_ch - 1) umma_commit(kv_empty);       // K and V are only read by the score MMAs
                    NA2D_TR(2, 2, n);
                }
                __syncwarp();
            }
            ++it;
        }
    } else if (warp == 10) {
        // ------------------------------------------------------------------ MMA issue: outputs
        // dV += P^T dO, dK += dS^T Q of chunk n out of stage n % NSTG, when the chunk's softmax group
        // has written the operands (and, for a tile's first chunk, the epilogue has read the
        // previous tile's accumulators).
        reg_dec<kDkvRegsCtl>();
        constexpr uint32_t idesc_o = umma_idesc(TM, D, IsBf16<DT>::value, IsBf16<DT>::value, false, true);
        constexpr uint32_t hi = smem_desc_hi(C::ATOM, C::SWZ);
        const uint32_t qd_base = smem_u32(sQD);
        uint32_t n = 0, it = 0;
        for (int i = 0; i < n_my; ++i, walk.next()) {
            const TileGeo t = tile_geo(walk);
            if (t.n_ch == 0) continue;
            for (int ch = 0; ch < t.n_ch; ++ch, ++n) {
                const uint32_t q_addr = qd_base + (n % NSTQ) * C::STAGE, g_addr = q_addr + C::KV_BYTES;
                const uint32_t qm_lo = smem_desc_lo(q_addr, C::KV_SLAB), gm_lo = smem_desc_lo(g_addr, C::KV_SLAB);
                const uint32_t tm = tmem_base + (n % NSTG) * C::TMEM_STAGE;
                const uint32_t acc = ch == 0 ? 0u : 1u;
                mbar_wait(p_full + n % NSTG, (n / NSTG) & 1, wctx, kErrMmaWait);
                if (ch == 0) {
                    // A tile's first chunk overwrites the accumulators the epilogue warps are still
                    // reading out for the previous tile.  They read dV first and say so, so its dV
                    // MMAs go ahead of its dK MMAs and only the latter wait for the whole read-out.
                    mbar_wait(accv_free, (it & 1) ^ 1, wctx, kErrMmaWait);
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < C::NKP / 16; ++kk)
                            umma_ts(tmem_base + C::TMEM_DV, tm + C::TMEM_PT + 8 * kk,
                                    desc64(hi, gm_lo + ((kk * 16 * C::ROWB) >> 4)), idesc_o, kk > 0);
                    }
                    __syncwarp();
                    mbar_wait(acc_free, (it & 1) ^ 1, wctx, kErrMmaWait);
                }
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < C::NKP / 16; ++kk) {               // dK and dV chains alternate
                        umma_ts(tmem_base + C::TMEM_DK, tm + C::TMEM_DST + 8 * kk,
                                desc64(hi, qm_lo + ((kk * 16 * C::ROWB) >> 4)), idesc_o, acc | (kk > 0));
                        if (ch != 0)
                            umma_ts(tmem_base + C::TMEM_DV, tm + C::TMEM_PT + 8 * kk,
                                    desc64(hi, gm_lo + ((kk * 16 * C::ROWB) >> 4)), idesc_o, 1u);
                    }
                    if (SPLIT) {
#pragma unroll
                        for (int kk = 0; kk < C::NKP / 16; ++kk)
                            umma_ts(tmem_base + C::TMEM_DK, tm + C::TMEM_RES + 8 * kk,
                                    desc64(hi, qm_lo + ((kk * 16 * C::ROWB) >> 4)), idesc_o, 1u);
                    }
                    umma_commit(qd_empty + (n % NSTQ));
                    umma_commit(st_free + n % NSTG);
                    if (ch == t.n_ch - 1) umma_commit(acc_full);
                    NA2D_TR(2, 4, n);
                }
                __syncwarp();
            }
            ++it;
        }
    } else if (warp == 11) {
        // ------------------------------------------------------------------ producer of the K, V tile
        reg_dec<kDkvRegsCtl>();
        if (lane == 0) {
            uint32_t it = 0;                            // non-empty tile counter
            LoadTracker lt(bars);
            for (int i = 0; i < n_my; ++i, walk.next()) {
                const TileGeo t = tile_geo(walk);
                if (t.n_ch == 0) continue;
                if (!lt.acquire(kv_empty, (it & 1) ^ 1, wctx)) break;
                lt.arm(kv_full, it & 1, 2u * C::Q_BYTES);
#pragma unroll
                for (int s = 0; s < C::NS; ++s) {
                    tma_load_5d(sK + s * C::Q_SLAB, &tm_k, kv_full, s * 64, t.kc0, t.kr0, t.hn, t.hb);
                    tma_load_5d(sV + s * C::Q_SLAB, &tm_v, kv_full, s * 64, t.kc0, t.kr0, t.hn, t.hb);
                }
                ++it;
                // The single K, V buffer is only free again after this tile's last score MMAs, and a
                // load from HBM issued then is what the next tile would wait for: bring the next
                // tile's K, V into L2 now.
                if (i + 1 < n_my) {
                    TileWalk ahead = walk;
                    ahead.next();
                    const TileGeo tn = tile_geo(ahead);
#pragma unroll
                    for (int s = 0; s < C::NS; ++s) {
                        tma_prefetch_5d(&tm_k, s * 64, tn.kc0, tn.kr0, tn.hn, tn.hb);
                        tma_prefetch_5d(&tm_v, s * 64, tn.kc0, tn.kr0, tn.hn, tn.hb);
                    }
                }
            }
            lt.drain(wctx);
        }
    } else if (warp >= 12) {
        // ------------------------------------------------------------------ epilogue warps
        reg_dec<kDkvRegsEpi>();
        const int quarter = warp & 3;
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        uint8_t* stage = sOut + quarter * 2 * OutStage<32>::BYTES;
        constexpr int RPO = D / 32;                          // 32-channel rounds per output
        uint32_t it = 0, seq = 0;
        for (int i = 0; i < n_my; ++i, walk.next()) {
            const TileGeo t = tile_geo(walk);
            if (t.n_ch == 0) {                               // no local query sees this tile: zeros
                uint32_t z[32];
#pragma unroll
                for (int e = 0; e < 32; ++e) z[e] = 0u;
#pragma unroll
                for (int j = 0; j < 2 * RPO; ++j) {
                    if (f32_out)
                        stage_and_store_f32<32, 2>(j / RPO == 0 ? &tm_dv : &tm_dk, stage, z, 1.f, 32 * (j % RPO), t.kc0,
                                                   t.kr0 + quarter * (32 / TW), t.hn, t.hb, lane, &seq);
                    else
                        stage_and_store<DT, 32, 2>(j / RPO == 0 ? &tm_dv : &tm_dk, stage, z, 1.f, 32 * (j % RPO), t.kc0,
                                                   t.kr0 + quarter * (32 / TW), t.hn, t.hb, lane, &seq);
                }
                continue;
            }
            if (warp == 12 && lane == 0) NA2D_TR(0, 0, it);
            mbar_wait(acc_full, it & 1, wctx, kErrMmaWait);
            tc_fence_after();
            if (warp == 12 && lane == 0) NA2D_TR(0, 1, it);
            const int h0 = t.kr0 + quarter * (32 / TW);
            // 2 * RPO rounds of 32 columns, the load of the next round in flight while one is stored
            uint32_t v[2][32];
            tmem_ld_32x32(tmem_lane + C::TMEM_DV, v[0]);
#pragma unroll
            for (int j = 0; j < 2 * RPO; ++j) {
                tmem_ld_wait();
                if (j == RPO - 1) {                          // dV is in registers (or stored)
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accv_free);
                }
                if (j + 1 < 2 * RPO) {
                    const int which = (j + 1) / RPO, r = (j + 1) % RPO;
                    tmem_ld_32x32(tmem_lane + (which == 0 ? C::TMEM_DV : C::TMEM_DK) + 32 * r, v[(j + 1) & 1]);
                } else {                                     // both accumulators are in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_free);
                    if (warp == 12 && lane == 0) NA2D_TR(0, 2, it);
                }
                // (the softmax scale of dK is already in dS^T: the epilogue only converts)
                if (f32_out)
                    stage_and_store_f32<32, 2, false>(j / RPO == 0 ? &tm_dv : &tm_dk, stage, v[j & 1], 1.f, 32 * (j % RPO),
                                                      t.kc0, h0, t.hn, t.hb, lane, &seq);
                else
                    stage_and_store<DT, 32, 2, false>(j / RPO == 0 ? &tm_dv : &tm_dk, stage, v[j & 1], 1.f, 32 * (j % RPO),
                                                      t.kc0, h0, t.hn, t.hb, lane, &seq);
            }
            if (warp == 12 && lane == 0) NA2D_TR(0, 3, it);
            ++it;
        }
        if (lane == 0) bulk_wait<0>();                       // the staging buffer has been read, the rows written
    } else {
        // ------------------------------------------------------------------ softmax groups
        // Both groups work on every chunk: warps w and w + 4 own the same 32 keys (tensor-memory
        // lanes) and take alternate 8-column blocks of the warp's active range, so a chunk's S^T and
        // dP^T spend half as long in registers before the output MMAs may start - that time is part
        // of the chain that bounds the kernel (score MMAs -> this -> output MMAs -> stage free).  The blocks an inner tile
        // needs are done without a branch between them: their chains of loads, exponentials and conversions overlap.
        reg_inc<kDkvRegsSoftmax>();
        const int quarter = warp & 3, group = warp >> 2;
        const int row = quarter * 32 + lane;                 // key of the tile = tensor-memory lane
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        const uint64_t sl2 = pair2(g.sl2, g.sl2), scale2 = pair2(g.scale, g.scale);
        constexpr int NOWN = C::NOWN, NALL = C::NALL;

        uint32_t n = 0;
        for (int i = 0; i < n_my; ++i, walk.next()) {
            const TileGeo t = tile_geo(walk);
            if (t.n_ch == 0) continue;
            const int kr = min(t.kr0 + (row / TW), g.Hkv - 1), kc = min(t.kc0 + (row % TW), g.W - 1);
            // the queries that see this thread's key: box rows [row_lo, row_hi), box columns [col_lo, col_hi)
            const int kg = g.kv_row0 + kr;
            const int row_lo = max(na2d_bws(kg, KS), g.q_row0) - t.qb_r0;
            const int row_hi = min(na2d_bwe(kg, g.Hg, KS), g.q_row0 + g.Hq) - t.qb_r0;
            const int col_lo = na2d_bws(kc, KS) - t.qb_c0;
            const int col_hi = na2d_bwe(kc, g.W, KS) - t.qb_c0;
            const int wrow_lo = __shfl_sync(0xffffffffu, row_lo, 0);
            const int wrow_hi = __shfl_sync(0xffffffffu, row_hi, 31);

            // of the chunk rows from r_off on: the warp's active blocks, the first one it takes, and this key's rows in
            // them (one bit a query)
            int b_hi = 0, b0 = 0;
            uint32_t rows8[NALL];                            // of the blocks b0 + 2 a + group
            unsigned long long rows64 = 0;                   // (general strips: of the chunk)
            auto row_part = [&](int r_off) {
                const int ra = max(wrow_lo - r_off, 0), rb = min(wrow_hi - r_off, C::RC);
                b_hi = rb > ra ? (min(rb * C::HW, C::NK) + 7) >> 3 : 0;
                b0 = min(rb > ra ? (ra * C::HW) >> 3 : 0, C::NB8 - 2 * NOWN);
                const int ta = max(row_lo - r_off, 0) * C::HW, tb = max(min(row_hi - r_off, C::RC), 0) * C::HW;
                if constexpr (C::PATTERN) {
#pragma unroll
                    for (int a = 0; a < NALL; ++a) rows8[a] = range_bits<8>(ta, tb, 8 * (b0 + 2 * a + group));
                } else {
                    rows64 = tb > ta ? (tb >= 64 ? ~0ull : (1ull << tb) - 1ull) & ~((1ull << ta) - 1ull) : 0ull;      // ta < 64
                }
            };
            row_part(0);

            for (int ch = 0, rc = 0, cc = 0; ch < t.n_ch; ++ch, ++n) {
                const uint32_t stage = n % NSTG, k = n / NSTG;  // tensor-memory stage and its use counter
                const uint32_t t_stage = tmem_lane + stage * C::TMEM_STAGE;
                const int c_off = first_col(t, cc);         // chunk ch = rc * n_cc + cc
                if (quarter == 0 && lane == 0) NA2D_TR(3 - 2 * group, 0, n);
                const float* x_lse = s_x + (n % NSTQ) * 2 * C::NKP;
                const float* x_delta = x_lse + C::NKP;
                // this thread's column segment inside a chunk row; the chunk's queries that see its key
                const int cl = C::PATTERN ? max(col_lo, cc * C::HW) - c_off : max(col_lo - c_off, 0), seg_len = min(col_hi - c_off, C::HW) - cl;
                const uint32_t seg = seg_len > 0 ? ((1u << seg_len) - 1u) : 0u;
                uint32_t cols8 = 0;
                unsigned long long m64 = 0;
                if constexpr (C::PATTERN) cols8 = (seg << cl) * C::REP8;
                else m64 = ((C::ROW_REP * seg) << cl) & rows64;
                auto seen = [&](int a) {                    // of block b0 + 2 a + group
                    return C::PATTERN ? rows8[a] & cols8 : static_cast<uint32_t>(m64 >> (8 * (b0 + 2 * a + group))) & 0xffu;
                };

                mbar_wait(s_full + stage, k & 1, wctx, kErrMmaWait);
                tc_fence_after();
                if (quarter == 0 && lane == 0) NA2D_TR(3 - 2 * group, 2, n);
                uint32_t s[NALL][8], dp[NALL][8];
#pragma unroll
                for (int a = 0; a < NALL; ++a) {
                    const int blk = b0 + 2 * a + group;
                    if (a < NOWN || blk < b_hi) {                           // warp-uniform
                        tmem_ld_32x8(t_stage + C::TMEM_ST + 8 * blk, s[a]);
                        tmem_ld_32x8(t_stage + C::TMEM_DPT + 8 * blk, dp[a]);
                    }
                }
                tmem_ld_wait();
                // The 16-bit operands go over S^T / dP^T, a block's over other blocks' columns: the
                // partner warp must have its blocks in registers too before either of them writes.
                bar_sync(1 + quarter, 64);
                if (quarter == 0 && lane == 0) NA2D_TR(3 - 2 * group, 3, n);
                auto block = [&](int a, uint32_t (&wp)[4], uint32_t (&wd)[4], uint32_t (&wr2)[4]) {
                    const int blk = b0 + 2 * a + group;
                    const uint32_t vmask = seen(a);
#pragma unroll
                    for (int e4 = 0; e4 < 2; ++e4) {
                        const ulonglong2 nl = *reinterpret_cast<const ulonglong2*>(x_lse + 8 * blk + 4 * e4);
                        const ulonglong2 nd = *reinterpret_cast<const ulonglong2*>(x_delta + 8 * blk + 4 * e4);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int e = 4 * e4 + 2 * h, e2 = e / 2;
                            const bool ok0 = (vmask >> e) & 1u, ok1 = (vmask >> (e + 1)) & 1u;
                            const uint64_t x = fma2(pair2(s[a][e], s[a][e + 1]), sl2, h ? nl.y : nl.x);
                            const uint64_t pe = pair2(fast_exp2(lo2(x)), fast_exp2(hi2(x)));
                            const uint64_t de = mul2(pe, fma2(pair2(dp[a][e], dp[a][e + 1]), scale2, h ? nd.y : nd.x));
                            const float ds0 = ok0 ? lo2(de) : 0.f, ds1 = ok1 ? hi2(de) : 0.f;    // select, never multiply by zero
                            wp[e2] = pack2<DT>(ok0 ? lo2(pe) : 0.f, ok1 ? hi2(pe) : 0.f);
                            wd[e2] = pack2<DT>(ds0, ds1);
                            wr2[e2] = SPLIT ? pack2_residual_bf16(ds0, ds1, wd[e2]) : 0u;
                        }
                    }
                };
                auto store = [&](int a, const uint32_t (&wp)[4], const uint32_t (&wd)[4], const uint32_t (&wr2)[4]) {
                    const int blk = b0 + 2 * a + group;
                    tmem_st_32x4(t_stage + C::TMEM_PT + 4 * blk, wp);
                    tmem_st_32x4(t_stage + C::TMEM_DST + 4 * blk, wd);
                    if (SPLIT) tmem_st_32x4(t_stage + C::TMEM_RES + 4 * blk, wr2);
                };
                {   // blocks outside the active range hold zeros (this warp: every other one of them)
                    const uint32_t z[4] = {0u, 0u, 0u, 0u};
                    const int b_end = max(b_hi, b0 + 2 * NOWN);
#pragma unroll
                    for (int b = 0; b < C::NB8 / 2; ++b) {
                        const int blk = 2 * b + ((group ^ b0) & 1);         // the blocks of b0's parity are group 0's
                        if (blk < b0 || blk >= b_end) {
                            tmem_st_32x4(t_stage + C::TMEM_PT + 4 * blk, z);
                            tmem_st_32x4(t_stage + C::TMEM_DST + 4 * blk, z);
                            if (SPLIT) tmem_st_32x4(t_stage + C::TMEM_RES + 4 * blk, z);
                        }
                    }
                }
                if (quarter == 0 && lane == 0) NA2D_TR(3 - 2 * group, 6, n);
                // (all blocks first, then their stores: a store waits for its block's conversions)
                uint32_t wp[NOWN][4], wd[NOWN][4], wr2[NOWN][4];
#pragma unroll
                for (int a = 0; a < NOWN; ++a) block(a, wp[a], wd[a], wr2[a]);
#pragma unroll
                for (int a = 0; a < NOWN; ++a) store(a, wp[a], wd[a], wr2[a]);
#pragma unroll
                for (int a = NOWN; a < NALL; ++a)
                    if (b0 + 2 * a + group < b_hi) {
                        block(a, wp[0], wd[0], wr2[0]);
                        store(a, wp[0], wd[0], wr2[0]);
                    }
                if (quarter == 0 && lane == 0) NA2D_TR(3 - 2 * group, 4, n);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + stage);
                if (quarter == 0 && lane == 0) NA2D_TR(3 - 2 * group, 5, n);
                if (++cc == t.n_cc) {
                    cc = 0;
                    if (ch + 1 < t.n_ch) row_part(++rc * C::RC);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <typename DT, int D, int KS, bool STRIPS>
int launch_dkdv_as(const LaunchCtx& lc, const TensorArg& q, const TensorArg& k, const TensorArg& v, const float* lse,
                   const TensorArg& d_o, const float* delta, const TensorArg& d_k, const TensorArg& d_v) {
    using C = DkvCfg<D, KS, STRIPS>;
    const Na2dGeom& g = lc.g;
    CUtensorMap tk, tv, tq, tg, tdk, tdv;
    int rc = make_map(&tk, k, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, TW, TH);
    const int out_c = lc.dkdv_f32 ? 16 : 32;
    if (rc == NA2D_OK) rc = make_map(&tdk, d_k, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, TW, 32 / TW, out_c, lc.dkdv_f32);
    if (rc == NA2D_OK) rc = make_map(&tdv, d_v, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, TW, 32 / TW, out_c, lc.dkdv_f32);
    if (rc == NA2D_OK) rc = make_map(&tv, v, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, TW, TH);
    if (rc == NA2D_OK) rc = make_map(&tq, q, lc.dtype, lc.B, g.N, g.Hq, g.W, D, C::HW, C::RC);
    if (rc == NA2D_OK) rc = make_map(&tg, d_o, lc.dtype, lc.B, g.N, g.Hq, g.W, D, C::HW, C::RC);
    if (rc != NA2D_OK) return rc;
    const int tiles_r = (g.Hkv + TH - 1) / TH, tiles_c = (g.W + TW - 1) / TW;
    const long long tiles = (long long)g.BN * tiles_r * tiles_c;
    if (tiles > 0x7fffffffLL) return NA2D_ERR_TOO_LARGE;
    auto kern = dkdv_kernel<DT, D, KS, STRIPS>;
    static std::atomic<unsigned long long> opted{0};
    if (opt_in_smem(kern, C::SMEM, lc.device, opted) != cudaSuccess) return NA2D_ERR_CUDA;
    const int grid = persistent_grid(lc, tiles);
    *lc.launched += 1;
    return na2d_launch::launch(lc.overlap, kern, grid, 512, C::SMEM, lc.st,
                               tk, tv, tq, tg, tdk, tdv, lse, delta, lc.dkdv_f32 ? 1 : 0, lc.errors, g, tiles_r, tiles_c, (int)tiles) == cudaSuccess
               ? NA2D_OK
               : NA2D_ERR_CUDA;
}

// What the chunks of one unit cost in one of the forms: each `per_chunk`, and `per_block` for an 8-query block of its busiest warp.
template <class C>
long long dkv_cost(const Na2dGeom& g, int per_chunk, int per_block) {
    long long rows = 0, strips = 0;
    for (int r0 = 0; r0 < g.Hkv; r0 += TH) {
        const int first = g.kv_row0 + r0, last = g.kv_row0 + std::min(r0 + TH, g.Hkv) - 1;
        const int top = std::max(na2d_bws(first, g.ks), g.q_row0), end = std::min(na2d_bwe(last, g.Hg, g.ks), g.q_row0 + g.Hq);
        for (int at = top; at < end; at += C::RC) {
            int busiest = C::PATTERN ? (C::kInner * C::HW + 7) / 8 : 0;
            for (int key = first; key <= last; key += 32 / TW) {
                const int lo = std::max(na2d_bws(key, g.ks) - at, 0);
                const int hi = std::min(na2d_bwe(std::min(key + 32 / TW - 1, last), g.Hg, g.ks) - at, C::RC);
                if (hi > lo) busiest = std::max(busiest, (hi * C::HW + 7) / 8 - lo * C::HW / 8);
            }
            rows += per_chunk + per_block * busiest;
        }
    }
    for (int c0 = 0; c0 < g.W; c0 += TW)
        strips += (na2d_bwe(std::min(c0 + TW, g.W) - 1, g.W, g.ks) - na2d_bws(c0, g.ks) + C::HW - 1) / C::HW;
    return rows * strips;
}

// Whether column strips are the faster form.  On a border tile, whose box is smaller, a strip is still a whole inner box tall, and on
// images of less than two or three windows most tiles are border tiles: 4 x 8 x 18 x 64 x 128, window 11, bf16 33 % slower than with
// the groups of rows that strips replaced.  The weights are fitted to 216 points (head dims 32, 64, 128, windows 7 to 13, images of
// 14 x 14 to 128 x 128, one B200): the form chosen takes 1.007 times the better one's time on average, 1.17 times at worst
// (2 x 8 x 100 x 14 x 128, window 7).
template <int D, int KS>
bool strips_pay(const Na2dGeom& g) {
    return dkv_cost<DkvCfg<D, KS, true>>(g, 3, 6) <= dkv_cost<DkvCfg<D, KS, false>>(g, 12, 4);
}

template <typename DT, int D, int KS>
int launch_dkdv(const LaunchCtx& lc, const TensorArg& q, const TensorArg& k, const TensorArg& v, const float* lse,
                const TensorArg& d_o, const float* delta, const TensorArg& d_k, const TensorArg& d_v) {
    if constexpr (KS >= 7) {
        if (strips_pay<D, KS>(lc.g)) return launch_dkdv_as<DT, D, KS, true>(lc, q, k, v, lse, d_o, delta, d_k, d_v);
    }
    return launch_dkdv_as<DT, D, KS, false>(lc, q, k, v, lse, d_o, delta, d_k, d_v);
}

}  // namespace na2d_tc
