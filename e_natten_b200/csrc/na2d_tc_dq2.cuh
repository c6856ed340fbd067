// Persistent, warp-specialised tcgen05 dQ kernel of the larger windows (several key chunks), for calls that bring an
// estimate of delta.  Included by na2d_tc_dq.cu.  Math, operands and warps are those of na2d_tc_bwd.cuh, but a
// tile's chunks are walked once, and two chunks are in flight.
//
// One walk.  delta needs every chunk before any dS can be formed exactly.  The caller hands in an estimate d~ of it
// (in `delta`: dO . o from the stored output, see na2d_delta.cuh; off by the rounding of o, a few 1e-2 at most).  Every
// unit forms dS~ = p (dP - d~), adds dS~ K_c to dQ and, with one more MMA, p K_c to a second accumulator B, while
// the exact delta = sum_j p dP builds up in registers.  Since
// sum_j p (dP - delta) k = sum_j p (dP - d~) k - (delta - d~) sum_j p k, the epilogue stores
// scale (dQ - (delta - d~) B).  B only meets the small factor (delta - d~), so a single 16-bit p is enough for
// it.  The exact delta is what the kernel writes out for the dK/dV kernel.
//
// Two chunks in flight.  With one S / dP buffer the walk is bound by latency: score MMAs, softmax and dQ MMAs run
// one after the other.  Here a chunk is smaller (dq2_nmax keys), tensor memory holds two S / dP buffers beside dQ
// and B, and the score MMAs of the next chunk (of the next tile, too) run under a chunk's softmax, its dQ MMAs
// under the next chunk's.  Chunks are column strips (na2d_tc_strip.cuh), four warps of their own do the epilogue, and the next
// tile's state is worked out before this one's last chunk is waited for.
//
// What bounds it: at head dim 128 the issuing warp and the tensor pipe (28 MMAs a chunk, some 1500 cycles of pipe, 2000 to 2100
// a chunk as run), below that the softmax warps' chain.  Measured on one B200, query half with the delta estimate, one chunk
// in flight -> two chunks of box rows -> two column strips: 32 x 2 x 56 x 56 x 32, window 7, bf16 130 -> 97 -> 63 us;
// 16 x 8 x 28 x 28 x 64, window 13, bf16 130 -> 92 -> 74 us; 8 heads of 1024 x 1024 x 128, window 13, bf16 - -> 7.86 -> 7.16 ms.
// (At head dim 128, window 9, two columns fill 48 of the 64 keys a chunk can have, eight chunks for six of rows: the same time on large images,
// 2 to 7 % more on small ones, 4 x 4 x 32 x 32 15.9 -> 17.0 us.)
#pragma once

namespace na2d_tc {

// Keys per chunk at most: 2 x (S + dP) + dQ + B in 512 columns.
constexpr int dq2_nmax(int d) { return (512 - 2 * d) / 4 / 16 * 16; }
constexpr int dq2_strip(int d, int ks) { return (TH + ks - 1) * 4 <= dq2_nmax(d) ? 4 : 2; }

template <int D, int KS>
struct Dq2Cfg : StripCfg<D, KS, dq2_strip(D, KS)> {
    using B = StripCfg<D, KS, dq2_strip(D, KS)>;
    static constexpr int NMAX = dq2_nmax(D);
    static constexpr int TMEM_S = 0;                                   // per buffer
    static constexpr int TMEM_DP = NMAX;
    static constexpr int TMEM_BUF = 2 * NMAX;                          // columns of a buffer
    static constexpr int TMEM_DQ = 4 * NMAX;
    static constexpr int TMEM_BK = TMEM_DQ + D;                        // sum_j p k
    static constexpr int TMEM_DSH = TMEM_DP;                           // dS (head) over dP
    static constexpr int TMEM_RES = TMEM_S;                            // dS residual: lower half of S
    static constexpr int TMEM_PH = TMEM_S + B::NKP / 2;                // p: upper half of S
    static constexpr int OUT_BYTES = 4 * 2 * OutStage<32>::BYTES;      // two staging buffers for each epilogue warp
    static constexpr int XCHG_BYTES = (2 + 2) * 128 * 4;               // delta parts [2][128], corrections [2][128]
    static constexpr int FIXED = OUT_BYTES + XCHG_BYTES + 256 + 1024;
    // Ring depths.  A K slot is free when the dQ MMAs that read it are done, and the scores of the chunk after next are
    // the next thing the pipe is given: with two slots it would wait there for a load, with three or four the
    // chunk is in place.  A second Q / dO tile where it fits beside those.
    static constexpr bool fits(int nq, int nk, int nv) {
        return FIXED + nq * 2 * B::Q_BYTES + (nk + nv) * B::KV_BYTES <= kSmemLimit;
    }
    static constexpr int NSTK = fits(1, 4, 3) ? 4 : 3;
    static constexpr int NSTV = fits(1, NSTK, 3) ? 3 : 2;
    static constexpr int NQ = fits(2, NSTK, NSTV) ? 2 : 1;
    static constexpr int SMEM = FIXED + NQ * 2 * B::Q_BYTES + (NSTK + NSTV) * B::KV_BYTES;
    static constexpr int NB8 = B::NKP / 8;                             // 8-column blocks of S
    // A warp pair works on blocks b0 .. b0 + 2 NOWN - 1 in any case (what ks + 3 rows fill where they start on a block
    // boundary, as they do away from the borders), and on one more pair where the rows reach past those.
    static constexpr int NOWN = (((KS + 3) * B::HW + 7) / 8 + 1) / 2;
    static_assert(NB8 % 2 == 0 && 2 * NOWN <= NB8, "blocks in pairs");
    static_assert(SMEM <= kSmemLimit, "dQ kernel shared memory");
    static_assert(B::NKP <= NMAX && TMEM_BK + D <= 512, "tensor memory layout");
    static_assert((B::NKP / 2) % 8 == 0, "operand halves start on a block boundary");
};

template <typename DT, int D, int KS>
__global__ void __launch_bounds__(512, 1)
dq2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
           const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
           const __grid_constant__ CUtensorMap tm_dq, const float* __restrict__ lse, float* delta, const ErrorState* __restrict__ errors,
           const Na2dGeom g, const int tiles_r, const int tiles_c, const int total_tiles) {
    constexpr bool SPLIT = IsBf16<DT>::value;
    using C = Dq2Cfg<D, KS>;
    constexpr int NCH = C::NCH;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;
    constexpr int NSTK = C::NSTK, NSTV = C::NSTV, NQ = C::NQ;
    uint8_t* sDO = sQ + NQ * C::Q_BYTES;              // NQ x dO tile (and NQ x Q tile before it)
    uint8_t* sK = sDO + NQ * C::Q_BYTES;              // NSTK x key chunk   [NKP x D]
    uint8_t* sV = sK + NSTK * C::KV_BYTES;            // NSTV x value chunk [NKP x D]
    uint8_t* sOut = sV + NSTV * C::KV_BYTES;          // 4 x 2 output staging (1024-byte aligned)
    float* x_sum = reinterpret_cast<float*>(sOut + C::OUT_BYTES);     // [tile parity][row] half 1's part of delta
    float* x_corr = x_sum + 2 * 128;                                  // [tile parity][row] delta - estimate
    uint64_t* bars = reinterpret_cast<uint64_t*>(x_corr + 2 * 128);
    uint64_t* q_full = bars + 0;             // [2] TMA -> MMA (Q and dO tile)
    uint64_t* q_empty = bars + 2;            // [2] MMA (commit) -> TMA
    uint64_t* k_full = bars + 4;             // [4]
    uint64_t* k_empty = bars + 8;            // [4]
    uint64_t* v_full = bars + 12;            // [4]
    uint64_t* v_empty = bars + 16;           // [4]
    uint64_t* s_full = bars + 20;            // [2] MMA (commit) -> softmax: S and dP are complete, per buffer
    uint64_t* p_full = bars + 22;            // [2] softmax -> MMA: dS and p are in tensor memory, per buffer
    uint64_t* dq_full = bars + 24;           // MMA (commit) -> epilogue
    uint64_t* dq_free = bars + 25;           // epilogue -> MMA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
    const WaitCtx wctx{reinterpret_cast<WaitState*>(bars + 27)};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_my = total_tiles > (int)blockIdx.x ? (total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const uint32_t total_units = (uint32_t)n_my * NCH;

    if (tid == 0) {
        wait_state_init(wctx.st, errors, kWaitLimitNs);
        for (int i = 0; i < 4; ++i) {
            mbar_init(k_full + i, 1);
            mbar_init(k_empty + i, 1);
            mbar_init(v_full + i, 1);
            mbar_init(v_empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full + i, 1);
            mbar_init(q_empty + i, 1);
            mbar_init(s_full + i, 1);
            mbar_init(p_full + i, 8);
        }
        mbar_init(dq_full, 1);
        mbar_init(dq_free, 4);
        mbar_fence_init();
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_do);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        tma_prefetch_desc(&tm_dq);
    }
    // K rows [NK, NKP) of every stage are contraction rows of dQ = dS K that TMA never writes: zero them once.
    if constexpr (C::NKP > C::NK) {
        constexpr int pad16 = (C::NKP - C::NK) * C::ROWB / 16;
        for (int i = tid; i < NSTK * C::NS * pad16; i += 512) {
            const int which = i / pad16, off = i - which * pad16;             // which = stage * NS + slab
            st_shared_v4(smem_u32(sK + (which / C::NS) * C::KV_BYTES + (which % C::NS) * C::KV_SLAB + C::NK * C::ROWB +
                                  off * 16), 0u, 0u, 0u, 0u);
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

    if (warp == 8) {
        // ------------------------------------------------------------------ producer
        reg_dec<kDkvRegsCtl>();
        if (lane == 0) {
            uint32_t n = 0;
            LoadTracker lt(bars);
            TileWalk walk((int)blockIdx.x, (int)gridDim.x, tiles_r, tiles_c);
            for (int i = 0; i < n_my && lt.ok; ++i) {
                const int r0 = walk.row(), c0 = walk.col();
                int hn, hb;
                split_unit(walk.bn, g, hn, hb);
                walk.next();                                               // from here on: the tile after
                const int box_r0 = na2d_ws(g.q_row0 + r0, g.Hg, KS) - g.kv_row0;
                const int box_c0 = na2d_ws(c0, g.W, KS);
                const int qb = i % NQ, qp = (i / NQ) & 1;
                if (!lt.acquire(q_empty + qb, qp ^ 1, wctx)) break;
                lt.arm(q_full + qb, qp, 2u * C::Q_BYTES);
#pragma unroll
                for (int s = 0; s < C::NS; ++s) {
                    tma_load_5d(sQ + qb * C::Q_BYTES + s * C::Q_SLAB, &tm_q, q_full + qb, s * 64, c0, r0, hn, hb);
                    tma_load_5d(sDO + qb * C::Q_BYTES + s * C::Q_SLAB, &tm_do, q_full + qb, s * 64, c0, r0, hn, hb);
                }
                // a single Q / dO buffer is only free again after this tile's last score MMAs: bring the next tile's into L2
                if (NQ == 1 && i + 1 < n_my) {
                    int hn1, hb1;
                    split_unit(walk.bn, g, hn1, hb1);
#pragma unroll
                    for (int s = 0; s < C::NS; ++s) {
                        tma_prefetch_5d(&tm_q, s * 64, walk.col(), walk.row(), hn1, hb1);
                        tma_prefetch_5d(&tm_do, s * 64, walk.col(), walk.row(), hn1, hb1);
                    }
                }
                for (int c = 0; c < NCH; ++c, ++n) {
                    const uint32_t sk = n % NSTK, pk = (n / NSTK) & 1, sv = n % NSTV, pv = (n / NSTV) & 1;
                    if (!lt.acquire(v_empty + sv, pv ^ 1, wctx)) break;
                    lt.arm(v_full + sv, pv, (uint32_t)C::NS * C::NK * C::ROWB);
#pragma unroll
                    for (int s = 0; s < C::NS; ++s)
                        tma_load_5d(sV + sv * C::KV_BYTES + s * C::KV_SLAB, &tm_v, v_full + sv, s * 64,
                                    box_c0 + C::first_col(c), box_r0, hn, hb);
                    if (!lt.acquire(k_empty + sk, pk ^ 1, wctx)) break;
                    lt.arm(k_full + sk, pk, (uint32_t)C::NS * C::NK * C::ROWB);
#pragma unroll
                    for (int s = 0; s < C::NS; ++s)
                        tma_load_5d(sK + sk * C::KV_BYTES + s * C::KV_SLAB, &tm_k, k_full + sk, s * 64,
                                    box_c0 + C::first_col(c), box_r0, hn, hb);
                }
            }
            lt.drain(wctx);
        }
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issue
        reg_dec<kDkvRegsCtl>();
        constexpr uint32_t idesc_s = umma_idesc(TM, C::NKP, IsBf16<DT>::value, IsBf16<DT>::value, false, false);
        constexpr uint32_t idesc_o = umma_idesc(TM, D, IsBf16<DT>::value, IsBf16<DT>::value, false, true);
        constexpr uint32_t hi = smem_desc_hi(C::ATOM, C::SWZ);
        // (the issuing warp is as busy as the pipe: 28 MMAs a chunk at head dim 128)
        const uint32_t q_lo0 = smem_desc_lo(smem_u32(sQ), 16), g_lo0 = smem_desc_lo(smem_u32(sDO), 16);
        const uint32_t k_lo0 = smem_desc_lo(smem_u32(sK), 16), v_lo0 = smem_desc_lo(smem_u32(sV), 16);
        const uint32_t km_lo0 = smem_desc_lo(smem_u32(sK), C::KV_SLAB);
        constexpr uint32_t kKvStep = C::KV_BYTES >> 4, kQStep = C::Q_BYTES >> 4;
        // S = Q K_c^T and dP = dO V_c^T of the next chunk into buffer `buffer`
        Ring rk, rv, rq;
        int c_s = 0;
        uint32_t n_s = 0;
        auto scores = [&]() {
            if (c_s == 0) mbar_wait(q_full + rq.at, rq.phase, wctx, kErrLoadWait);
            mbar_wait(k_full + rk.at, rk.phase, wctx, kErrLoadWait);
            mbar_wait(v_full + rv.at, rv.phase, wctx, kErrLoadWait);
            tc_fence_after();
            const uint32_t q_lo = q_lo0 + rq.at * kQStep, g_lo = g_lo0 + rq.at * kQStep;
            const uint32_t k_lo = k_lo0 + rk.at * kKvStep, v_lo = v_lo0 + rv.at * kKvStep;
            const uint32_t buf = tmem_base + (n_s & 1) * C::TMEM_BUF;
            if (elect_one()) {
                NA2D_TR(2, 0, n_s);
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    constexpr int kPerSlab = C::SLAB_C / 16;
                    const int slab = kk / kPerSlab, in_slab = kk % kPerSlab;
                    umma_ss(buf + C::TMEM_S, desc64(hi, q_lo + ((slab * C::Q_SLAB) >> 4) + 2 * in_slab),
                            desc64(hi, k_lo + ((slab * C::KV_SLAB) >> 4) + 2 * in_slab), idesc_s, kk > 0);
                }
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    constexpr int kPerSlab = C::SLAB_C / 16;
                    const int slab = kk / kPerSlab, in_slab = kk % kPerSlab;
                    umma_ss(buf + C::TMEM_DP, desc64(hi, g_lo + ((slab * C::Q_SLAB) >> 4) + 2 * in_slab),
                            desc64(hi, v_lo + ((slab * C::KV_SLAB) >> 4) + 2 * in_slab), idesc_s, kk > 0);
                }
                umma_commit(s_full + (n_s & 1));
                umma_commit(v_empty + rv.at);
                if (c_s == NCH - 1) umma_commit(q_empty + rq.at);          // last score MMAs of the tile
                NA2D_TR(2, 1, n_s);
            }
            __syncwarp();
            rk.next(NSTK);
            rv.next(NSTV);
            ++n_s;
            if (++c_s == NCH) {
                c_s = 0;
                rq.next(NQ);
            }
        };
        // dQ (+)= dS K_c and B (+)= p K_c of the next chunk, both operands read from its buffer
        Ring ok;
        int c_o = 0;
        uint32_t n_o = 0, tile_phase = 1;
        auto outputs = [&]() {
            if (c_o == 0) {                                                // the tile before has been read out
                mbar_wait(dq_free, tile_phase, wctx, kErrMmaWait);
                tile_phase ^= 1;
            }
            mbar_wait(p_full + (n_o & 1), (n_o >> 1) & 1, wctx, kErrMmaWait);
            tc_fence_after();
            const uint32_t km_lo = km_lo0 + ok.at * kKvStep;
            const uint32_t buf = tmem_base + (n_o & 1) * C::TMEM_BUF;
            const uint32_t acc = c_o > 0;
            if (elect_one()) {
                NA2D_TR(2, 3, n_o);
#pragma unroll
                for (int kk = 0; kk < C::NKP / 16; ++kk)
                    umma_ts(tmem_base + C::TMEM_DQ, buf + C::TMEM_DSH + 8 * kk, desc64(hi, km_lo + ((kk * 16 * C::ROWB) >> 4)),
                            idesc_o, acc | (kk > 0));
                if (SPLIT) {
#pragma unroll
                    for (int kk = 0; kk < C::NKP / 16; ++kk)
                        umma_ts(tmem_base + C::TMEM_DQ, buf + C::TMEM_RES + 8 * kk,
                                desc64(hi, km_lo + ((kk * 16 * C::ROWB) >> 4)), idesc_o, 1u);
                }
#pragma unroll
                for (int kk = 0; kk < C::NKP / 16; ++kk)
                    umma_ts(tmem_base + C::TMEM_BK, buf + C::TMEM_PH + 8 * kk, desc64(hi, km_lo + ((kk * 16 * C::ROWB) >> 4)),
                            idesc_o, acc | (kk > 0));
                umma_commit(k_empty + ok.at);
                if (c_o == NCH - 1) umma_commit(dq_full);
                NA2D_TR(2, 4, n_o);
            }
            __syncwarp();
            ok.next(NSTK);
            ++n_o;
            if (++c_o == NCH) c_o = 0;
        };
        // On the pipe: scores(0) scores(1) | outputs(0) scores(2) | outputs(1) scores(3) | ...  scores(n + 2) go into
        // the buffer whose operands outputs(n) has just read; the pipe runs its MMAs in the order they were issued.
        for (uint32_t n = 0; n < 2 && n < total_units; ++n) scores();
        for (uint32_t n = 0; n < total_units; ++n) {
            outputs();
            if (n + 2 < total_units) scores();
        }
    } else if (warp == 10 || warp == 11) {
        reg_dec<kDkvRegsCtl>();
    } else if (warp >= 12) {
        // ------------------------------------------------------------------ epilogue warps
        // dQ - (delta - estimate) B of a tile, while the softmax warps are at the next one
        reg_dec<kDkvRegsEpi>();
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;                 // query of the tile = tensor-memory lane
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        uint8_t* stage = sOut + quarter * 2 * OutStage<32>::BYTES;
        uint32_t out_seq = 0;
        TileWalk walk((int)blockIdx.x, (int)gridDim.x, tiles_r, tiles_c);
        for (int i = 0; i < n_my; ++i, walk.next()) {
            const int r0 = walk.row(), c0 = walk.col();
            int hn, hb;
            split_unit(walk.bn, g, hn, hb);
            mbar_wait(dq_full, i & 1, wctx, kErrMmaWait);     // also: the softmax warps' corrections are written
            tc_fence_after();
            const float corr = x_corr[(i & 1) * 128 + row];
#pragma unroll
            for (int j = 0; j < D / 32; ++j) {
                uint32_t acc[32];
                tmem_ld_32x32(tmem_lane + C::TMEM_DQ + 32 * j, acc);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t bk[16];
                    tmem_ld_32x16(tmem_lane + C::TMEM_BK + 32 * j + 16 * h, bk);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        acc[16 * h + e] = __float_as_uint(fmaf(-corr, __uint_as_float(bk[e]), __uint_as_float(acc[16 * h + e])));
                }
                if (j + 1 == D / 32) {                        // both accumulators have been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(dq_free);
                }
                stage_and_store<DT, 32, 2>(&tm_dq, stage, acc, g.scale, 32 * j, c0, r0 + quarter * (32 / TW), hn, hb, lane, &out_seq);
            }
        }
        if (lane == 0) bulk_wait<0>();                       // the staging buffers have been read, the rows written
    } else {
        // ------------------------------------------------------------------ softmax warps
        reg_inc<kDkvRegsSoftmax>();
        const int quarter = warp & 3, half = warp >> 2;
        const int row = quarter * 32 + lane;                 // query of the tile = tensor-memory lane
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);

        // What a warp needs to know of a tile before its scores arrive; worked out for the next tile before the last
        // chunk of this one is waited for.
        struct TileState {
            size_t qi;
            bool q_valid;
            int wr, wr_lo, wr_hi;
            uint32_t window;
            float lse, d_est;
        };
        TileWalk walk((int)blockIdx.x, (int)gridDim.x, tiles_r, tiles_c);
        auto prepare = [&]() {                               // of the next tile
            TileState t;
            const int r0 = walk.row(), c0 = walk.col();
            const int box_r0 = na2d_ws(g.q_row0 + r0, g.Hg, KS) - g.kv_row0;
            const int box_c0 = na2d_ws(c0, g.W, KS);
            const int qr_raw = r0 + (row / TW), qc_raw = c0 + (row % TW);
            t.q_valid = qr_raw < g.Hq && qc_raw < g.W;
            const int qr = min(qr_raw, g.Hq - 1), qc = min(qc_raw, g.W - 1);
            t.qi = (static_cast<size_t>(walk.bn) * g.Hq + qr) * g.W + qc;
            t.wr = na2d_ws(g.q_row0 + qr, g.Hg, KS) - g.kv_row0 - box_r0;           // in [0, TH)
            t.window = ((1u << KS) - 1u) << (na2d_ws(qc, g.W, KS) - box_c0);        // this query's columns of the box
            t.wr_lo = __shfl_sync(0xffffffffu, t.wr, 0);
            t.wr_hi = __shfl_sync(0xffffffffu, t.wr, 31);
            t.lse = lse[t.qi];
            // delta holds the estimate here and the exact value afterwards.  It is read before the tile's first partner
            // barrier and written (by the warp of half 0) after its last one, so the read never sees the new
            // value: `delta` must not be declared __restrict__, which would let the read sink past those.
            t.d_est = delta[t.qi];
            walk.next();
            return t;
        };

        uint32_t n = 0;                                      // units so far
        TileState cur;
        if (n_my > 0) cur = prepare();
        for (int i = 0; i < n_my; ++i) {
            const float lse2 = cur.lse * kLog2e, d_est = cur.d_est;
            // the warp's queries see strip rows [wr_lo, wr_hi + ks), the same in every strip: 8-column blocks from b0 on, of which
            // this warp takes every other one; of those, this query's rows
            constexpr int NOWN = C::NOWN;
            const int b0 = min((cur.wr_lo * C::HW) >> 3, C::NB8 - 2 * NOWN);
            const bool extra = (cur.wr_hi + KS) * C::HW > 8 * (b0 + 2 * NOWN + half);
            uint32_t rows[NOWN + 1];
#pragma unroll
            for (int a = 0; a <= NOWN; ++a)
                rows[a] = range_bits<8>(cur.wr * C::HW, (cur.wr + KS) * C::HW, 8 * (b0 + half + 2 * a));
            const uint64_t scale2 = pair2(g.sl2, g.sl2), nlse2 = pair2(-lse2, -lse2), nest2 = pair2(-d_est, -d_est);
            uint64_t delta2 = 0;                             // this half's part of delta
            TileState nxt = cur;

            for (int ch = 0; ch < NCH; ++ch, ++n) {
                const uint32_t tmem_buf = tmem_lane + (n & 1) * C::TMEM_BUF;
                const uint32_t cols = C::seen_cols(cur.window, ch) * C::REP;
                if (ch == NCH - 1 && i + 1 < n_my) nxt = prepare();

                if (tid == 0) NA2D_TR(3, 0, n);
                mbar_wait(s_full + (n & 1), (n >> 1) & 1, wctx, kErrMmaWait);
                tc_fence_after();
                if (tid == 0) NA2D_TR(3, 1, n);
                uint32_t s[NOWN + 1][8], dp[NOWN + 1][8];
                auto load = [&](int a) {
                    tmem_ld_32x8(tmem_buf + C::TMEM_S + 8 * (b0 + half + 2 * a), s[a]);
                    tmem_ld_32x8(tmem_buf + C::TMEM_DP + 8 * (b0 + half + 2 * a), dp[a]);
                };
#pragma unroll
                for (int a = 0; a < NOWN; ++a) load(a);
                if (extra) load(NOWN);                                       // warp-uniform
                tmem_ld_wait();
                // the partner must have read its blocks before 16-bit operands go over them
                bar_sync(1 + quarter, 64);
                if (tid == 0) NA2D_TR(3, 2, n);

                // p = exp(s - lse), dS~ = p (dP - estimate) as packed 16-bit pairs (dS~ head, and residual on the bf16 path);
                // this half's part of delta.  Masked columns may hold anything (padding keys): they are kept out by
                // selection, never by multiplying with zero.
                auto block = [&](int a, uint32_t (&wd)[4], uint32_t (&wr2)[4], uint32_t (&wp)[4]) {
                    const uint32_t seen = rows[a] & cols;
#pragma unroll
                    for (int e2 = 0; e2 < 4; ++e2) {
                        const bool ok0 = (seen >> (2 * e2)) & 1u, ok1 = (seen >> (2 * e2 + 1)) & 1u;
                        const uint64_t x = fma2(pair2(s[a][2 * e2], s[a][2 * e2 + 1]), scale2, nlse2);
                        const float p0 = ok0 ? fast_exp2(lo2(x)) : 0.f, p1 = ok1 ? fast_exp2(hi2(x)) : 0.f;
                        const uint64_t p = pair2(p0, p1), d = pair2(ok0 ? dp[a][2 * e2] : 0u, ok1 ? dp[a][2 * e2 + 1] : 0u);
                        delta2 = fma2(p, d, delta2);
                        const uint64_t ds = mul2(p, add2(d, nest2));
                        wd[e2] = pack2<DT>(lo2(ds), hi2(ds));
                        wr2[e2] = SPLIT ? pack2_residual_bf16(lo2(ds), hi2(ds), wd[e2]) : 0u;
                        wp[e2] = pack2<DT>(p0, p1);
                    }
                };
                auto store = [&](int a, const uint32_t (&wd)[4], const uint32_t (&wr2)[4], const uint32_t (&wp)[4]) {
                    const int blk = b0 + half + 2 * a;
                    tmem_st_32x4(tmem_buf + C::TMEM_DSH + 4 * blk, wd);
                    if (SPLIT) tmem_st_32x4(tmem_buf + C::TMEM_RES + 4 * blk, wr2);
                    tmem_st_32x4(tmem_buf + C::TMEM_PH + 4 * blk, wp);
                };
                {   // blocks outside the range hold zeros (this warp: every other one of them)
                    const uint32_t z[4] = {0u, 0u, 0u, 0u};
                    const int b_end = b0 + half + 2 * (NOWN + (extra ? 1 : 0));
#pragma unroll
                    for (int b = 0; b < C::NB8 / 2; ++b) {
                        const int blk = 2 * b + ((half ^ b0) & 1);          // the blocks of b0's parity are half 0's
                        if (blk < b0 || blk >= b_end) {
                            tmem_st_32x4(tmem_buf + C::TMEM_DSH + 4 * blk, z);
                            if (SPLIT) tmem_st_32x4(tmem_buf + C::TMEM_RES + 4 * blk, z);
                            tmem_st_32x4(tmem_buf + C::TMEM_PH + 4 * blk, z);
                        }
                    }
                }
                // (all blocks first, then their stores: a store waits for its block's conversions)
                uint32_t wd[NOWN][4], wr2[NOWN][4], wp[NOWN][4];
#pragma unroll
                for (int a = 0; a < NOWN; ++a) block(a, wd[a], wr2[a], wp[a]);
#pragma unroll
                for (int a = 0; a < NOWN; ++a) store(a, wd[a], wr2[a], wp[a]);
                if (extra) {
                    block(NOWN, wd[0], wr2[0], wp[0]);
                    store(NOWN, wd[0], wr2[0], wp[0]);
                }
                if (tid == 0) NA2D_TR(3, 3, n);
                if (ch == NCH - 1) {
                    // all chunks seen: add the partner's part
                    const float part = lo2(delta2) + hi2(delta2);
                    if (half == 1) x_sum[(i & 1) * 128 + row] = part;
                    bar_sync(1 + quarter, 64);
                    if (half == 0) {
                        const float dl = part + x_sum[(i & 1) * 128 + row];
                        x_corr[(i & 1) * 128 + row] = dl - d_est;
                        if (cur.q_valid) delta[cur.qi] = dl;
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + (n & 1));
                if (tid == 0) NA2D_TR(3, 4, n);
            }
            cur = nxt;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <typename DT, int D, int KS>
int launch_dq2(const LaunchCtx& lc, const TensorArg& q, const TensorArg& k, const TensorArg& v, const float* lse,
               const TensorArg& d_o, const TensorArg& d_q, float* delta) {
    using C = Dq2Cfg<D, KS>;
    const Na2dGeom& g = lc.g;
    CUtensorMap tq, tg, tk, tv, tdq;
    int rc = make_map(&tq, q, lc.dtype, lc.B, g.N, g.Hq, g.W, D, TW, TH);
    if (rc == NA2D_OK) rc = make_map(&tdq, d_q, lc.dtype, lc.B, g.N, g.Hq, g.W, D, TW, 32 / TW, 32);
    if (rc == NA2D_OK) rc = make_map(&tg, d_o, lc.dtype, lc.B, g.N, g.Hq, g.W, D, TW, TH);
    if (rc == NA2D_OK) rc = make_map(&tk, k, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, C::HW, C::HH);
    if (rc == NA2D_OK) rc = make_map(&tv, v, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, C::HW, C::HH);
    if (rc != NA2D_OK) return rc;
    const int tiles_r = (g.Hq + TH - 1) / TH, tiles_c = (g.W + TW - 1) / TW;
    const long long tiles = (long long)g.BN * tiles_r * tiles_c;
    if (tiles > 0x7fffffffLL / C::NCH) return NA2D_ERR_TOO_LARGE;
    auto kern = dq2_kernel<DT, D, KS>;
    static std::atomic<unsigned long long> opted{0};
    if (opt_in_smem(kern, C::SMEM, lc.device, opted) != cudaSuccess) return NA2D_ERR_CUDA;
    const int grid = persistent_grid(lc, tiles);
    *lc.launched += 1;
    return na2d_launch::launch(lc.overlap, kern, grid, 512, C::SMEM, lc.st,
                               tq, tg, tk, tv, tdq, lse, delta, lc.errors, g, tiles_r, tiles_c, (int)tiles) == cudaSuccess
               ? NA2D_OK
               : NA2D_ERR_CUDA;
}

}  // namespace na2d_tc
