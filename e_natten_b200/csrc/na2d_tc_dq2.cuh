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
// under the next chunk's.  Measured against one chunk in flight, query half with the delta estimate:
// 32 x 2 x 56 x 56 x 32, window 7, bf16 130 -> 100 us; 16 x 8 x 28 x 28 x 64, window 13, bf16 130 -> 95 us;
// 2 x 6 x 97 x 131 x 64, window 9, fp16 138 -> 89 us; 1024 x 1024 x 128, window 13, bf16 1.35 -> 0.97 ms (1.24 with
// two K slots instead of the three or four below).
#pragma once

namespace na2d_tc {

// Keys per chunk at most: 2 x (S + dP) + dQ + B in 512 columns.
constexpr int dq2_nmax(int d) { return (512 - 2 * d) / 4 / 16 * 16; }

template <int D, int KS>
struct Dq2Cfg : Cfg<D, KS, dq2_nmax(D)> {
    using B = Cfg<D, KS, dq2_nmax(D)>;
    static constexpr int NMAX = dq2_nmax(D);
    static constexpr int TMEM_S = 0;                                   // per buffer
    static constexpr int TMEM_DP = NMAX;
    static constexpr int TMEM_BUF = 2 * NMAX;                          // columns of a buffer
    static constexpr int TMEM_DQ = 4 * NMAX;
    static constexpr int TMEM_BK = TMEM_DQ + D;                        // sum_j p k
    static constexpr int TMEM_DSH = TMEM_DP;                           // dS (head) over dP
    static constexpr int TMEM_RES = TMEM_S;                            // dS residual: lower half of S
    static constexpr int TMEM_PH = TMEM_S + B::NKP / 2;                // p: upper half of S
    static constexpr int OUT_BYTES = 8 * OutStage<D / 2>::BYTES;       // output staging of the 8 softmax warps
    static constexpr int FIXED = OUT_BYTES + 2 * 2 * 128 * 4 /*delta exchange*/ + 256 + 1024;
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
    static constexpr int NB16 = (B::NKP + 15) / 16;
    static_assert(B::NCH > 1, "several chunks");
    static_assert(SMEM <= kSmemLimit, "dQ kernel shared memory");
    static_assert(B::NKP <= NMAX && TMEM_BK + D <= 512, "tensor memory layout");
    static_assert((B::NKP / 2) % 8 == 0, "operand halves start on a block boundary");
};

template <typename DT, int D, int KS>
__global__ void __launch_bounds__(384, 1)
dq2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
           const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
           const __grid_constant__ CUtensorMap tm_dq, const float* __restrict__ lse, float* delta, unsigned int* __restrict__ err_word,
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
    uint8_t* sOut = sV + NSTV * C::KV_BYTES;          // 8 x output staging (1024-byte aligned)
    float* x_sum = reinterpret_cast<float*>(sOut + C::OUT_BYTES);     // [tile parity][half][row]
    uint64_t* bars = reinterpret_cast<uint64_t*>(x_sum + 2 * 2 * 128);
    uint64_t* q_full = bars + 0;             // [2] TMA -> MMA (Q and dO tile)
    uint64_t* q_empty = bars + 2;            // [2] MMA (commit) -> TMA
    uint64_t* k_full = bars + 4;             // [4]
    uint64_t* k_empty = bars + 8;            // [4]
    uint64_t* v_full = bars + 12;            // [4]
    uint64_t* v_empty = bars + 16;           // [4]
    uint64_t* s_full = bars + 20;            // [2] MMA (commit) -> softmax: S and dP are complete, per buffer
    uint64_t* p_full = bars + 22;            // [2] softmax -> MMA: dS and p are in tensor memory, per buffer
    uint64_t* dq_full = bars + 24;           // MMA (commit) -> softmax (epilogue)
    uint64_t* dq_free = bars + 25;           // softmax -> MMA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
    const WaitCtx wctx{reinterpret_cast<WaitState*>(bars + 27)};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_my = total_tiles > (int)blockIdx.x ? (total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const uint32_t total_units = (uint32_t)n_my * NCH;

    if (tid == 0) {
        wait_state_init(wctx.st, err_word, kWaitLimitNs);
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
        mbar_init(dq_free, 8);
        mbar_fence_init();
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_do);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        tma_prefetch_desc(&tm_dq);
    }
    if (warp == 0) {
        __syncwarp();
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    // K rows [NK, NKP) of every stage are contraction rows of dQ = dS K that TMA never writes: zero them once.
    if constexpr (C::NKP > C::NK) {
        constexpr int pad16 = (C::NKP - C::NK) * C::ROWB / 16;
        for (int i = tid; i < NSTK * C::NS * pad16; i += 384) {
            const int which = i / pad16, off = i - which * pad16;             // which = stage * NS + slab
            st_shared_v4(smem_u32(sK + (which / C::NS) * C::KV_BYTES + (which % C::NS) * C::KV_SLAB + C::NK * C::ROWB +
                                  off * 16), 0u, 0u, 0u, 0u);
        }
        fence_proxy_async();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // my i-th tile: unit bn (head bn % N of batch bn / N, split where a TMA coordinate needs it),
    // first row r0, first column c0
    auto decode = [&](int i, int& bn, int& r0, int& c0) {
        int t = (int)blockIdx.x + i * (int)gridDim.x;
        const int tc = t % tiles_c;
        t /= tiles_c;
        r0 = (t % tiles_r) * TH;
        c0 = tc * TW;
        bn = t / tiles_r;
    };
    if (warp == 8) {
        // ------------------------------------------------------------------ producer
        reg_dec<kRegsDonor>();
        if (lane == 0) {
            uint32_t n = 0;
            LoadTracker lt(bars);
            for (int i = 0; i < n_my && lt.ok; ++i) {
                int bn, r0, c0, hn, hb;
                decode(i, bn, r0, c0);
                split_unit(bn, g, hn, hb);
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
                for (int c = 0; c < NCH; ++c, ++n) {
                    const uint32_t sk = n % NSTK, pk = (n / NSTK) & 1, sv = n % NSTV, pv = (n / NSTV) & 1;
                    if (!lt.acquire(v_empty + sv, pv ^ 1, wctx)) break;
                    lt.arm(v_full + sv, pv, (uint32_t)C::NS * C::NK * C::ROWB);
#pragma unroll
                    for (int s = 0; s < C::NS; ++s)
                        tma_load_5d(sV + sv * C::KV_BYTES + s * C::KV_SLAB, &tm_v, v_full + sv, s * 64, box_c0,
                                    box_r0 + c * C::RC, hn, hb);
                    if (!lt.acquire(k_empty + sk, pk ^ 1, wctx)) break;
                    lt.arm(k_full + sk, pk, (uint32_t)C::NS * C::NK * C::ROWB);
#pragma unroll
                    for (int s = 0; s < C::NS; ++s)
                        tma_load_5d(sK + sk * C::KV_BYTES + s * C::KV_SLAB, &tm_k, k_full + sk, s * 64, box_c0,
                                    box_r0 + c * C::RC, hn, hb);
                }
            }
            lt.drain(wctx);
        }
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issue
        reg_dec<kRegsDonor>();
        constexpr uint32_t idesc_s = umma_idesc(TM, C::NKP, IsBf16<DT>::value, IsBf16<DT>::value, false, false);
        constexpr uint32_t idesc_o = umma_idesc(TM, D, IsBf16<DT>::value, IsBf16<DT>::value, false, true);
        constexpr uint32_t hi = smem_desc_hi(C::ATOM, C::SWZ);
        // S(n) = Q K_c^T and dP(n) = dO V_c^T into buffer n & 1
        auto scores = [&](uint32_t n) {
            const uint32_t i = n / NCH, c = n % NCH, sk = n % NSTK, sv = n % NSTV, qb = i % NQ;
            if (lane == 0) NA2D_TR(2, 0, n);
            if (c == 0) mbar_wait(q_full + qb, (i / NQ) & 1, wctx, kErrLoadWait);
            mbar_wait(k_full + sk, (n / NSTK) & 1, wctx, kErrLoadWait);
            mbar_wait(v_full + sv, (n / NSTV) & 1, wctx, kErrLoadWait);
            tc_fence_after();
            const uint32_t q_lo = smem_desc_lo(smem_u32(sQ + qb * C::Q_BYTES), 16);
            const uint32_t g_lo = smem_desc_lo(smem_u32(sDO + qb * C::Q_BYTES), 16);
            const uint32_t k_lo = smem_desc_lo(smem_u32(sK + sk * C::KV_BYTES), 16);
            const uint32_t v_lo = smem_desc_lo(smem_u32(sV + sv * C::KV_BYTES), 16);
            const uint32_t buf = tmem_base + (n & 1) * C::TMEM_BUF;
            if (elect_one()) {
                NA2D_TR(2, 1, n);
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
                umma_commit(s_full + (n & 1));
                umma_commit(v_empty + sv);
                if (c == NCH - 1) umma_commit(q_empty + qb);               // last score MMAs of the tile
                NA2D_TR(2, 2, n);
            }
            __syncwarp();
        };
        // dQ (+)= dS(n) K_c and B (+)= p(n) K_c, both operands read from buffer n & 1
        auto outputs = [&](uint32_t n) {
            const uint32_t i = n / NCH, c = n % NCH, sk = n % NSTK;
            mbar_wait(p_full + (n & 1), (n >> 1) & 1, wctx, kErrMmaWait);
            if (c == 0) mbar_wait(dq_free, (i & 1) ^ 1, wctx, kErrMmaWait);        // the tile before has been read out
            tc_fence_after();
            const uint32_t km_lo = smem_desc_lo(smem_u32(sK + sk * C::KV_BYTES), C::KV_SLAB);
            const uint32_t buf = tmem_base + (n & 1) * C::TMEM_BUF;
            if (elect_one()) {
                NA2D_TR(2, 3, n);
                const uint32_t acc = c > 0;
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
                umma_commit(k_empty + sk);
                if (c == NCH - 1) umma_commit(dq_full);
                NA2D_TR(2, 4, n);
            }
            __syncwarp();
        };
        // On the pipe: scores(0) scores(1) | outputs(0) scores(2) | outputs(1) scores(3) | ...  scores(n + 2) go into
        // the buffer whose operands outputs(n) has just read; the pipe runs its MMAs in the order they were issued.
        if (total_units > 0) scores(0);
        if (total_units > 1) scores(1);
        for (uint32_t n = 0; n < total_units; ++n) {
            outputs(n);
            if (n + 2 < total_units) scores(n + 2);
        }
    } else if (warp >= 10) {
        reg_dec<kRegsDonor>();
    } else {
        // ------------------------------------------------------------------ softmax warps
        reg_inc<kRegsSoftmax>();
        const int quarter = warp & 3, half = warp >> 2;
        const int row = quarter * 32 + lane;                 // query of the tile = tensor-memory lane
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        constexpr int DH = D / 2;                            // output columns stored by this half
        constexpr int NBH = (C::NB16 + 1) / 2;               // own blocks at most
        constexpr int kRows = (32 / TW - 1 + KS) < C::RC ? (32 / TW - 1 + KS) : C::RC;
        constexpr int kBlocks = (kRows * C::HW - 1) / 16 + 2;
        constexpr int NACT = (kBlocks + 1) / 2 < NBH ? (kBlocks + 1) / 2 : NBH;

        uint32_t n = 0, n_x = 0;                             // units, delta exchanges so far
        for (int i = 0; i < n_my; ++i) {
            int bn, r0, c0;
            decode(i, bn, r0, c0);
            const int box_r0 = na2d_ws(g.q_row0 + r0, g.Hg, KS) - g.kv_row0;
            const int box_c0 = na2d_ws(c0, g.W, KS);
            const int qr_raw = r0 + (row / TW), qc_raw = c0 + (row % TW);
            const bool q_valid = qr_raw < g.Hq && qc_raw < g.W;
            const int qr = min(qr_raw, g.Hq - 1), qc = min(qc_raw, g.W - 1);
            const size_t qi = (static_cast<size_t>(bn) * g.Hq + qr) * g.W + qc;
            const int wr = na2d_ws(g.q_row0 + qr, g.Hg, KS) - g.kv_row0 - box_r0;   // in [0, TH)
            const int wc = na2d_ws(qc, g.W, KS) - box_c0;                            // in [0, TW)
            const int wr_lo = __shfl_sync(0xffffffffu, wr, 0);
            const int wr_hi = __shfl_sync(0xffffffffu, wr, 31);
            const float lse2 = lse[qi] * kLog2e;
            float dl_part = 0.f;                             // this half's part of delta
            float dl = 0.f;                                  // delta, once every chunk has been seen
            // delta holds the estimate here and the exact value afterwards.  It is read before this tile's first
            // partner barrier and written (by the partner warp of half 0) after its last one, so the read never sees
            // the new value: `delta` must not be declared __restrict__, which would let the read sink past those.
            const float d_est = delta[qi];

            for (int ch = 0; ch < NCH; ++ch, ++n) {
                const uint32_t tmem_buf = tmem_lane + (n & 1) * C::TMEM_BUF;
                const int row_off = ch * C::RC;
                const int j_lo = max(wr_lo - row_off, 0) * C::HW;
                const int j_hi = min(min(wr_hi + KS - row_off, C::RC) * C::HW, C::NK);       // exclusive
                const int b_hi = (max(j_hi, 0) + 15) >> 4;
                const int bi_lo = ((j_lo >> 4) - half + 1) >> 1;

                if (tid == 0) NA2D_TR(3, 0, n);
                mbar_wait(s_full + (n & 1), (n >> 1) & 1, wctx, kErrMmaWait);
                tc_fence_after();
                if (tid == 0) NA2D_TR(3, 1, n);
                uint32_t s[NACT][16], dp[NACT][16];
                uint32_t vmask[NACT];
#pragma unroll
                for (int a = 0; a < NACT; ++a) {
                    const int blk = half + 2 * (bi_lo + a);
                    if (blk < b_hi) {                                        // warp-uniform
                        tmem_ld_32x16(tmem_buf + C::TMEM_S + 16 * blk, s[a]);
                        tmem_ld_32x16(tmem_buf + C::TMEM_DP + 16 * blk, dp[a]);
                    }
                }
#pragma unroll
                for (int a = 0; a < NACT; ++a) {                             // validity masks, loads in flight
                    const int blk = half + 2 * (bi_lo + a);
                    vmask[a] = (blk < b_hi) ? block_mask16<C::HW, KS, C::RC>(blk, wr - row_off, wc) : 0u;
                }
                tmem_ld_wait();
                if (tid == 0) NA2D_TR(3, 2, n);

                // p = exp(s - lse) in place of s; this half's part of delta
                float d0 = 0.f, d1 = 0.f;
#pragma unroll
                for (int a = 0; a < NACT; ++a) {
                    if (half + 2 * (bi_lo + a) < b_hi) {
#pragma unroll
                        for (int e = 0; e < 16; e += 2) {
                            const float p0 = ((vmask[a] >> e) & 1u)
                                                 ? fast_exp2(fmaf(__uint_as_float(s[a][e]), g.sl2, -lse2)) : 0.f;
                            const float p1 = ((vmask[a] >> (e + 1)) & 1u)
                                                 ? fast_exp2(fmaf(__uint_as_float(s[a][e + 1]), g.sl2, -lse2)) : 0.f;
                            s[a][e] = __float_as_uint(p0);
                            s[a][e + 1] = __float_as_uint(p1);
                            // masked columns may hold anything (padding keys): keep them out by
                            // selection, never by multiplying with zero
                            if (!((vmask[a] >> e) & 1u)) dp[a][e] = 0u;
                            if (!((vmask[a] >> (e + 1)) & 1u)) dp[a][e + 1] = 0u;
                            d0 = fmaf(p0, __uint_as_float(dp[a][e]), d0);
                            d1 = fmaf(p1, __uint_as_float(dp[a][e + 1]), d1);
                        }
                    }
                }
                dl_part += d0 + d1;

                if (ch == NCH - 1) {
                    // all chunks seen: add the partner's part; both now hold delta
                    x_sum[((n_x & 1) * 2 + half) * 128 + row] = dl_part;
                    bar_sync(1 + quarter, 64);
                    dl = dl_part + x_sum[((n_x & 1) * 2 + (half ^ 1)) * 128 + row];
                    ++n_x;
                    if (q_valid && half == 0) delta[qi] = dl;
                } else {
                    // the partner must have read its blocks before 16-bit operands go over them
                    bar_sync(1 + quarter, 64);
                }

                if (tid == 0) NA2D_TR(3, 3, n);
                // dS~ = p (dP - estimate) as packed 16-bit pairs (head, and residual on the bf16 path), and p
#pragma unroll
                for (int a = 0; a < NACT; ++a) {
                    const int blk = half + 2 * (bi_lo + a);
                    if (blk < b_hi) {
                        uint32_t wd[8], wr2[8];
#pragma unroll
                        for (int e2 = 0; e2 < 8; ++e2) {
                            const float ds0 = ((vmask[a] >> (2 * e2)) & 1u)
                                ? __uint_as_float(s[a][2 * e2]) * (__uint_as_float(dp[a][2 * e2]) - d_est) : 0.f;
                            const float ds1 = ((vmask[a] >> (2 * e2 + 1)) & 1u)
                                ? __uint_as_float(s[a][2 * e2 + 1]) * (__uint_as_float(dp[a][2 * e2 + 1]) - d_est) : 0.f;
                            wd[e2] = pack2<DT>(ds0, ds1);
                            wr2[e2] = SPLIT ? pack2_residual_bf16(ds0, ds1, wd[e2]) : 0u;
                        }
                        tmem_st_32x8(tmem_buf + C::TMEM_DSH + 8 * blk, wd);
                        if (SPLIT) tmem_st_32x8(tmem_buf + C::TMEM_RES + 8 * blk, wr2);
#pragma unroll
                        for (int e2 = 0; e2 < 8; ++e2)           // p of masked columns is an exact zero
                            wd[e2] = pack2<DT>(__uint_as_float(s[a][2 * e2]), __uint_as_float(s[a][2 * e2 + 1]));
                        tmem_st_32x8(tmem_buf + C::TMEM_PH + 8 * blk, wd);
                    }
                }
                {   // own blocks outside the range hold zeros
                    const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
                    for (int bi = 0; bi < NBH; ++bi) {
                        const int blk = half + 2 * bi;
                        const bool in_range = bi >= bi_lo && bi < bi_lo + NACT && blk < b_hi;
                        if (!in_range && 16 * blk < C::NKP) {
                            tmem_st_32x8(tmem_buf + C::TMEM_DSH + 8 * blk, z);
                            if (SPLIT) tmem_st_32x8(tmem_buf + C::TMEM_RES + 8 * blk, z);
                            tmem_st_32x8(tmem_buf + C::TMEM_PH + 8 * blk, z);
                        }
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + (n & 1));
                if (tid == 0) NA2D_TR(3, 4, n);
            }

            // ---- epilogue: this half's columns of the thread's dQ row
            mbar_wait(dq_full, i & 1, wctx, kErrMmaWait);
            tc_fence_after();
            if (tid == 0) NA2D_TR(3, 5, n - 1);
            uint32_t acc[DH];
#pragma unroll
            for (int piece = 0; piece < DH / 16; ++piece)
                tmem_ld_32x16(tmem_lane + C::TMEM_DQ + half * DH + 16 * piece,
                              *reinterpret_cast<uint32_t(*)[16]>(&acc[16 * piece]));
            // dQ - (delta - estimate) B, piece by piece
            const float corr = dl - d_est;
#pragma unroll
            for (int piece = 0; piece < DH / 16; ++piece) {
                uint32_t bk[16];
                tmem_ld_32x16(tmem_lane + C::TMEM_BK + half * DH + 16 * piece, bk);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    acc[16 * piece + e] = __float_as_uint(fmaf(-corr, __uint_as_float(bk[e]), __uint_as_float(acc[16 * piece + e])));
            }
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(dq_free);
            if (tid == 0) NA2D_TR(3, 6, n - 1);
            int hn, hb;
            split_unit(bn, g, hn, hb);
            stage_and_store<DT, DH>(&tm_dq, sOut + warp * OutStage<DH>::BYTES, acc, g.scale, half * DH, c0,
                                    r0 + quarter * (32 / TW), hn, hb, lane);
            if (tid == 0) NA2D_TR(3, 7, n - 1);
        }
    }

    if (warp < 8 && lane == 0) bulk_wait<0>();          // the staging buffers have been read, the rows written
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
    if (rc == NA2D_OK) rc = make_map(&tdq, d_q, lc.dtype, lc.B, g.N, g.Hq, g.W, D, TW, 32 / TW, OutStage<D / 2>::RW);
    if (rc == NA2D_OK) rc = make_map(&tg, d_o, lc.dtype, lc.B, g.N, g.Hq, g.W, D, TW, TH);
    if (rc == NA2D_OK) rc = make_map(&tk, k, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, C::HW, C::RC);
    if (rc == NA2D_OK) rc = make_map(&tv, v, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, C::HW, C::RC);
    if (rc != NA2D_OK) return rc;
    const int tiles_r = (g.Hq + TH - 1) / TH, tiles_c = (g.W + TW - 1) / TW;
    const long long tiles = (long long)g.BN * tiles_r * tiles_c;
    if (tiles > 0x7fffffffLL / C::NCH) return NA2D_ERR_TOO_LARGE;
    auto kern = dq2_kernel<DT, D, KS>;
    static std::atomic<unsigned long long> opted{0};
    if (opt_in_smem(kern, C::SMEM, lc.device, opted) != cudaSuccess) return NA2D_ERR_CUDA;
    const int grid = persistent_grid(lc, tiles);
    kern<<<grid, 384, C::SMEM, lc.st>>>(tq, tg, tk, tv, tdq, lse, delta, lc.err_word, g, tiles_r, tiles_c,
                                        (int)tiles);
    *lc.launched += 1;
    return cudaGetLastError() == cudaSuccess ? NA2D_OK : NA2D_ERR_CUDA;
}

}  // namespace na2d_tc
