// Persistent, warp-specialised tcgen05 forward kernel for the larger windows (kernel sizes >= 7), two query tiles in
// flight, for calls of more tiles than SMs (at head dim 128 from window 11 on; na2d_tc_fwd.cuh).  Included by na2d_tc_fwd.cu.
//
// A CTA's tiles alternate between two softmax groups of four warps (warps 0-3 the even ones, 4-7 the odd ones).  Each
// group has an S / P buffer and an output accumulator of its own in tensor memory, and the tensor pipe takes turns:
//     S_a(0) S_b(0) | PV_a(0) S_a(1) | PV_b(0) S_b(1) | PV_a(1) S_a(2) | ...
// so that one group's MMAs run while the other group's warps work on its scores.  With all eight warps on one chunk
// (na2d_tc_fwd.cuh) what bounds a tile is the chain load scores -> maximum -> exchange with the partner warp -> exp -> store, in
// which the two warps of a scheduler wait at the same places.  Here they are in different phases, and as a thread has
// a whole row of S, no maximum or sum is exchanged.  Chunks are column strips (na2d_tc_strip.cuh).
//
//   warps 0-7   softmax: a thread owns a query (tensor-memory lane), reads the blocks of its row that its warp can see
//               once, writes P over S as packed 16-bit pairs; O accumulates in tensor memory over the tile's chunks and is
//               rescaled where a row's maximum grows;
//   warps 8, 10 producers: TMA loads of the two Q tiles and of K chunks, and of V chunks (a ring each);
//   warp 9      MMA issue;
//   warps 12-15 epilogue: normalise and store O of either group while its next tile is under way;
//   warp 11     idle (register donor).
//
// What bounds it: exponentials (8 cycles a warp instruction; a warp's rows see 1.3 to 2.5 times the window) and the chain wait,
// load, maximum, exp, store of a group, of which two are in flight; at head dim 128 the MMAs are as long.  Measured against
// na2d_tc_fwd.cuh on one B200: 32 x 2 x 56 x 56 x 32, window 7, bf16 51 -> 39 us; 16 x 8 x 28 x 28 x 64, window 13, bf16 53 -> 39 us;
// 2 x 6 x 97 x 131 x 64, window 9, fp16 45 -> 37 us; 8 heads of 1024 x 1024 x 128, window 13, bf16 3.34 -> 2.69 ms.
#pragma once

namespace na2d_tc {

constexpr int fwd2_strip(int d, int ks) { return d <= 64 && ks <= 9 ? 8 : 4; }

template <int D, int KS>
struct Fwd2Cfg : StripCfg<D, KS, fwd2_strip(D, KS)> {
    using B = StripCfg<D, KS, fwd2_strip(D, KS)>;
    // The K chunk keeps only the rows TMA writes (rounded to the swizzle period): what the MMA reads past the end feeds S
    // columns that are masked.  The V chunk keeps all NKP rows, the padding ones zeroed: they are contraction rows.
    static constexpr int K_ROWS = B::ROWB == 128 ? (B::NK + 7) / 8 * 8 : B::NKP;
    static constexpr int K_SLAB = K_ROWS * B::ROWB;
    static constexpr int K_BYTES = B::NS * K_SLAB;
    static constexpr int V_BYTES = B::KV_BYTES;
    static constexpr int OUT_BYTES = 4 * (D / 32) * OutStage<32>::BYTES; // a tile's output rows, staged by the 4 epilogue warps
    static constexpr int XCHG_BYTES = 2 * 2 * 128 * 4;                   // row sum, final maximum [group][row]
    static constexpr int FIXED = 2 * B::Q_BYTES + OUT_BYTES + XCHG_BYTES + 256 /*barriers*/ + 1024 /*alignment*/;
    static constexpr bool fits(int nk, int nv) { return FIXED + nk * K_BYTES + nv * V_BYTES <= kSmemLimit; }
    static constexpr int NSTV = fits(4, 4) ? 4 : (fits(3, 3) ? 3 : 2);
    static constexpr int NSTK = NSTV < 4 && fits(NSTV + 1, NSTV) ? NSTV + 1 : NSTV;
    static constexpr int SMEM = FIXED + NSTK * K_BYTES + NSTV * V_BYTES;
    static constexpr int NB16 = B::NKP / 16;                             // 16-column blocks of S
    // Blocks that a warp's ks + 3 rows fill where they start on a block boundary (away from the borders they do), which are
    // read in any case, and one more where they do not.
    static constexpr int NACT = ((KS + 3) * B::HW + 15) / 16;
    static constexpr int ROWS16 = 16 / B::HW;                            // strip rows of a block
    static constexpr int TMEM_S = 0, TMEM_SSTRIDE = D <= 64 ? 192 : 128; // S / P of group g
    static constexpr int TMEM_O = 2 * TMEM_SSTRIDE, TMEM_OSTRIDE = D;    // O of group g
    static_assert(SMEM <= kSmemLimit, "forward kernel shared memory");
    static_assert(B::NKP <= TMEM_SSTRIDE && TMEM_O + 2 * D <= 512, "tensor memory layout");
};

template <typename DT, int D, int KS>
__global__ void __launch_bounds__(512, 1)
fwd2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
            const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
            float* __restrict__ lse, const ErrorState* __restrict__ errors,
            const Na2dGeom g, const int tiles_r, const int tiles_c, const int total_tiles) {
    using C = Fwd2Cfg<D, KS>;
    constexpr int NSTK = C::NSTK, NSTV = C::NSTV;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;                                   // Q tile of each group
    uint8_t* sV = sQ + 2 * C::Q_BYTES;                    // NSTV x V chunk
    uint8_t* sK = sV + NSTV * C::V_BYTES;                 // NSTK x K chunk
    uint8_t* sOut = sK + NSTK * C::K_BYTES;               // output staging (1024-byte aligned)
    float* x_sum = reinterpret_cast<float*>(sOut + C::OUT_BYTES);     // [group][row]
    float* x_fin = x_sum + 2 * 128;                                   // [group][row]  final maximum * log2(e)
    uint64_t* bars = reinterpret_cast<uint64_t*>(x_fin + 2 * 128);
    uint64_t* q_full = bars;                 // [2] TMA -> MMA, per group
    uint64_t* q_empty = bars + 2;            // [2] MMA (commit) -> TMA
    uint64_t* o_full = bars + 4;             // [2] MMA (commit) -> epilogue
    uint64_t* o_free = bars + 6;             // [2] epilogue -> MMA
    uint64_t* s_full = bars + 8;             // [2] MMA (commit) -> softmax
    uint64_t* p_full = bars + 10;            // [2] softmax -> MMA
    uint64_t* k_full = bars + 12;            // [4] TMA -> MMA
    uint64_t* k_empty = bars + 16;           // [4] MMA (commit) -> TMA
    uint64_t* v_full = bars + 20;            // [4] TMA -> MMA
    uint64_t* v_empty = bars + 24;           // [4] MMA (commit) -> TMA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
    const WaitCtx wctx{reinterpret_cast<WaitState*>(bars + 29)};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_my = total_tiles > (int)blockIdx.x ? (total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;

    if (tid == 0) {
        wait_state_init(wctx.st, errors, kWaitLimitNs);
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full + i, 1);
            mbar_init(q_empty + i, 1);
            mbar_init(o_full + i, 1);
            mbar_init(o_free + i, 4);
            mbar_init(s_full + i, 1);
            mbar_init(p_full + i, 4);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(k_full + i, 1);
            mbar_init(k_empty + i, 1);
            mbar_init(v_full + i, 1);
            mbar_init(v_empty + i, 1);
        }
        mbar_fence_init();
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        tma_prefetch_desc(&tm_o);
    }
    // V rows [NK, NKP) of every stage are contraction rows of P V that TMA never writes.
    if constexpr (C::NKP > C::NK) {
        constexpr int pad16 = (C::NKP - C::NK) * C::ROWB / 16;
        for (int i = tid; i < NSTV * C::NS * pad16; i += 512) {
            const int which = i / pad16, off = i - which * pad16;
            st_shared_v4(smem_u32(sV + (which / C::NS) * C::V_BYTES + (which % C::NS) * C::KV_SLAB + C::NK * C::ROWB + off * 16),
                         0u, 0u, 0u, 0u);
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

    if (warp == 8 || warp == 10) {
        // ------------------------------------------------------------------ producers
        // Warp 8 fetches the Q tiles and the K chunks, whose buffers the score MMAs release early; warp 10 the V
        // chunks, whose buffers are released by P V.  One producer for both would hold K back behind the wait for a V buffer
        // (8 heads of 1024 x 1024 x 128, window 13: 3.8 instead of 2.6 ms).
        reg_dec<kDkvRegsCtl>();
        if (lane == 0) {
            LoadTracker lt(bars);
            uint32_t at = 0, phase = 0;
            TileWalk walk((int)blockIdx.x, (int)gridDim.x, tiles_r, tiles_c), ahead = walk;     // ahead: two tiles on
            ahead.next();
            ahead.next();
            for (int pair = 0; 2 * pair < n_my && lt.ok; ++pair) {
                int hn[2], hb[2], box_r0[2], box_c0[2];
                const int members = min(2, n_my - 2 * pair);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    if (x >= members) break;
                    const int r0 = walk.row(), c0 = walk.col();
                    split_unit(walk.bn, g, hn[x], hb[x]);
                    walk.next();
                    box_r0[x] = na2d_ws(g.q_row0 + r0, g.Hg, KS) - g.kv_row0;
                    box_c0[x] = na2d_ws(c0, g.W, KS);
                    if (warp == 8) {
                        if (!lt.acquire(q_empty + x, (pair & 1) ^ 1, wctx)) break;
                        lt.arm(q_full + x, pair & 1, C::Q_BYTES);
#pragma unroll
                        for (int s = 0; s < C::NS; ++s)
                            tma_load_5d(sQ + x * C::Q_BYTES + s * C::Q_SLAB, &tm_q, q_full + x, s * 64, c0, r0, hn[x], hb[x]);
                        if (2 * (pair + 1) + x < n_my) {       // the group's next Q tile: into L2, until its buffer is free
                            int hn1, hb1;
                            split_unit(ahead.bn, g, hn1, hb1);
#pragma unroll
                            for (int s = 0; s < C::NS; ++s) tma_prefetch_5d(&tm_q, s * 64, ahead.col(), ahead.row(), hn1, hb1);
                            ahead.next();
                        }
                    }
                }
                for (int c = 0; c < C::NCH && lt.ok; ++c) {
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        if (x >= members) break;
                        // (the tensor map is named in each call: a map chosen through a run-time pointer may be
                        // copied to local memory, where TMA cannot read it)
                        if (warp == 8) {
                            if (!lt.acquire(k_empty + at, phase ^ 1, wctx)) break;
                            lt.arm(k_full + at, phase, (uint32_t)C::NS * C::NK * C::ROWB);
#pragma unroll
                            for (int s = 0; s < C::NS; ++s)
                                tma_load_5d(sK + at * C::K_BYTES + s * C::K_SLAB, &tm_k, k_full + at, s * 64,
                                            box_c0[x] + C::first_col(c), box_r0[x], hn[x], hb[x]);
                        } else {
                            if (!lt.acquire(v_empty + at, phase ^ 1, wctx)) break;
                            lt.arm(v_full + at, phase, (uint32_t)C::NS * C::NK * C::ROWB);
#pragma unroll
                            for (int s = 0; s < C::NS; ++s)
                                tma_load_5d(sV + at * C::V_BYTES + s * C::KV_SLAB, &tm_v, v_full + at, s * 64,
                                            box_c0[x] + C::first_col(c), box_r0[x], hn[x], hb[x]);
                        }
                        if (++at == (uint32_t)(warp == 8 ? NSTK : NSTV)) {
                            at = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
            lt.drain(wctx);
        }
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issue
        // (the whole warp walks the loop so that addresses stay warp-uniform; one lane issues)
        reg_dec<kDkvRegsCtl>();
        constexpr uint32_t idesc_s = umma_idesc(TM, C::NKP, IsBf16<DT>::value, IsBf16<DT>::value, false, false);
        constexpr uint32_t idesc_o = umma_idesc(TM, D, IsBf16<DT>::value, IsBf16<DT>::value, false, true);
        constexpr uint32_t hi = smem_desc_hi(C::ATOM, C::SWZ);
        // the chunks in their order: group x, chunk c and pair of tiles
        struct Place {
            int x = 0, c = 0, pair = 0;
            __device__ __forceinline__ void next() {
                x ^= 1;
                if (x == 0 && ++c == C::NCH) { c = 0; ++pair; }
            }
        };
        const uint32_t q_lo0 = smem_desc_lo(smem_u32(sQ), 16), k_lo0 = smem_desc_lo(smem_u32(sK), 16);
        const uint32_t v_lo0 = smem_desc_lo(smem_u32(sV), C::KV_SLAB);
        // S = Q K_c^T of the next chunk into its group's buffer
        Ring rk;
        Place ps;
        auto scores = [&]() {
            if (2 * ps.pair + ps.x < n_my) {                  // an odd number of tiles: the last one has no partner
                if (ps.c == 0) mbar_wait(q_full + ps.x, ps.pair & 1, wctx, kErrLoadWait);
                mbar_wait(k_full + rk.at, rk.phase, wctx, kErrLoadWait);
                tc_fence_after();
                const uint32_t q_lo = q_lo0 + ps.x * (C::Q_BYTES >> 4), k_lo = k_lo0 + rk.at * (C::K_BYTES >> 4);
                const uint32_t t_s = tmem_base + C::TMEM_S + ps.x * C::TMEM_SSTRIDE;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        constexpr int kPerSlab = C::SLAB_C / 16;
                        const int slab = kk / kPerSlab, in_slab = kk % kPerSlab;
                        umma_ss(t_s, desc64(hi, q_lo + ((slab * C::Q_SLAB) >> 4) + 2 * in_slab),
                                desc64(hi, k_lo + ((slab * C::K_SLAB) >> 4) + 2 * in_slab), idesc_s, kk > 0);
                    }
                    umma_commit(s_full + ps.x);                               // and P V of the group's chunk before
                    umma_commit(k_empty + rk.at);
                    if (ps.c == C::NCH - 1) umma_commit(q_empty + ps.x);      // the tile's Q buffer is free
                }
                __syncwarp();
                rk.next(NSTK);
            }
            ps.next();
        };
        // O (+)= P V_c of the next chunk
        Ring rv;
        Place po;
        auto outputs = [&]() {
            if (2 * po.pair + po.x < n_my) {
                if (po.c == 0) mbar_wait(o_free + po.x, (po.pair & 1) ^ 1, wctx, kErrMmaWait);     // the tile before has been read out
                mbar_wait(v_full + rv.at, rv.phase, wctx, kErrLoadWait);
                mbar_wait(p_full + po.x, (po.pair * C::NCH + po.c) & 1, wctx, kErrMmaWait);
                tc_fence_after();
                const uint32_t v_lo = v_lo0 + rv.at * (C::V_BYTES >> 4);
                const uint32_t t_p = tmem_base + C::TMEM_S + po.x * C::TMEM_SSTRIDE;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < C::NKP / 16; ++kk)
                        umma_ts(tmem_base + C::TMEM_O + po.x * C::TMEM_OSTRIDE, t_p + 8 * kk,
                                desc64(hi, v_lo + ((kk * 16 * C::ROWB) >> 4)), idesc_o, (po.c > 0) || (kk > 0));
                    umma_commit(v_empty + rv.at);
                    if (po.c == C::NCH - 1) umma_commit(o_full + po.x);
                }
                __syncwarp();
                rv.next(NSTV);
            }
            po.next();
        };
        // The group's next scores go into the buffer P V has just read; the pipe runs its MMAs in the order they
        // were issued.
        const uint32_t slots = (uint32_t)((n_my + 1) / 2) * 2u * C::NCH;
        for (uint32_t s = 0; s < 2 && s < slots; ++s) scores();
        for (uint32_t s = 0; s < slots; ++s) {
            outputs();
            if (s + 2 < slots) scores();
        }
    } else if (warp == 11) {
        reg_dec<kDkvRegsCtl>();
    } else if (warp >= 12) {
        // ------------------------------------------------------------------ epilogue warps
        reg_dec<kDkvRegsEpi>();
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;                 // query of the tile = tensor-memory lane
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        uint8_t* stage = sOut + quarter * (D / 32) * OutStage<32>::BYTES;
        TileWalk walk((int)blockIdx.x, (int)gridDim.x, tiles_r, tiles_c);
        for (int i = 0; i < n_my; ++i, walk.next()) {
            int hn, hb;
            const int bn = walk.bn, r0 = walk.row(), c0 = walk.col();
            split_unit(bn, g, hn, hb);
            const int x = i & 1;
            const int qr = r0 + (row / TW), qc = c0 + (row % TW);
            mbar_wait(o_full + x, (i >> 1) & 1, wctx, kErrMmaWait);          // also: the group's sums are written
            tc_fence_after();
            const float total = x_sum[x * 128 + row], fin = x_fin[x * 128 + row];
            const float inv = 1.f / total;
            if (lane == 0) bulk_wait_read<0>();                               // the stores of the tile before have read the staging
            __syncwarp();
#pragma unroll
            for (int j = 0; j < D / 32; ++j) {
                uint32_t v[32];
                tmem_ld_32x32(tmem_lane + C::TMEM_O + x * C::TMEM_OSTRIDE + 32 * j, v);
                tmem_ld_wait();
                if (j + 1 == D / 32) {                                        // O has been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(o_free + x);
                }
                stage_rows<DT>(stage + j * OutStage<32>::BYTES, v, inv, lane);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < D / 32; ++j)
                    tma_store_5d(&tm_o, smem_u32(stage + j * OutStage<32>::BYTES), 32 * j, c0, r0 + quarter * (32 / TW), hn, hb);
                bulk_commit();
            }
            if (qr < g.Hq && qc < g.W)
                lse[(static_cast<size_t>(bn) * g.Hq + qr) * g.W + qc] = (fin + log2f(total)) * kLn2;
        }
        if (lane == 0) bulk_wait<0>();                       // the staging buffers have been read, the rows written
    } else {
        // ------------------------------------------------------------------ softmax warps
        reg_inc<kDkvRegsSoftmax>();
        const int quarter = warp & 3, group = warp >> 2;
        const int row = quarter * 32 + lane;                 // query of the tile = tensor-memory lane
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        const uint32_t s_addr = tmem_lane + C::TMEM_S + group * C::TMEM_SSTRIDE;
        const uint32_t o_addr = tmem_lane + C::TMEM_O + group * C::TMEM_OSTRIDE;
        constexpr int NACT = C::NACT;
        uint32_t m = 0;                          // chunks of this group so far
        TileWalk walk((int)blockIdx.x + group * (int)gridDim.x, 2 * (int)gridDim.x, tiles_r, tiles_c);
        for (int i = group; i < n_my; i += 2, walk.next()) {
            const int r0 = walk.row(), c0 = walk.col();
            const int box_r0 = na2d_ws(g.q_row0 + r0, g.Hg, KS) - g.kv_row0;
            const int box_c0 = na2d_ws(c0, g.W, KS);
            const int qr = min(r0 + (row / TW), g.Hq - 1), qc = min(c0 + (row % TW), g.W - 1);
            const int wr = na2d_ws(g.q_row0 + qr, g.Hg, KS) - g.kv_row0 - box_r0;   // in [0, TH)
            const int wc = na2d_ws(qc, g.W, KS) - box_c0;                            // in [0, TW)
            const int wr_lo = __shfl_sync(0xffffffffu, wr, 0);
            const int wr_hi = __shfl_sync(0xffffffffu, wr, 31);
            // The warp's queries see strip rows [wr_lo, wr_hi + ks), the same in every strip: 16-column blocks b_lo ..
            // b_lo + NACT - 1, and one more if `extra`.  row_cap: infinity for the rows of those that this query sees, -infinity
            // for the others.
            const int b_lo = min((wr_lo * C::HW) >> 4, C::NB16 - NACT);
            const bool extra = (wr_hi + KS) * C::HW > 16 * (b_lo + NACT);
            float row_cap[(NACT + 1) * C::ROWS16];
#pragma unroll
            for (int r = 0; r < (NACT + 1) * C::ROWS16; ++r)
                row_cap[r] = (unsigned)(b_lo * C::ROWS16 + r - wr) < (unsigned)KS ? CUDART_INF_F : -CUDART_INF_F;
            const uint32_t window = ((1u << KS) - 1u) << wc;                         // this query's columns of the box
            float run_max = -CUDART_INF_F, run_sum = 0.f;

            for (int ch = 0; ch < C::NCH; ++ch, ++m) {
                const uint32_t cols = C::seen_cols(window, ch);
                float col_cap[C::HW];
#pragma unroll
                for (int c = 0; c < C::HW; ++c) col_cap[c] = ((cols >> c) & 1u) ? CUDART_INF_F : -CUDART_INF_F;
                if ((tid & 127) == 0) NA2D_TR(group ? 0 : 3, 0, m);
                mbar_wait(s_full + group, m & 1, wctx, kErrMmaWait);
                tc_fence_after();
                if ((tid & 127) == 0) NA2D_TR(group ? 0 : 3, 1, m);
                uint32_t s[NACT + 1][16];
#pragma unroll
                for (int a = 0; a < NACT; ++a) tmem_ld_32x16(s_addr + 16 * (b_lo + a), s[a]);
                if (extra) tmem_ld_32x16(s_addr + 16 * (b_lo + NACT), s[NACT]);                       // warp-uniform
                tmem_ld_wait();
                if ((tid & 127) == 0) NA2D_TR(group ? 0 : 3, 2, m);
                // Columns outside the window become -inf, whatever they hold (the minimum with -inf; a NaN of the window
                // becomes +inf here and a NaN again in exp2(inf - inf)).  One three-input minimum and half a three-input
                // maximum an element: selecting by mask bits took twice the time, on the same pipe.
                float mx[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
                auto mask_block = [&](int a) {
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        const float x0 = min3(__uint_as_float(s[a][e]), col_cap[e % C::HW], row_cap[a * C::ROWS16 + e / C::HW]);
                        const float x1 = min3(__uint_as_float(s[a][e + 1]), col_cap[(e + 1) % C::HW], row_cap[a * C::ROWS16 + e / C::HW]);
                        s[a][e] = __float_as_uint(x0);
                        s[a][e + 1] = __float_as_uint(x1);
                        mx[(e / 2) & 3] = max3(mx[(e / 2) & 3], x0, x1);
                    }
                };
#pragma unroll
                for (int a = 0; a < NACT; ++a) mask_block(a);
                if (extra) mask_block(NACT);
                const float cmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * g.sl2;
                if ((tid & 127) == 0) NA2D_TR(group ? 0 : 3, 3, m);
                // Whenever a row's maximum grows its sums are rescaled, so that the largest weight of a row so far is an exact 1: kept
                // at an older maximum, as long as the weights stay in range, it would be rounded, and o be up to 4 % further off (and 5 %
                // faster at head dim 128).
                const bool grow = cmax > run_max;
                if (ch > 0 && __any_sync(0xffffffffu, grow && run_max != -CUDART_INF_F)) {
                    // (O holds the chunks before: their P V went ahead of this chunk's scores)
                    const float alpha = grow ? fast_exp2(run_max - cmax) : 1.f;
                    const uint64_t alpha2 = pair2(alpha, alpha);
#pragma unroll
                    for (int piece = 0; piece < D / 16; ++piece) {
                        uint32_t v[16];
                        tmem_ld_32x16(o_addr + 16 * piece, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; e += 2) {
                            const uint64_t x = mul2(pair2(v[e], v[e + 1]), alpha2);
                            v[e] = __float_as_uint(lo2(x));
                            v[e + 1] = __float_as_uint(hi2(x));
                        }
                        tmem_st_32x16(o_addr + 16 * piece, v);
                    }
                    run_sum *= alpha;
                }
                if (grow) run_max = cmax;
                const float safe_max = (run_max == -CUDART_INF_F) ? 0.f : run_max;
                // P = exp2(s * log2e - max) as packed 16-bit pairs -> tensor memory (over S), row sum; zeros in the
                // blocks the warp cannot see
                {
                    const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
                    for (int t = 0; t < C::NB16; ++t)
                        if (t < b_lo || t >= b_lo + NACT + (extra ? 1 : 0)) tmem_st_32x8(s_addr + 8 * t, z);
                }
                uint64_t sum2[2] = {0, 0};
                const uint64_t scale2 = pair2(g.sl2, g.sl2), max2 = pair2(-safe_max, -safe_max);
                // (a block is stored after the next one's exponentials have been issued: its conversions are done by then)
                uint32_t w[2][8];
                auto exp_block = [&](int a) {
#pragma unroll
                    for (int e2 = 0; e2 < 8; ++e2) {
                        const uint64_t x = fma2(pair2(s[a][2 * e2], s[a][2 * e2 + 1]), scale2, max2);
                        const float p0 = fast_exp2(lo2(x)), p1 = fast_exp2(hi2(x));
                        sum2[e2 & 1] = add2(sum2[e2 & 1], pair2(p0, p1));
                        w[a & 1][e2] = pack2<DT>(p0, p1);
                    }
                };
#pragma unroll
                for (int a = 0; a < NACT; ++a) {
                    exp_block(a);
                    if (a > 0) tmem_st_32x8(s_addr + 8 * (b_lo + a - 1), w[(a - 1) & 1]);
                }
                if (extra) {
                    exp_block(NACT);
                    tmem_st_32x8(s_addr + 8 * (b_lo + NACT), w[NACT & 1]);
                }
                tmem_st_32x8(s_addr + 8 * (b_lo + NACT - 1), w[(NACT - 1) & 1]);
                const uint64_t sum = add2(sum2[0], sum2[1]);
                run_sum += lo2(sum) + hi2(sum);
                if (ch == C::NCH - 1) {          // for the epilogue warps, ahead of the arrival that lets the last P V go
                    x_sum[group * 128 + row] = run_sum;
                    x_fin[group * 128 + row] = safe_max;
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + group);
                if ((tid & 127) == 0) NA2D_TR(group ? 0 : 3, 4, m);
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

template <typename DT, int D, int KS>
int launch_forward2(const LaunchCtx& lc, const TensorArg& q, const TensorArg& k, const TensorArg& v, const TensorArg& o,
                    float* lse, long long tiles, int tiles_r, int tiles_c) {
    using C = Fwd2Cfg<D, KS>;
    const Na2dGeom& g = lc.g;
    CUtensorMap tq, tk, tv, to;
    int rc = make_map(&tq, q, lc.dtype, lc.B, g.N, g.Hq, g.W, D, TW, TH);
    if (rc == NA2D_OK) rc = make_map(&to, o, lc.dtype, lc.B, g.N, g.Hq, g.W, D, TW, 32 / TW, 32);
    if (rc == NA2D_OK) rc = make_map(&tk, k, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, C::HW, C::HH);
    if (rc == NA2D_OK) rc = make_map(&tv, v, lc.dtype, lc.B, g.N, g.Hkv, g.W, D, C::HW, C::HH);
    if (rc != NA2D_OK) return rc;
    auto kern = fwd2_kernel<DT, D, KS>;
    static std::atomic<unsigned long long> opted{0};
    if (opt_in_smem(kern, C::SMEM, lc.device, opted) != cudaSuccess) return NA2D_ERR_CUDA;
    *lc.launched += 1;
    return na2d_launch::launch(lc.overlap, kern, persistent_grid(lc, tiles), 512, C::SMEM, lc.st,
                               tq, tk, tv, to, lse, lc.errors, g, tiles_r, tiles_c, (int)tiles) == cudaSuccess
               ? NA2D_OK
               : NA2D_ERR_CUDA;
}

}  // namespace na2d_tc
