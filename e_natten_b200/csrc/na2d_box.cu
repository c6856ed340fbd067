// Launchers of the box kernels.
#include "na2d_box_entry.h"

#include "na2d_box_key.cuh"
#include "na2d_tc.cuh"

namespace na2d_box {
namespace {

using na2d_tile::Tensor;

// Calls f(Shape) for the window size.
template <typename F>
int by_size(const Na2dGeom& g, F&& f) {
    switch (g.ks) {
        case 3: return f(Shape<3>{});
        case 5: return f(Shape<5>{});
        case 7: return f(Shape<7>{});
        case 9: return f(Shape<9>{});
        case 11: return f(Shape<11>{});
        case 13: return f(Shape<13>{});
        default: return NA2D_ERR_UNSUPPORTED;
    }
}

// Blocks of a launch over `rows` rows of tiles of `units` units.
template <typename S>
int tiles(const Na2dGeom& g, long long units, int rows, unsigned* n) {
    const long long t = units * rows * ((g.W + S::kTw - 1) / S::kTw);
    if (t > 0x7fffffffLL) return NA2D_ERR_TOO_LARGE;
    *n = (unsigned)t;
    return NA2D_OK;
}
template <typename S> int tile_rows(int H) { return (H + S::kTh - 1) / S::kTh; }

Operand operand(const Tensor& t) { return Operand{t.ptr, t.st, 1}; }

// Map of boxes of channels x w x h pixels of a tensor of `rows` image rows; false where there is none.
bool map(CUtensorMap* m, const Call& c, const Tensor& t, int rows, int w, int h, int channels) {
    return na2d_tc::try_map(m, na2d_tc::TensorArg{t.ptr, t.st}, NA2D_F32, c.g.BN / c.g.N, c.g.N, rows, c.g.W, c.g.C, w, h, channels, true);
}
template <typename S> bool map_own(CUtensorMap* m, const Call& c, const Tensor& t) { return map(m, c, t, c.g.Hq, S::kOwnW, S::kTh, kDotC); }
template <typename S> bool map_dot(CUtensorMap* m, const Call& c, const Tensor& t) { return map(m, c, t, c.g.Hkv, S::kBoxW, S::kHaloH, kDotC); }
template <typename S> bool map_halo(CUtensorMap* m, const Call& c, const Tensor& t) { return map(m, c, t, c.g.Hkv, S::kHaloW, S::kHaloH, kChunk); }
template <typename S> bool map_key(CUtensorMap* m, const Call& c, const Tensor& t, bool wide) {
    using K = KeyShape<S>;
    return map(m, c, t, c.g.Hq, wide ? K::kWideW : S::kBoxW, wide ? K::kWideH : S::kHaloH, kChunk);
}

// (`Tag` tells one kernel's opt-in from another's.)
template <typename Tag, typename... P, typename... A>
int launch(const Call& c, void (*kernel)(P...), dim3 grid, int threads, int smem, A&&... args) {
    static std::atomic<unsigned long long> opted_in{0};
    if (na2d_tc::opt_in_smem(kernel, smem, c.device, opted_in) != cudaSuccess) return NA2D_ERR_CUDA;
    kernel<<<grid, threads, smem, c.st>>>(static_cast<P>(args)...);
    return cudaPeekAtLastError() == cudaSuccess ? NA2D_OK : NA2D_ERR_CUDA;
}
template <int KS, int WHICH, bool FLAG> struct Tag {};

// Channels that a block of the apply and key sum kernels takes, whose blocks need not take all of them.  `blocks` tiles on a GPU with room
// for `per_sm` blocks an SM.  A wave of k blocks an SM lasts 0.73 + 0.27 k times as long as one block, or k * alone times where that is more: the
// part of an SM's throughput that a block uses which has it to itself.  Fetching the weights, which each block does, takes as long as `fetch` chunks
// of channels.  Fitted to times of all splits of 2 to 4 chunks, 20 to 1536 tiles, windows 3 to 13, one B200: on average the split taken is within
// 1 % of the best one's time for the apply, 2 to 7 % for the pair's key sums and 1 to 3 % for the backward's.  One chunk's time for
// fetching, and no `alone`, gave 0 to 2, 9 to 18 and 4 to 7 %, and calls slower than the tiled kernels: apply of 6 x 50 x 52 x 64,
// window 9, 18.5 -> 22.5 us, now 18.5; apply and key sums of 6 x 64 x 64 x 128, window 7, 100 -> 106, now 82.  Left: apply of 150 tiles, two more than
// SMs, at 0.77 (window 11) and 0.86 (9) of the tiled kernels' speed.
struct Split {
    float fetch, alone;
};
template <typename S> constexpr Split kApplySplit{0.75f, S::kKs <= 5 ? 0.4f : S::kKs == 9 ? 0.55f : 0.8f};
template <typename S> constexpr Split kKeySplit{0.1f, S::kKs <= 5 ? 0.3f : S::kKs == 9 ? 0.5f : 0.85f};
int channels_of_block(const Call& c, const Split& split, long long blocks, int per_sm) {
    const int sms = na2d_tc::sm_count(c.device), chunks = (c.g.C + kChunk - 1) / kChunk;
    const auto wave = [&](long long k) { return fmaxf(0.73f + 0.27f * (float)k, split.alone * (float)k); };
    float best = 0.f;
    int span = chunks;
    for (int parts = 1; parts <= chunks; ++parts) {
        const int per = (chunks + parts - 1) / parts, used = (chunks + per - 1) / per;
        const long long all = blocks * used, slots = (long long)sms * per_sm, rest = all % slots;
        const float waves = (float)(all / slots) * wave(per_sm) + (rest ? wave((rest + sms - 1) / sms) : 0.f);
        const float time = waves * (split.fetch + (float)chunks / (float)used);
        if (parts == 1 || time < 0.97f * best) {
            best = time;
            span = per;
        }
    }
    return span * kChunk;
}

}  // namespace

int forward(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, float* lse) {
    return by_size(c.g, [&](auto shape) -> int {
        using S = decltype(shape);
        unsigned n = 0;
        if (int rc = tiles<S>(c.g, c.g.BN, tile_rows<S>(c.g.Hq), &n)) return rc;
        CUtensorMap mq, mk, mv;
        if (!map_own<S>(&mq, c, q) || !map_dot<S>(&mk, c, k) || !map_halo<S>(&mv, c, v)) return kNoMap;
        auto run = [&](auto park) {
            constexpr bool kPark = decltype(park)::value;
            return launch<Tag<S::kKs, 0, kPark>>(c, fwd_kernel<S::kKs, kPark>, n, S::kThreads, S::kSmem, mq, mk, mv, operand(o), lse, c.errors, c.g);
        };
        return c.g.C > kParkAbove ? run(std::true_type{}) : run(std::false_type{});
    });
}

int query_half(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& d_o, const Tensor& d_q, const float* lse,
               float* delta, float* row_factor, float4* p, float4* ds, int units, const Rows& rows) {
    return by_size(c.g, [&](auto shape) -> int {
        using S = decltype(shape);
        unsigned n = 0;
        if (int rc = tiles<S>(c.g, units, rows.rows, &n)) return rc;
        CUtensorMap mg, mv, mq, mk, mk32;
        if (!map_own<S>(&mg, c, d_o) || !map_dot<S>(&mv, c, v) || !map_own<S>(&mq, c, q) || !map_dot<S>(&mk, c, k) || !map_halo<S>(&mk32, c, k))
            return kNoMap;
        const Band band{rows.unit0, rows.row0, rows.rows, rows.ring};
        auto run = [&](auto park) {
            constexpr bool kPark = decltype(park)::value;
            return launch<Tag<S::kKs, 1, kPark>>(c, dq_kernel<S::kKs, kPark>, n, S::kThreads, S::kSmem, mg, mv, mq, mk, mk32, operand(d_q), lse,
                                                 delta, row_factor, p, ds, c.errors, band, c.g);
        };
        return c.g.C > kParkAbove ? run(std::true_type{}) : run(std::false_type{});
    });
}

int key_half(const Call& c, const Tensor& q, const Tensor& d_o, const Tensor& d_k, const Tensor& d_v, const float4* p, const float4* ds, int units,
             const Rows& rows) {
    return by_size(c.g, [&](auto shape) -> int {
        using S = decltype(shape);
        using K = KeyShape<S>;
        unsigned n = 0;
        if (int rc = tiles<S>(c.g, units, rows.rows, &n)) return rc;
        CUtensorMap xq, wq, xg, wg;
        if (!map_key<S>(&xq, c, q, false) || !map_key<S>(&wq, c, q, true) || !map_key<S>(&xg, c, d_o, false) || !map_key<S>(&wg, c, d_o, true))
            return kNoMap;
        const int span = channels_of_block(c, kKeySplit<S>, 2ll * n, K::kBlocks);
        return launch<Tag<S::kKs, 2, true>>(c, key_sum_kernel<true, S::kKs>, dim3(n, 2, (c.g.C + span - 1) / span), K::kThreads, K::kSmem, xq, wq,
                                            xg, wg, KeyOut{ds, operand(d_k)}, KeyOut{p, operand(d_v)}, span, c.errors,
                                            Band{rows.unit0, rows.row0, rows.rows, rows.ring}, c.g);
    });
}

int pair_dot(const Call& c, const Tensor& x, const Tensor& y, float* attn) {
    return by_size(c.g, [&](auto shape) -> int {
        using S = decltype(shape);
        unsigned n = 0;
        if (int rc = tiles<S>(c.g, c.g.BN, tile_rows<S>(c.g.Hq), &n)) return rc;
        CUtensorMap mx, my;
        if (!map_own<S>(&mx, c, x) || !map_dot<S>(&my, c, y)) return kNoMap;
        auto run = [&](auto park) {
            constexpr bool kPark = decltype(park)::value;
            return launch<Tag<S::kKs, 3, kPark>>(c, window_dot_kernel<S::kKs, kPark>, n, S::kThreads, PairShape<S>::kDotSmem, mx, my, attn, c.errors, c.g);
        };
        return c.g.C > kParkAbove ? run(std::true_type{}) : run(std::false_type{});
    });
}

int pair_apply(const Call& c, const float* attn, const Tensor& y, const Tensor& out) {
    return by_size(c.g, [&](auto shape) -> int {
        using S = decltype(shape);
        unsigned n = 0;
        if (int rc = tiles<S>(c.g, c.g.BN, tile_rows<S>(c.g.Hq), &n)) return rc;
        CUtensorMap my;
        if (!map_halo<S>(&my, c, y)) return kNoMap;
        using P = PairShape<S>;
        const int span = channels_of_block(c, kApplySplit<S>, n, P::kApplyBlocks);
        return launch<Tag<S::kKs, 4, true>>(c, window_apply_kernel<S::kKs>, dim3(n, 1, (c.g.C + span - 1) / span), P::kApplyThreads, P::kApplySmem,
                                            attn, my, operand(out), span, c.errors, c.g);
    });
}

int pair_inverse(const Call& c, const float* attn, const Tensor& x, const Tensor& out) {
    return by_size(c.g, [&](auto shape) -> int {
        using S = decltype(shape);
        using K = KeyShape<S>;
        unsigned n = 0;
        const int rows = tile_rows<S>(c.g.Hkv);
        if (int rc = tiles<S>(c.g, c.g.BN, rows, &n)) return rc;
        CUtensorMap mx, mw;
        if (!map_key<S>(&mx, c, x, false) || !map_key<S>(&mw, c, x, true)) return kNoMap;
        const KeyOut sum{attn, operand(out)};
        const int span = channels_of_block(c, kKeySplit<S>, n, K::kBlocks);
        return launch<Tag<S::kKs, 5, true>>(c, key_sum_kernel<false, S::kKs>, dim3(n, 1, (c.g.C + span - 1) / span), K::kThreads, K::kSmem, mx, mw,
                                            mx, mw, sum, sum, span, c.errors,
                                            Band{0, 0, rows, rows}, c.g);
    });
}

}  // namespace na2d_box
