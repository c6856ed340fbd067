// fp32 kernels of the 2D operator and the unfused pair, kernel sizes 3 to 13, for operands that a tensor map can describe (rows that
// start on 16-byte boundaries): what na2d_tile.cuh does, with the boxes brought by TMA.
//
// A block owns a tile of 8 x (4 * kStrips) pixels of one (batch, head) image.  Two loops do the work:
//   dot    a thread holds the scores of a strip of four neighbouring pixels against one window row, 16 channels of the tile's own
//          pixels and of its halo at a time, the next 16 on their way meanwhile;
//   apply  a thread holds four channels of an output for a strip (kRows image rows of it), 32 channels of the halo at a time.
// In the key half of the backward a thread holds four channels of a strip of keys, and the weights come from the query half.
//
// What bounds them: the FMA pipe (a packed fma.f32x2 takes it for two cycles: no more multiply-adds a cycle, but half the issue
// slots) and shared-memory reads.  A warp's float4 load takes a cycle for every 128 bytes of different words, so lanes are laid out to
// share them: eight rows x four window rows in the dot loop, eight channel quads x four rows in the apply loop.  Copying with the
// block's own threads (cp.async) took a quarter of all instructions and as much of the shared-memory pipe's time; a second buffer
// for such copies gained nothing.  A TMA box costs one thread one instruction.
//
// Measured on one B200 against the tiled kernels (na2d_tile.cuh): forward / query half of 2 x 4 x 56 x 56 x 128, us: window 3 33 -> 21 / 47 -> 29,
// 5 45 -> 40 / 66 -> 57, 7 59 -> 57 / 90 -> 84, 9 83 -> 72 / 126 -> 107, 11 100 -> 95 / 159 -> 140, 13 142 -> 138 / 209 -> 216; of 2 x 200 x 260 x 64:
// 44 -> 28 / 62 -> 39, 56 -> 46 / 79 -> 66, 90 -> 80 / 129 -> 114, 137 -> 127 / 208 -> 180, 178 -> 165 / 269 -> 242, 252 -> 221 / 380 -> 355.
//
// Boxes.  Pixel after pixel, 64 or 128 bytes each, in the swizzle that goes with that size, rows an odd number of pixels long: eight
// rows of a column then lie on different banks, as do the channels of a pixel.
#pragma once

#include <cuda.h>
#include <float.h>
#include <math_constants.h>

#include <type_traits>

#include "na2d_tile_bwd.cuh"

namespace na2d_box {

using na2d_ptx::add2;
using na2d_ptx::ErrorState;
using na2d_ptx::fma2;
using na2d_ptx::hi2;
using na2d_ptx::lo2;
using na2d_ptx::mul2;
using na2d_ptx::pair2;
using na2d_ptx::WaitCtx;
using na2d_ptx::WaitState;
using na2d_tile::Band;
using na2d_tile::copies_done;
using na2d_tile::copy16;
using na2d_tile::kR;
using na2d_tile::lane_of;
using na2d_tile::max_of;
using na2d_tile::Operand;
using na2d_tile::sum2;
using na2d_tile::sum_rows;
using na2d_tile::Tile;
using na2d_tile::tile_of_block;
using na2d_tile::unit;

constexpr int kDotC = 16, kDotPixel = 4 * kDotC;         // channels of a dot chunk, bytes of a pixel of it
constexpr int kChunk = 32, kPixel = 4 * kChunk;          // of an apply chunk
constexpr int kF = kChunk / 4;                           // float4 per pixel of an apply chunk

template <int KS>
constexpr int kTaps = KS * KS;

__host__ __device__ constexpr int whole_kb(int bytes) { return (bytes + 1023) / 1024 * 1024; }

// Geometry of a tile for window size KS.
template <int KS>
struct Shape {
    static constexpr int kKs = KS, kKh = KS;
    static constexpr int kTh = 8, kStrips = KS <= 7 ? 4 : 2, kTw = kR * kStrips;
    static constexpr int kU = KS + kR - 1;                // halo columns a strip reaches
    static constexpr int kHaloH = kTh + KS - 1, kHaloW = kTw + KS - 1;
    static constexpr int kOwnW = kTw | 1, kBoxW = kHaloW | 1;            // columns of the boxes
    static constexpr int kItems = kTh * kStrips * KS;     // (row, strip, window row) of the dot loop
    // Image rows of a thread in the apply loop, and lanes that share the halo rows that those meet: two rows read a halo pixel once for
    // both; from window 7 on that leaves threads idle, and two lanes take every other halo row (window 13 would spill with it).
    // Forward of 2 x 4 x 56 x 56 x 128, window 9, one row / two lanes of two: 77 / 73 us, window 11 104 / 96, window 13 137 / 151.
    static constexpr int kHalves = KS >= 7 && KS <= 11 ? 2 : 1, kRows = KS <= 11 ? 2 : 1;
    static constexpr int kApply = kTh / kRows * kHalves * kStrips * kF;
    static constexpr int kThreads = max_of((kItems + 31) / 32 * 32, max_of(kApply, 128));
    // Weights as the key half gets them: a slot of four pixels for each column of a strip's halo band.
    static constexpr int kBand = kTh * kStrips * KS * kU;
    // Shared memory, in bytes: two stages of a dot chunk (own pixels, halo), in whose place come one or, where that costs no block,
    // two apply chunks' halos; the weights, a slot of four pixels for each member of a window row; barriers.
    // The last dot chunk lies in the first stage and the first halo from the second one on, or at the start if it is the only
    // one and would cost a block there.
    static constexpr int kOwn = whole_kb(kTh * kOwnW * kDotPixel), kStage = kOwn + whole_kb(kHaloH * kBoxW * kDotPixel);
    static constexpr int kHalo = whole_kb(kHaloH * kHaloW * kPixel);
    static constexpr int kWeights = kTh * kStrips * KS * KS;             // slots
    static constexpr int kExchange = 2 * kTh * kStrips * KS;             // row maxima and sums, float4
    static constexpr int kBarriers = 64;
    static constexpr int kBlocksReg = 65536 / (kThreads * (KS >= 9 ? 144 : 128)) < 1 ? 1 : 65536 / (kThreads * (KS >= 9 ? 144 : 128));
    static constexpr int kSecondHalo = max_of(kStage, kHalo);
    static constexpr int kHaloBuffers = KS <= 5 ? 2 : 1;
    static constexpr int kHaloAt = kHaloBuffers == 2 ? kSecondHalo : 0, kExchangeAt = kHaloBuffers == 2 ? 0 : kHalo;
    static constexpr int kStaged = max_of(max_of(2 * kStage, kHaloAt + kHalo), kExchangeAt + kExchange * 16);
    static constexpr int kWeightsAt = kStaged, kBarriersAt = kStaged + kWeights * 16;
    static constexpr int kSmem = kBarriersAt + kBarriers;
    static constexpr int kBlocksSmem = na2d_tile::kSmemPerSm / (kSmem + 1024);
    static constexpr int kBlocks = kBlocksSmem < kBlocksReg ? kBlocksSmem : kBlocksReg;
    static_assert(kHaloBuffers == 1 || kExchange * 16 <= kHaloAt, "the exchange is clear of the first halo");
    static_assert(kBlocks >= 1 && kApply <= kThreads, "a block fits an SM, an apply item a thread");
};

// Where a pixel of a box lies, its first channels' place in the swizzle included: float4 f of it at (that ^ 16 f).
__device__ __forceinline__ int dot_pixel(int p) { return p * kDotPixel + (p << 3 & 0x30); }
__device__ __forceinline__ int pixel(int p) { return p * kPixel + (p << 4 & 0x70); }
__device__ __forceinline__ ulonglong2 quad_at(const uint8_t* smem, int at) { return *reinterpret_cast<const ulonglong2*>(smem + at); }

// ------------------------------------------------------------------------------------ loads
// Buffers of a block: the two dot stages, the two halos of the apply loop.  Each has a barrier that its loads complete, and a count
// of the warps that are done reading it: the last one loads what comes next, so that no warp waits for another between chunks.
struct Loads {
    static constexpr int kBuffers = 4;
    uint64_t* bars;
    unsigned* done;
    WaitCtx wc;
    uint32_t phases;              // parity of each barrier's next phase
    bool gave_up;                 // a wait of this thread
    __device__ __forceinline__ explicit Loads(uint8_t* at, const ErrorState* errors)
        : bars(reinterpret_cast<uint64_t*>(at)), done(reinterpret_cast<unsigned*>(at + 32)), wc{reinterpret_cast<WaitState*>(at + 48)},
          phases(0), gave_up(false) {
        if (threadIdx.x == 0) {
            na2d_ptx::wait_state_init(wc.st, errors, na2d_ptx::kWaitLimitNs);
            for (int i = 0; i < kBuffers; ++i) {
                na2d_ptx::mbar_init(bars + i, 1);
                done[i] = 0;
            }
            na2d_ptx::mbar_fence_init();
        }
    }
    // The barrier for the buffer's next load, which expects so many bytes; null, and no load may start, once a wait of this thread has given
    // up: the phase that it waited for may still be open, and a second arrival in it would be an error of its own.  A phase that this thread
    // has seen complete is over for all, also where others have given up on it.  (The block's abort flag says less, and reading it
    // here, between a buffer's last reader and its next load, took 4 to 10 % of the kernels' time.)
    __device__ __forceinline__ uint64_t* expect(int b, int bytes) const {
        if (gave_up) return nullptr;
        na2d_ptx::mbar_expect_tx(bars + b, bytes);
        return bars + b;
    }
    __device__ __forceinline__ void wait(int b) {
        if (!na2d_ptx::mbar_wait(bars + b, phases >> b & 1, wc, na2d_ptx::kErrLoadWait)) gave_up = true;
        phases ^= 1u << b;
    }
    // The warp has read the buffer; true in one thread of the last warp to say so.
    __device__ __forceinline__ bool last(int b) const {
        __syncwarp();
        if (threadIdx.x % 32 != 0) return false;
        unsigned before;
        asm volatile("atom.acq_rel.cta.shared::cta.inc.u32 %0, [%1], %2;"
                     : "=r"(before) : "r"(na2d_ptx::smem_u32(done + b)), "r"(blockDim.x / 32 - 1) : "memory");
        return before == blockDim.x / 32 - 1;
    }
    // After a wait that gave up: waits once more, about a millisecond for each barrier at most, before the block's shared memory becomes
    // another one's.  A load that this thread has started and not seen land is in its barrier's open phase, since none follows it; of the two
    // parities the other one's phase is over.  A load that another thread started is that one's to wait for.
    __device__ __forceinline__ void drain() const {
        if (!gave_up) return;
        for (int b = 0; b < kBuffers; ++b)
            for (uint32_t parity = 0; parity < 2; ++parity) na2d_ptx::mbar_wait(bars + b, parity, wc, na2d_ptx::kErrLoadWait);
    }
};

// The tile's own pixels and their halo, 16 channels, to a stage.
template <typename S>
__device__ __forceinline__ void load_dot(const CUtensorMap* own, const CUtensorMap* halo, uint8_t* stage, uint64_t* bar, int chunk, const Tile& t,
                                         int ky0, int kx0) {
    na2d_ptx::tma_load_5d(stage, own, bar, chunk * kDotC, t.x0, t.y0, t.n, t.b);
    na2d_ptx::tma_load_5d(stage + S::kOwn, halo, bar, chunk * kDotC, kx0, ky0, t.n, t.b);
}
template <typename S>
constexpr int kDotBytes = S::kTh * S::kOwnW * kDotPixel + S::kHaloH * S::kBoxW * kDotPixel;
template <typename S>
constexpr int kHaloBytes = S::kHaloH * S::kHaloW * kPixel;
// Buffer of an apply chunk, and where it lies.
template <typename S>
__device__ __forceinline__ int halo_buffer(int i) { return S::kHaloBuffers == 2 ? i & 1 : 0; }
template <typename S>
__device__ __forceinline__ int halo_at(int i) { return halo_buffer<S>(i) ? 0 : S::kHaloAt; }

// False, and reported, where the swizzle would not fit the shared memory's start; never seen.
__device__ __forceinline__ bool starts_right(const uint8_t* smem, const ErrorState* errors) {
    if ((na2d_ptx::smem_u32(smem) & 1023u) == 0) return true;
    if (threadIdx.x == 0) na2d_ptx::report_error(errors->error_bytes, na2d_ptx::kErrSmemBase);
    return false;
}

// ------------------------------------------------------------------------------------ strips, scores
// The windows of a strip of four query columns starting at c0: column r's window covers halo columns
// [off[r], off[r] + KS) counted from `start`, the window start of column c0.
struct Strip {
    int start, off[kR];
    bool regular;                 // off[r] is r, and all four columns are in the image
};
template <int KS>
__device__ __forceinline__ Strip strip_at(int c0, int W) {
    Strip s;
    s.start = na2d_ws(min(c0, W - 1), W, KS);
#pragma unroll
    for (int r = 0; r < kR; ++r) s.off[r] = na2d_ws(min(c0 + r, W - 1), W, KS) - s.start;
    s.regular = c0 >= KS / 2 && c0 + kR - 1 + KS / 2 < W;
    return s;
}

// A score's running sum: even and odd channels apart in a register pair, where that many registers are to be had.
template <typename S>
using Sum = std::conditional_t<(S::kKs > 5), float, uint64_t>;
__device__ __forceinline__ void add_pair(uint64_t& acc, uint64_t x) { acc = add2(acc, x); }
__device__ __forceinline__ void add_pair(float& acc, uint64_t x) { acc += sum2(x); }
__device__ __forceinline__ float value(uint64_t acc) { return sum2(acc); }
__device__ __forceinline__ float value(float acc) { return acc; }
__device__ __forceinline__ void set(uint64_t& acc, float x) { acc = pair2(x, 0.f); }
__device__ __forceinline__ void set(float& acc, float x) { acc = x; }

// Scores over the channels so far, parked in the thread's local memory (na2d_tile.cuh says why): what the addition to the parked sum
// rounds off starts the next one.  Up to 64 channels that is at 16 and 48, since 16 + 32 + 16 round less than 32 + 32, beyond
// that every 32; up to 32 not at all.
constexpr int kParkAbove = 32;
__device__ __forceinline__ bool park_at(int c, int C) { return c < C && (C <= 64 ? c % 32 != 0 : c % 32 == 0); }
template <typename A, int N>
__device__ __forceinline__ void park(A (&acc)[kR][N], float4* parked, bool first) {
    float largest = 0.f;
#pragma unroll
    for (int i = 0; i < kR * N; i += kR) {
        const float4 old = first ? make_float4(0.f, 0.f, 0.f, 0.f) : parked[i / kR];
        float sum[kR] = {old.x, old.y, old.z, old.w};
#pragma unroll
        for (int e = 0; e < kR; ++e) {
            A& own = acc[(i + e) / N][(i + e) % N];
            const float a = value(own), total = __fadd_rn(sum[e], a);
            set(own, __fsub_rn(a, __fsub_rn(total, sum[e])));
            largest = fmaxf(largest, fabsf(total));
            sum[e] = total;
        }
        parked[i / kR] = make_float4(sum[0], sum[1], sum[2], sum[3]);
    }
    if (largest > FLT_MAX) {                               // an infinite sum stays one
#pragma unroll
        for (int i = 0; i < kR * N; i += kR) {
            const float4 sum = parked[i / kR];
#pragma unroll
            for (int e = 0; e < kR; ++e)
                if (fabsf(lane_of(sum, e)) > FLT_MAX) acc[(i + e) / N][(i + e) % N] = 0;
        }
    }
}

// What a thread does in the dot loop: window row u of the strip `strip` of tile row `row`.
struct DotItem {
    int row, u, strip;
    bool active;
    int hy, hx;                   // first halo pixel
    bool all_regular;             // every strip of the tile is
    Strip s;
};
// ky0, kx0: local row and column of halo pixel (0, 0).
template <typename S>
__device__ __forceinline__ DotItem score_item(const Tile& t, const Na2dGeom& g, int ky0, int kx0) {
    DotItem d;
    d.row = threadIdx.x % S::kTh;
    const int it = threadIdx.x / S::kTh;
    d.u = it % S::kKh;
    d.strip = it / S::kKh;
    d.active = threadIdx.x < S::kItems && d.row < t.rows && kR * d.strip < t.cols;
    if (!d.active) { d.row = 0; d.u = 0; d.strip = 0; }
    d.s = strip_at<S::kKs>(t.x0 + kR * d.strip, g.W);
    d.hy = na2d_ws(g.q_row0 + t.y0 + d.row, g.Hg, S::kKh) - g.kv_row0 - ky0 + d.u;
    d.hx = d.s.start - kx0;
    d.all_regular = t.x0 >= S::kKs / 2 && t.x0 + S::kTw - 1 + S::kKs / 2 < g.W;
    return d;
}

// acc[r][i] += own pixel r . halo column i of the strip over a stage, or (N = KS) member i of its window row, eight channels at a time:
// even and odd channels in the two lanes of a register pair, four products of a lane summed first and added as one number: five
// instructions where eight multiply-adds would stand.
template <typename S, bool REGULAR, typename A, int N>
__device__ __forceinline__ void dot_staged(A (&acc)[kR][N], const uint8_t* stage, const DotItem& d) {
    const int own = d.row * S::kOwnW + kR * d.strip, halo = d.hy * S::kBoxW + d.hx;
    const uint8_t* hs = stage + S::kOwn;
#pragma unroll (REGULAR ? kDotC / 8 : 1)
    for (int f = 0; f < kDotC / 4; f += 2) {
        ulonglong2 q0[kR], q1[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            q0[r] = quad_at(stage, dot_pixel(own + r) ^ 16 * f);
            q1[r] = quad_at(stage, dot_pixel(own + r) ^ 16 * f + 16);
        }
        if constexpr (!REGULAR && N == S::kKs) {
#pragma unroll
            for (int r = 0; r < kR; ++r)
#pragma unroll
                for (int m = 0; m < N; ++m) {
                    const int at = dot_pixel(halo + d.s.off[r] + m) ^ 16 * f;
                    const ulonglong2 x0 = quad_at(hs, at), x1 = quad_at(hs, at ^ 16);
                    add_pair(acc[r][m], fma2(q1[r].y, x1.y, fma2(q1[r].x, x1.x, fma2(q0[r].y, x0.y, mul2(q0[r].x, x0.x)))));
                }
        } else
#pragma unroll
        for (int j = 0; j < S::kU; ++j) {
            const int at = dot_pixel(halo + j) ^ 16 * f;
            const ulonglong2 x0 = quad_at(hs, at), x1 = quad_at(hs, at ^ 16);
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                const int i = REGULAR ? j - r : j;
                if (i >= 0 && i < N) add_pair(acc[r][i], fma2(q1[r].y, x1.y, fma2(q1[r].x, x1.x, fma2(q0[r].y, x0.y, mul2(q0[r].x, x0.x)))));
            }
        }
    }
}

__device__ __forceinline__ int dot_chunks(const Na2dGeom& g) { return (g.C + kDotC - 1) / kDotC; }

// Scores of the whole tile, all channel chunks; s[r][m] pixel r of the thread's strip and member m of its window row.  `at`: chunks of
// earlier dot loops of the kernel, `all`: of all of them.  Chunk i of all lies in stage (all - 1 - i) & 1, and the first two are on
// their way; next(i) starts what comes into the place of chunk i once nobody reads it (one thread).
// REGULAR: all strips of the tile are; one way for all of them, since warps hold parts of two strips.  In other tiles a strip reads the
// columns of each pixel's window by themselves up to window 5, and from 7 on gets the scores of all KS + 3 columns it reaches, for each
// pixel, to keep those of its windows at the end (dQ of 4 x 8 x 28 x 30 x 64, window 7, 55 -> 49 us, window 11 134 -> 103).
template <typename S, bool PARK, bool REGULAR, typename F>
__device__ __forceinline__ void tile_dot(float (&s)[kR][S::kKs], const uint8_t* smem, Loads& loads, const DotItem& d, const Na2dGeom& g,
                                         int at, int all, F&& next) {
    constexpr bool kAll = !REGULAR && S::kKs >= 7;
    constexpr int N = kAll ? S::kU : S::kKs;
    using A = std::conditional_t<kAll, float, Sum<S>>;
    A acc[kR][N];
#pragma unroll
    for (int i = 0; i < kR * N; ++i) acc[i / N][i % N] = 0;
    float4 local[PARK ? N : 1];
    float4* parked = local;
    if constexpr (PARK) asm volatile("" : "+l"(parked));    // not in registers: those are needed for the loop
    bool first = true;
    const int n = dot_chunks(g);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int stage = (all - 1 - at - i) & 1;
        loads.wait(stage);
        if (d.active) {
            dot_staged<S, REGULAR>(acc, smem + stage * S::kStage, d);
            if (PARK && park_at((i + 1) * kDotC, g.C)) {
                park(acc, parked, first);
                first = false;
            }
        }
        if (loads.last(stage)) next(at + i);
    }
    float sum[kR][N];
#pragma unroll
    for (int i = 0; i < kR * N; ++i) sum[i / N][i % N] = value(acc[i / N][i % N]);
    if (PARK && !first) {
#pragma unroll
        for (int i = 0; i < kR * N; i += kR) {
            const float4 old = parked[i / kR];
#pragma unroll
            for (int e = 0; e < kR; ++e) sum[(i + e) / N][(i + e) % N] += lane_of(old, e);
        }
    }
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
        for (int m = 0; m < S::kKs; ++m) {
            if constexpr (!kAll) {
                s[r][m] = sum[r][m];
            } else {                                       // off[r] is at most r
                s[r][m] = sum[r][m];
#pragma unroll
                for (int o = 1; o <= r; ++o) s[r][m] = d.s.off[r] == o ? sum[r][m + o] : s[r][m];
            }
        }
}

// The thread's weight slots: member m of its window row, for the four pixels of its strip, at [m * kTh].
template <typename S>
__device__ __forceinline__ float4* weight_slots(float4* w, const DotItem& d) {
    return w + (d.strip * S::kKh + d.u) * S::kKs * S::kTh + d.row;
}
template <typename S>
__device__ __forceinline__ void store_weights(float4* slots, const float (&s)[kR][S::kKs]) {
#pragma unroll
    for (int m = 0; m < S::kKs; ++m) slots[m * S::kTh] = make_float4(s[0][m], s[1][m], s[2][m], s[3][m]);
}

// ------------------------------------------------------------------------------------ apply
// Four channels as two register pairs.
struct Channels {
    uint64_t a, b;
};
__device__ __forceinline__ Channels scaled(float w, const ulonglong2& x) {
    const uint64_t ww = pair2(w, w);
    return Channels{mul2(ww, x.x), mul2(ww, x.y)};
}
__device__ __forceinline__ void add_scaled(Channels& acc, float w, const ulonglong2& x) {
    const uint64_t ww = pair2(w, w);
    acc.a = fma2(ww, x.x, acc.a);
    acc.b = fma2(ww, x.y, acc.b);
}
__device__ __forceinline__ void add(Channels& acc, const Channels& x) {
    acc.a = add2(acc.a, x.a);
    acc.b = add2(acc.b, x.b);
}
__device__ __forceinline__ float4 channels(const Channels& c) { return make_float4(lo2(c.a), hi2(c.a), lo2(c.b), hi2(c.b)); }

// A halo row meets a row of the strip's pixels: acc[r] += sum over its window there, w member m of it at [m * kTh], x the KS + 3 columns
// that the strip reaches.  Each such row is summed by itself first: many short sums round less than a long one.
template <typename S>
__device__ __forceinline__ void apply_band(Channels (&acc)[kR], const float4* w, const ulonglong2 (&x)[S::kU]) {
    Channels t[kR];
#pragma unroll
    for (int m = 0; m < S::kKs; ++m) {
        const float4 wt = w[m * S::kTh];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            if (m == 0) t[r] = scaled(lane_of(wt, r), x[r + m]);
            else add_scaled(t[r], lane_of(wt, r), x[r + m]);
        }
    }
#pragma unroll
    for (int r = 0; r < kR; ++r) add(acc[r], t[r]);
}
// The same where the windows are shifted, for all rows at once (a row that the halo row does not meet gets nothing).
template <typename S, int N, typename X>
__device__ __forceinline__ void apply_shifted(Channels (&acc)[N][kR], const float4* const (&w)[N], const bool (&meets)[N], const Strip& s, X&& x) {
    Channels t[N][kR];
#pragma unroll
    for (int m = 0; m < S::kKs; ++m) {
        float4 wt[N];
#pragma unroll
        for (int p = 0; p < N; ++p) wt[p] = w[p][m * S::kTh];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const ulonglong2 v = x(s.off[r] + m);
#pragma unroll
            for (int p = 0; p < N; ++p) {
                if (m == 0) t[p][r] = scaled(lane_of(wt[p], r), v);
                else add_scaled(t[p][r], lane_of(wt[p], r), v);
            }
        }
    }
#pragma unroll
    for (int p = 0; p < N; ++p)
#pragma unroll
        for (int r = 0; r < kR; ++r)
            if (meets[p]) add(acc[p][r], t[p][r]);
}

// What a thread does in the apply loop: four channels of kRows image rows of a strip, and every kHalves-th of the halo rows that they meet.
template <typename S>
struct ApplyItem {
    int f, half, row, strip;
    bool active;
    __device__ __forceinline__ explicit ApplyItem(const Tile& t) {
        f = threadIdx.x % kF;
        int it = threadIdx.x / kF;
        half = it % S::kHalves;
        it /= S::kHalves;
        row = it % (S::kTh / S::kRows) * S::kRows;
        strip = it / (S::kTh / S::kRows);
        active = threadIdx.x < S::kApply && row < t.rows && kR * strip < t.cols;
    }
};

// out = factor * sum over the window of weight * (what load(i) brings to the halo as chunk i), the chunks of channels [ch0, ch_end); as many
// as there are buffers are on their way.
template <typename S, int BUFFERS, typename F>
__device__ __forceinline__ void tile_apply(const Operand& out, const uint8_t* smem, Loads& loads, const float4* w, const ApplyItem<S>& a,
                                           const float4 (&factor)[S::kRows], const Tile& t, const Na2dGeom& g, int ky0, int kx0, int ch0,
                                           int ch_end, F&& load) {
    const Strip s = strip_at<S::kKs>(t.x0 + kR * a.strip, g.W);
    int off[S::kRows];                                     // first halo row of each pixel row, from the first one's
    const int hy0 = na2d_ws(g.q_row0 + t.y0 + a.row, g.Hg, S::kKh) - g.kv_row0 - ky0;
#pragma unroll
    for (int p = 0; p < S::kRows; ++p)
        off[p] = a.row + p < t.rows ? na2d_ws(g.q_row0 + t.y0 + a.row + p, g.Hg, S::kKh) - g.kv_row0 - ky0 - hy0 : 1 << 20;
    const int n_rows = (S::kRows > 1 && a.row + 1 < t.rows ? off[S::kRows - 1] : 0) + S::kKh;
    const int first = hy0 * S::kHaloW + s.start - kx0;      // the halo pixel of the strip's first column
    const float4* wr = w + a.strip * S::kKh * S::kKs * S::kTh + a.row;
    float* o = unit<float>(out, t) + (t.y0 + a.row) * out.st.h + (t.x0 + kR * a.strip) * out.st.w + 4 * a.f;
#pragma unroll 1
    for (int c0 = ch0, i = 0; c0 < ch_end; c0 += kChunk, ++i) {
        const int buffer = BUFFERS == 2 ? i & 1 : 0;
        loads.wait(2 + buffer);
        const uint8_t* halo = smem + (buffer ? 0 : BUFFERS == 2 ? S::kHaloAt : 0);
        if (a.active) {
            Channels acc[S::kRows][kR];
#pragma unroll
            for (int e = 0; e < S::kRows * kR; ++e) acc[e / kR][e % kR] = Channels{0, 0};
#pragma unroll 1
            for (int h = a.half; h < n_rows; h += S::kHalves) {
                const int at = first + h * S::kHaloW;
                auto column = [&](int j) { return quad_at(halo, pixel(at + j) ^ 16 * a.f); };
                if (s.regular) {
                    ulonglong2 x[S::kU];
#pragma unroll
                    for (int j = 0; j < S::kU; ++j) x[j] = column(j);
#pragma unroll
                    for (int p = 0; p < S::kRows; ++p)
                        if ((unsigned)(h - off[p]) < (unsigned)S::kKh) apply_band<S>(acc[p], wr + (h - off[p]) * (S::kKs * S::kTh) + p, x);
                } else {
                    const float4* wp[S::kRows];
                    bool meets[S::kRows];
#pragma unroll
                    for (int p = 0; p < S::kRows; ++p) {
                        meets[p] = (unsigned)(h - off[p]) < (unsigned)S::kKh;
                        wp[p] = wr + (meets[p] ? h - off[p] : 0) * (S::kKs * S::kTh) + p;
                    }
                    apply_shifted<S>(acc, wp, meets, s, column);
                }
            }
            if constexpr (S::kHalves == 2) {               // each half finishes a row and hands the other one on
                static_assert(S::kRows == 2, "a row each");
                const unsigned both = 0xffffu << (threadIdx.x & 16);
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    const Channels keep = a.half ? acc[1][r] : acc[0][r], give = a.half ? acc[0][r] : acc[1][r];
                    acc[0][r] = keep;
                    add(acc[0][r], Channels{__shfl_xor_sync(both, give.a, kF), __shfl_xor_sync(both, give.b, kF)});
                }
            }
            if (c0 + 4 * a.f < g.C) {
#pragma unroll
                for (int p = 0; p < S::kRows / S::kHalves; ++p) {
                    const int row = S::kHalves == 2 ? a.half : p;
                    if (a.row + row >= t.rows) break;
                    const float4 fac = S::kHalves == 2 && a.half ? factor[S::kRows - 1] : factor[p];
#pragma unroll
                    for (int r = 0; r < kR; ++r) {
                        const float m = lane_of(fac, r);
                        const float4 x = channels(acc[p][r]);
                        if (t.x0 + kR * a.strip + r < g.W)
                            *reinterpret_cast<float4*>(o + row * out.st.h + r * out.st.w + c0) = make_float4(x.x * m, x.y * m, x.z * m, x.w * m);
                    }
                }
            }
        }
        if (loads.last(2 + buffer) && c0 + BUFFERS * kChunk < ch_end) load(i + BUFFERS);
    }
}

// Rows and columns of the halo of a tile of queries.
template <typename S>
__device__ __forceinline__ void query_halo(const Tile& t, const Na2dGeom& g, int& ky0, int& kx0) {
    ky0 = na2d_ws(g.q_row0 + t.y0, g.Hg, S::kKh) - g.kv_row0;
    kx0 = na2d_ws(t.x0, g.W, S::kKs);
}

// ------------------------------------------------------------------------------------ forward
// tm_q: boxes of the tile's own pixels, 16 channels; tm_k, tm_v: halo boxes, 16 and 32 channels.
template <int KS, bool PARK>
__global__ void __launch_bounds__(Shape<KS>::kThreads, Shape<KS>::kBlocks)
fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
           const __grid_constant__ Operand o, float* __restrict__ lse, const ErrorState* __restrict__ errors, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS>;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (!starts_right(smem, errors)) return;
    float4 *w = reinterpret_cast<float4*>(smem + S::kWeightsAt), *mx = reinterpret_cast<float4*>(smem + S::kExchangeAt), *sum = mx + S::kExchange / 2;
    Loads loads(smem + S::kBarriersAt, errors);
    const Tile t = tile_of_block<S>(g, g.Hq);
    int ky0, kx0;
    query_halo<S>(t, g, ky0, kx0);
    const int n = dot_chunks(g);
    auto load_v = [&](int i) {
        if (uint64_t* bar = loads.expect(2 + halo_buffer<S>(i), kHaloBytes<S>))
            na2d_ptx::tma_load_5d(smem + halo_at<S>(i), &tm_v, bar, i * kChunk, kx0, ky0, t.n, t.b);
    };
    auto load_qk = [&](int i) {
        const int stage = (n - 1 - i) & 1;
        if (uint64_t* bar = loads.expect(stage, kDotBytes<S>)) load_dot<S>(&tm_q, &tm_k, smem + stage * S::kStage, bar, i, t, ky0, kx0);
    };
    if (threadIdx.x == 0) {
        load_qk(0);
        if (n > 1) load_qk(1);
        else if (S::kHaloBuffers == 2) load_v(0);
    }
    const DotItem d = score_item<S>(t, g, ky0, kx0);
    __syncthreads();
    float s[kR][KS];
    auto next = [&](int i) {
        if (i + 2 < n) load_qk(i + 2);
        else if (S::kHaloBuffers == 2 ? i + 2 == n : i + 1 == n) load_v(0);
    };
    if (d.all_regular) tile_dot<S, PARK, true>(s, smem, loads, d, g, 0, n, next);
    else tile_dot<S, PARK, false>(s, smem, loads, d, g, 0, n, next);
    __syncthreads();

    // Softmax over the kKh threads that share a strip: row maxima and sums go through shared memory.
    const int slot = (d.strip * S::kKh + d.u) * S::kTh + d.row;
    if (d.active) {
        float m[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            m[r] = -CUDART_INF_F;
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                s[r][i] *= g.scale;
                m[r] = fmaxf(m[r], s[r][i]);
            }
        }
        mx[slot] = make_float4(m[0], m[1], m[2], m[3]);
    }
    __syncthreads();
    float4 m4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (d.active) {
        m4 = mx[d.strip * S::kKh * S::kTh + d.row];
#pragma unroll
        for (int u = 1; u < S::kKh; ++u) {
            const float4 x = mx[(d.strip * S::kKh + u) * S::kTh + d.row];
            m4 = make_float4(fmaxf(m4.x, x.x), fmaxf(m4.y, x.y), fmaxf(m4.z, x.z), fmaxf(m4.w, x.w));
        }
        float l[4][kR] = {};                                // four short sums instead of a long one
#pragma unroll
        for (int i = 0; i < KS; ++i)
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                s[r][i] = expf(s[r][i] - lane_of(m4, r));
                l[i & 3][r] += s[r][i];
            }
        store_weights<S>(weight_slots<S>(w, d), s);
        auto total = [&](int r) { return (l[0][r] + l[1][r]) + (l[2][r] + l[3][r]); };
        sum[slot] = make_float4(total(0), total(1), total(2), total(3));
    }
    __syncthreads();
    if (d.active && d.u == 0) {
        const float4 l4 = sum_rows<S>(sum + d.strip * S::kKh * S::kTh + d.row);
        const int c0 = t.x0 + kR * d.strip;
        float* dst = lse + ((long long)t.bn * g.Hq + t.y0 + d.row) * g.W + c0;
#pragma unroll
        for (int r = 0; r < kR; ++r)
            if (c0 + r < g.W) dst[r] = lane_of(m4, r) + logf(lane_of(l4, r));
    }
    const ApplyItem<S> a(t);
    float4 inv[S::kRows];
#pragma unroll
    for (int p = 0; p < S::kRows; ++p) {
        if (!a.active || a.row + p >= t.rows) break;
        const float4 l4 = sum_rows<S>(sum + a.strip * S::kKh * S::kTh + a.row + p);
        inv[p] = make_float4(1.f / l4.x, 1.f / l4.y, 1.f / l4.z, 1.f / l4.w);
    }
    // The exchange has been read, and the second halo comes in its place.  It was written with ordinary stores: each thread's fence puts
    // those before the copy that the last warp asks for.
    if (S::kHaloBuffers == 2 && g.C > kChunk) {
        na2d_ptx::fence_proxy_async();
        if (loads.last(3)) load_v(1);
    }
    tile_apply<S, S::kHaloBuffers>(o, smem, loads, w, a, inv, t, g, ky0, kx0, 0, g.C, load_v);
    loads.drain();
}

// ------------------------------------------------------------------------------------ dQ (+ delta, P, dS)
// A thread's values of one window row as the key half reads them: slot j holds the four pixels' weights for column j of the strip's
// halo band, 0 outside a window.  `own`: the thread's weight slots, which hold the values where the strip is not regular.
template <typename S>
__device__ __forceinline__ void store_band(float4* slots, const DotItem& d, const float (&s)[kR][S::kKs], const float4* own) {
    if (d.s.regular) {
        auto at = [&](int r, int j) { return j >= r && j - r < S::kKs ? s[r][j < r ? 0 : j - r >= S::kKs ? 0 : j - r] : 0.f; };
#pragma unroll
        for (int j = 0; j < S::kU; ++j) slots[j * S::kTh] = make_float4(at(0, j), at(1, j), at(2, j), at(3, j));
    } else {
        const float* p = reinterpret_cast<const float*>(own);
        auto at = [&](int r, int j) { return (unsigned)(j - d.s.off[r]) < (unsigned)S::kKs ? p[(j - d.s.off[r]) * (S::kTh * kR) + r] : 0.f; };
#pragma unroll
        for (int j = 0; j < S::kU; ++j) slots[j * S::kTh] = make_float4(at(0, j), at(1, j), at(2, j), at(3, j));
    }
}

// delta = sum_j p_j dp_j, which equals dO . o exactly and does not depend on how o was rounded when it was stored.  d_q may be null:
// then only delta (and the weights) are produced.  p_out / ds_out, both or neither: the tiles' weights for the key half (kBand
// slots each), tile after tile in the rows of `band`'s ring.  row_factor (or null): what each row's exp(s - lse) is
// multiplied by to be P.  tm_do, tm_q: the tile's own pixels, tm_v, tm_k: halo, 16 channels; tm_k32: halo, 32 channels.
template <int KS, bool PARK>
__global__ void __launch_bounds__(Shape<KS>::kThreads, Shape<KS>::kBlocks)
dq_kernel(const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_q,
          const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_k32, const __grid_constant__ Operand d_q,
          const float* __restrict__ lse, float* __restrict__ delta, float* __restrict__ row_factor, float4* __restrict__ p_out,
          float4* __restrict__ ds_out, const ErrorState* __restrict__ errors, const __grid_constant__ Band band, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS>;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (!starts_right(smem, errors)) return;
    float4 *w = reinterpret_cast<float4*>(smem + S::kWeightsAt), *part = reinterpret_cast<float4*>(smem + S::kExchangeAt), *total = part + S::kExchange / 2;
    Loads loads(smem + S::kBarriersAt, errors);
    const Tile t = tile_of_block<S>(g, g.Hq, band.unit0, band.row0, band.rows);
    int ky0, kx0;
    query_halo<S>(t, g, ky0, kx0);
    const int n = dot_chunks(g), all = 2 * n;
    auto load_k = [&](int i) {
        if (uint64_t* bar = loads.expect(2 + halo_buffer<S>(i), kHaloBytes<S>))
            na2d_ptx::tma_load_5d(smem + halo_at<S>(i), &tm_k32, bar, i * kChunk, kx0, ky0, t.n, t.b);
    };
    auto load_pair = [&](int i) {
        const int stage = (all - 1 - i) & 1;
        if (uint64_t* bar = loads.expect(stage, kDotBytes<S>)) {
            if (i < n) load_dot<S>(&tm_do, &tm_v, smem + stage * S::kStage, bar, i, t, ky0, kx0);
            else load_dot<S>(&tm_q, &tm_k, smem + stage * S::kStage, bar, i - n, t, ky0, kx0);
        }
    };
    auto next = [&](int i) {
        if (i + 2 < all) load_pair(i + 2);
        else if (d_q.ptr && (S::kHaloBuffers == 2 ? i + 2 == all : i + 1 == all)) load_k(0);
    };
    if (threadIdx.x == 0) {
        load_pair(0);
        load_pair(1);
    }
    const DotItem d = score_item<S>(t, g, ky0, kx0);
    float4* slots = weight_slots<S>(w, d);
    const int c0 = t.x0 + kR * d.strip;
    const long long stat = ((long long)t.bn * g.Hq + t.y0 + d.row) * g.W + c0;
    __syncthreads();
    float s[kR][KS];
    // dP first, parked in the thread's own weight slots, then the scores (one copy of the loop: two strain the instruction cache)
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        if (pass > 0 && d.active) store_weights<S>(slots, s);
        if (d.all_regular) tile_dot<S, PARK, true>(s, smem, loads, d, g, pass * n, all, next);
        else tile_dot<S, PARK, false>(s, smem, loads, d, g, pass * n, all, next);
    }
    __syncthreads();
    if (d.active) {
        float dl[2][kR], l[2][kR];                          // two short sums instead of a long one
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            dl[0][r] = dl[1][r] = l[0][r] = l[1][r] = 0.f;
            const float row_lse = c0 + r < g.W ? lse[stat + r] : 0.f;
#pragma unroll
            for (int i = 0; i < KS; ++i) s[r][i] = expf(s[r][i] * g.scale - row_lse);
        }
#pragma unroll
        for (int i = 0; i < KS; ++i) {
            const float4 dp = slots[i * S::kTh];
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                l[i & 1][r] += s[r][i];
                dl[i & 1][r] = fmaf(s[r][i], lane_of(dp, r), dl[i & 1][r]);
            }
        }
        const int slot = (d.strip * S::kKh + d.u) * S::kTh + d.row;
        part[slot] = make_float4(dl[0][0] + dl[1][0], dl[0][1] + dl[1][1], dl[0][2] + dl[1][2], dl[0][3] + dl[1][3]);
        total[slot] = make_float4(l[0][0] + l[1][0], l[0][1] + l[1][1], l[0][2] + l[1][2], l[0][3] + l[1][3]);
    }
    __syncthreads();
    if (d.active) {
        float4 dl4;
        const float4 l4 = sum_rows<S>(total + d.strip * S::kKh * S::kTh + d.row);
        auto factor = [&](int r) { return na2d_row_factor(lane_of(l4, r), c0 + r < g.W ? lse[stat + r] : 0.f); };
        const float4 inv = make_float4(factor(0), factor(1), factor(2), factor(3));
        dl4 = sum_rows<S>(part + d.strip * S::kKh * S::kTh + d.row);
        dl4 = make_float4(dl4.x * inv.x, dl4.y * inv.y, dl4.z * inv.z, dl4.w * inv.w);
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int i = 0; i < KS; ++i) s[r][i] *= lane_of(inv, r);
        if (d.u == 0) {
#pragma unroll
            for (int r = 0; r < kR; ++r)
                if (c0 + r < g.W) {
                    delta[stat + r] = lane_of(dl4, r);
                    if (row_factor) row_factor[stat + r] = lane_of(inv, r);
                }
        }
        // P and dS go straight to the key half, dS to the slots as well
        const long long place = (((long long)(t.bn - band.unit0) * band.ring + t.y0 / S::kTh % band.ring) *
                                     ((g.W + S::kTw - 1) / S::kTw) + t.x0 / S::kTw) * S::kBand +
                                (d.strip * S::kKh + d.u) * S::kU * S::kTh + d.row;
        float4 dp[KS];
#pragma unroll
        for (int i = 0; i < KS; ++i) dp[i] = slots[i * S::kTh];
        if (p_out) {
            if (!d.s.regular) store_weights<S>(slots, s);
            store_band<S>(p_out + place, d, s, slots);
        }
#pragma unroll
        for (int i = 0; i < KS; ++i)
#pragma unroll
            for (int r = 0; r < kR; ++r) s[r][i] = g.scale * s[r][i] * (lane_of(dp[i], r) - lane_of(dl4, r));
        store_weights<S>(slots, s);
        if (ds_out) store_band<S>(ds_out + place, d, s, slots);
    }
    if (d_q.ptr) {
        if (S::kHaloBuffers == 2 && g.C > kChunk) {                                     // the sums have been read (fwd_kernel says why the fence)
            na2d_ptx::fence_proxy_async();
            if (loads.last(3)) load_k(1);
        }
        __syncthreads();
        float4 one[S::kRows];
#pragma unroll
        for (int p = 0; p < S::kRows; ++p) one[p] = make_float4(1.f, 1.f, 1.f, 1.f);
        tile_apply<S, S::kHaloBuffers>(d_q, smem, loads, w, ApplyItem<S>(t), one, t, g, ky0, kx0, 0, g.C, load_k);
    }
    loads.drain();
}

// ------------------------------------------------------------------------------------ unfused pair
// The weights of a tile's image row are one run of t.cols * KS * KS numbers in the dense array.
template <int KS>
__device__ __forceinline__ long long dense_row(const Tile& t, const Na2dGeom& g, int row) {
    return (((long long)t.bn * g.Hq + t.y0 + row) * g.W + t.x0) * (KS * KS);
}

// Each needs a part of the fused kernels' shared memory, which leaves room for more blocks: the stages and, in their place, the tile's
// scores; a halo and the weights.
template <typename S>
struct PairShape {
    static constexpr int blocks(int smem, int threads, int registers) {
        return na2d_tile::kSmemPerSm / (smem + 1024) < 65536 / (threads * registers) ? na2d_tile::kSmemPerSm / (smem + 1024) : 65536 / (threads * registers);
    }
    static constexpr int kRow = S::kTw * S::kKs * S::kKs + 1;            // floats of an image row's scores: lanes of eight rows write at once
    static constexpr int kDotBarriersAt = max_of(2 * S::kStage, whole_kb(S::kTh * kRow * 4)), kDotSmem = kDotBarriersAt + S::kBarriers;
    static constexpr int kDotBlocks = blocks(kDotSmem, S::kThreads, 128);
    static constexpr int kApplyThreads = S::kApply;
    static constexpr int kWeightsAt = S::kHalo, kApplyBarriersAt = kWeightsAt + S::kWeights * 16, kApplySmem = kApplyBarriersAt + S::kBarriers;
    static constexpr int kApplyBlocks = blocks(kApplySmem, kApplyThreads, 128);
};

// attn[pixel, member] = x[pixel] . y[member of the pixel's window]; tm_x, tm_y: own pixels and halo, 16 channels.
template <int KS, bool PARK>
__global__ void __launch_bounds__(Shape<KS>::kThreads, PairShape<Shape<KS>>::kDotBlocks)
window_dot_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_y, float* __restrict__ attn,
                  const ErrorState* __restrict__ errors, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS>;
    constexpr int kRow = PairShape<S>::kRow;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (!starts_right(smem, errors)) return;
    Loads loads(smem + PairShape<S>::kDotBarriersAt, errors);
    const Tile t = tile_of_block<S>(g, g.Hq);
    int ky0, kx0;
    query_halo<S>(t, g, ky0, kx0);
    const int n = dot_chunks(g);
    auto load = [&](int i) {
        const int stage = (n - 1 - i) & 1;
        if (uint64_t* bar = loads.expect(stage, kDotBytes<S>)) load_dot<S>(&tm_x, &tm_y, smem + stage * S::kStage, bar, i, t, ky0, kx0);
    };
    if (threadIdx.x == 0) {
        load(0);
        if (n > 1) load(1);
    }
    const DotItem d = score_item<S>(t, g, ky0, kx0);
    __syncthreads();
    float s[kR][KS];
    auto next = [&](int i) {
        if (i + 2 < n) load(i + 2);
    };
    if (d.all_regular) tile_dot<S, PARK, true>(s, smem, loads, d, g, 0, n, next);
    else tile_dot<S, PARK, false>(s, smem, loads, d, g, 0, n, next);
    loads.drain();
    __syncthreads();
    float* rows = reinterpret_cast<float*>(smem);
    if (d.active) {
        float* p = rows + d.row * kRow + kR * d.strip * kTaps<KS> + d.u * KS;
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int m = 0; m < KS; ++m) p[r * kTaps<KS> + m] = s[r][m];
    }
    __syncthreads();
    for (int row = 0; row < t.rows; ++row) {
        float* to = attn + dense_row<KS>(t, g, row);
        for (int i = threadIdx.x; i < t.cols * kTaps<KS>; i += S::kThreads) to[i] = rows[row * kRow + i];
    }
}

// out[pixel] = sum over the window of attn[pixel, member] * y[member], `span` channels a block; tm_y: halo, 32 channels.
template <int KS>
__global__ void __launch_bounds__(PairShape<Shape<KS>>::kApplyThreads, PairShape<Shape<KS>>::kApplyBlocks)
window_apply_kernel(const float* __restrict__ attn, const __grid_constant__ CUtensorMap tm_y, const __grid_constant__ Operand out, const int span,
                    const ErrorState* __restrict__ errors, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS>;
    using P = PairShape<S>;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (!starts_right(smem, errors)) return;
    float* w = reinterpret_cast<float*>(smem + P::kWeightsAt);
    Loads loads(smem + P::kApplyBarriersAt, errors);
    const Tile t = tile_of_block<S>(g, g.Hq);
    int ky0, kx0;
    query_halo<S>(t, g, ky0, kx0);
    const int ch0 = blockIdx.z * span;
    auto load = [&](int i) {
        if (uint64_t* bar = loads.expect(2, kHaloBytes<S>)) na2d_ptx::tma_load_5d(smem, &tm_y, bar, ch0 + i * kChunk, kx0, ky0, t.n, t.b);
    };
    if (threadIdx.x == 0) load(0);
    for (int row = 0; row < t.rows; ++row) {
        const float* from = attn + dense_row<KS>(t, g, row);
        for (int i = threadIdx.x; i < t.cols * kTaps<KS>; i += P::kApplyThreads) {
            const int q = i / kTaps<KS>, tap = i - q * kTaps<KS>;
            w[((q / kR * kTaps<KS> + tap) * S::kTh + row) * kR + q % kR] = __ldg(from + i);
        }
    }
    __syncthreads();
    float4 one[S::kRows];
#pragma unroll
    for (int p = 0; p < S::kRows; ++p) one[p] = make_float4(1.f, 1.f, 1.f, 1.f);
    tile_apply<S, 1>(out, smem, loads, reinterpret_cast<const float4*>(w), ApplyItem<S>(t), one, t, g, ky0, kx0, ch0, min(g.C, ch0 + span), load);
    loads.drain();
}

}  // namespace na2d_box
