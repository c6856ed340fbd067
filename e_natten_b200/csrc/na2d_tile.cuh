// Tiled CUDA-core kernels for neighborhood attention: fused forward, the query half of the backward
// (dQ, delta, and the P / dS weights the key half reads), the unfused pair, and the key-side sum over
// the inverse neighbourhood.  fp32 arithmetic throughout; fp32, bf16 and fp16 tensors.  fp32 calls in 2D whose rows start on 16-byte
// boundaries go to na2d_box.cuh.
//
// A block owns a tile of kTh x (4 * kStrips) pixels of one (batch, head) image.  Channels pass
// through shared memory 32 at a time (always as fp32): the tile's own rows and the halo of rows its
// windows reach.  Two loops do all the work:
//   dot    a thread holds the scores of a strip of four neighbouring pixels against one window row:
//          4 own and ks + 3 halo float4 loads feed 16 * ks multiply-adds.  No cross-lane sums: a score
//          is summed by one thread (four in 1D) over all channels.
//   apply  a thread holds 4 pixels x 4 channels of an output; per window row, ks + 3 halo float4 and as
//          many weight float4 (the strip's four weights for that halo column; a broadcast to the
//          eight lanes that share the strip) feed the same 16 * ks multiply-adds.
// Both are bound by shared-memory bandwidth (a float4 load of a warp takes four cycles, in which the SM
// issues 16 warp multiply-adds): the strip is what brings the loads per multiply-add down.
//
// Measured on one B200 against one warp per pixel with the channels over its lanes (na2d_simt.cuh, four loads and a
// butterfly of shuffles per 32 products), fp32: forward 4 x 4 x 256 x 256 x 128, window 5, 3.85 -> 0.84 ms;
// 4 x 4 x 117 x 93 x 64, window 7, 0.75 -> 0.15 ms.
//
// Windows are clamped at the borders, so the four windows of a strip need not be shifted by one
// column each.  A strip away from the borders ("regular") takes loops whose band is known at compile
// time; any other takes loops that test each pair.  Pairs outside a window never enter a sum, so an
// infinity or NaN reaches only the pixels whose windows hold it.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <float.h>
#include <math_constants.h>
#include <stdint.h>

#include "na2d_index.cuh"
#include "na2d_ptx.cuh"
#include "na2d_softmax.cuh"

namespace na2d_tile {

using na2d_ptx::fma2;
using na2d_ptx::mul2;

constexpr int kR = 4;             // pixels of a strip
constexpr int kF = 8;             // float4 per pixel and channel chunk
constexpr int kChunk = 4 * kF;    // channels per chunk
constexpr int kSmemPerSm = 227 * 1024;

// Geometry of a tile for window size KS (a 1 x KS window on one-row images with ONE_D).
template <int KS, bool ONE_D>
struct Shape {
    static constexpr int kKs = KS;
    static constexpr bool kOneD = ONE_D;
    static constexpr int kKh = ONE_D ? 1 : KS;
    static constexpr int kTh = ONE_D ? 1 : 8;
    static constexpr int kStrips = ONE_D ? 32 : (KS <= 7 ? 4 : 2);
    static constexpr int kSplit = ONE_D ? 4 : 1;          // lanes that share a strip's channels in the dot loop
    static constexpr int kTw = kR * kStrips;
    static constexpr int kU = KS + kR - 1;                // halo columns a strip reaches
    static constexpr int kHaloW = kTw + KS - 1;
    static constexpr int kHaloH = kTh + kKh - 1;
    static constexpr int kItems = kTh * kStrips * kKh * kSplit;
    static constexpr int kApply = kTh * kStrips * kF;     // (strip, float4 of a chunk) items of the apply loop
    // a thread per dot item; one more warp where that takes the apply loop from two rounds to one (KS 7)
    static constexpr int kDotThreads = (kItems + 31) / 32 * 32 < 128 ? 128 : (kItems + 31) / 32 * 32;
    static constexpr int kThreads = kApply == kDotThreads + 32 ? kApply : kDotThreads;
    // shared memory, in float4
    static constexpr int kWeights = kTh * kStrips * kKh * kU;
    static constexpr int kOwn = kTh * kTw * kF;
    static constexpr int kHalo = kHaloH * kHaloW * kF;
    static constexpr int kSmem = (kWeights + kOwn + kHalo) * 16;
    static constexpr int kBlocksSmem = kSmemPerSm / (kSmem + 1024);
    static constexpr int kBlocksReg = 65536 / (kThreads * (KS >= 9 ? 144 : 128));
    static constexpr int kBlocks = kBlocksSmem < kBlocksReg ? kBlocksSmem : (kBlocksReg < 1 ? 1 : kBlocksReg);
};

struct Operand {
    void* ptr;
    Na2dStride st;
    int vec;          // rows of channels can be read four elements at a time
};

template <typename T> __device__ __forceinline__ float to_f(T x);
template <> __device__ __forceinline__ float to_f<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_f<__half>(__half x) { return __half2float(x); }
template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }

template <typename T> struct Quad;                         // four elements as one load
template <> struct Quad<float> { using type = float4; };
template <> struct Quad<__nv_bfloat16> { using type = uint2; };
template <> struct Quad<__half> { using type = uint2; };

__device__ __forceinline__ float4 widen(float4 x, float) { return x; }
__device__ __forceinline__ float4 widen(uint2 x, __nv_bfloat16) {
    return make_float4(__uint_as_float(x.x << 16), __uint_as_float(x.x & 0xffff0000u), __uint_as_float(x.y << 16),
                       __uint_as_float(x.y & 0xffff0000u));
}
__device__ __forceinline__ float4 widen(uint2 x, __half) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&x.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&x.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store_quad(float* p, float4 x) { *reinterpret_cast<float4*>(p) = x; }
__device__ __forceinline__ void store_quad(__nv_bfloat16* p, float4 x) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
    *reinterpret_cast<uint2*>(p) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ void store_quad(__half* p, float4 x) {
    const __half2 a = __floats2half2_rn(x.x, x.y), b = __floats2half2_rn(x.z, x.w);
    *reinterpret_cast<uint2*>(p) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
template <typename T>
__device__ __forceinline__ void store_channels(T* row, float4 x, int c, int C, bool vec) {
    if (vec) {
        if (c < C) store_quad(row + c, x);
    } else {
        const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (c + e < C) row[c + e] = from_f<T>(v[e]);
    }
}

__device__ __forceinline__ void copy16(float4* dst, const void* src, bool take) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = take ? 16 : 0;                       // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Where float4 f of staged pixel (y, x) lies, counted from the pixel's first float4: the eight lanes of a quarter
// warp read the same f of eight rows (or, for one-row tiles, of eight strips) in the dot loop, and the exclusive
// or puts those on different banks.  With eight-row tiles it does not depend on the column.
template <int TH>
__device__ __forceinline__ int place_of(int f, int y, int x) {
    static_assert(TH == 1 || TH == 8, "eight rows, or one");
    if constexpr (TH == 8) return f ^ (y & 7);
    else return f ^ ((y + (x >> 2)) & 7);
}

// Four channels from c on of the pixel at p, as fp32, to d; zeros unless `in`, and beyond channel C.  p is
// readable either way.
template <typename T>
__device__ __forceinline__ void stage_quad(float4* d, const T* p, bool in, int c, int C, bool vec) {
    if (vec) {
        if constexpr (sizeof(T) == 4) {
            copy16(d, p, in);
        } else {
            // p can be read in any case: a load without a branch, so that those of an unrolled loop fly together
            const float4 x = widen(__ldg(reinterpret_cast<const typename Quad<T>::type*>(p)), T{});
            *d = in ? x : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = in && c + e < C ? to_f<T>(p[e]) : 0.f;
        *d = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// Stages channels [c0, c0 + 32) of pixels (y0 + y, x0 + x), y < rows, x < COLS, of the image at `src`.
// Rows y0 .. y0 + rows - 1 exist; columns at or beyond W and channels at or beyond C become zeros.  A thread keeps
// its channels and, where a pass of the block covers whole rows, its column: what is left per pixel is an
// addition to each address.
template <typename T, int TH, int THREADS, int COLS>
__device__ __forceinline__ void stage(float4* dst, const T* src, const Na2dStride& st, int y0, int rows, int x0, int W,
                                      int c0, int C, bool vec) {
    constexpr int kPx = THREADS / kF;
    const int f = threadIdx.x % kF, px = threadIdx.x / kF, c = c0 + 4 * f;
    if constexpr (kPx >= COLS) {
        constexpr int kRows = kPx / COLS;                  // rows per pass
        const int yy = px / COLS, x = px - yy * COLS;
        if (yy >= kRows) return;
        const bool in = x0 + x < W && c < C;
        const T* p = in ? src + (y0 + yy) * st.h + (x0 + x) * st.w + c : src;
        const long long step = in ? kRows * st.h : 0;
        float4* d = dst + (yy * COLS + x) * kF;
#pragma unroll (sizeof(T) == 2 ? 8 : 4)
        for (int y = yy; y < rows; y += kRows) {
            stage_quad<T>(d + place_of<TH>(f, y, x), p, in, c, C, vec);
            p += step;
            d += kRows * COLS * kF;
        }
    } else {
        for (int y = 0; y < rows; ++y) {
            const T* p = src + (y0 + y) * st.h + (x0 + px) * st.w + c;
            auto one = [&](int x) {
                const bool in = x0 + x < W && c < C;
                stage_quad<T>(dst + (y * COLS + x) * kF + place_of<TH>(f, y, x), in ? p : src, in, c, C, vec);
                p += kPx * st.w;
            };
#pragma unroll
            for (int i = 0; i < COLS / kPx; ++i) one(px + i * kPx);
            if (COLS % kPx != 0 && px < COLS % kPx) one(px + COLS / kPx * kPx);
        }
    }
}

// The tiles of a launch: tile rows [row0, row0 + rows) of each unit from `unit0` on.  `ring`: tile rows of a unit that the
// weights handed from the query half to the key half have room for; row r lies in place r % ring.
struct Band {
    int unit0, row0, rows, ring;
};

// Tile of this block in a (BN, H, W) grid of pixels.
struct Tile {
    int bn, b, n, y0, x0, rows, cols;
};
template <typename S>
__device__ __forceinline__ Tile tile_of_block(const Na2dGeom& g, int H, int unit0, unsigned row0, unsigned th) {
    const unsigned tw = (unsigned)(g.W + S::kTw - 1) / S::kTw;
    unsigned blk = blockIdx.x;
    Tile t;
    t.x0 = (int)(blk % tw) * S::kTw;
    blk /= tw;
    t.y0 = (int)(row0 + blk % th) * S::kTh;
    t.bn = unit0 + (int)(blk / th);
    t.b = t.bn / g.N;
    t.n = t.bn - t.b * g.N;
    t.rows = min(S::kTh, H - t.y0);
    t.cols = min(S::kTw, g.W - t.x0);
    return t;
}
template <typename S>
__device__ __forceinline__ Tile tile_of_block(const Na2dGeom& g, int H) {
    return tile_of_block<S>(g, H, 0, 0, (unsigned)(H + S::kTh - 1) / S::kTh);
}
template <typename T>
__device__ __forceinline__ T* unit(const Operand& o, const Tile& t) {
    return static_cast<T*>(o.ptr) + t.b * o.st.b + t.n * o.st.n;
}

// The windows of a strip of four query columns starting at c0: column r's window covers halo columns
// [off[r], off[r] + KS) counted from `start`, the window start of column c0.  A column outside the
// image gets an offset that no halo column reaches.
struct Strip {
    int start, off[kR];
    bool regular;
};
template <int KS>
__device__ __forceinline__ Strip strip_at(int c0, int W) {
    Strip s;
    s.start = na2d_ws(min(c0, W - 1), W, KS);
#pragma unroll
    for (int r = 0; r < kR; ++r) s.off[r] = c0 + r < W ? na2d_ws(c0 + r, W, KS) - s.start : 1 << 20;
    s.regular = c0 >= KS / 2 && c0 + kR - 1 + KS / 2 < W;
    return s;
}
template <int KS>
__device__ __forceinline__ bool in_window(const Strip& s, int r, int j) { return (unsigned)(j - s.off[r]) < (unsigned)KS; }

// Sum of the two fp32 lanes of a register pair.
__device__ __forceinline__ float sum2(unsigned long long a) {
    return __uint_as_float((unsigned)a) + __uint_as_float((unsigned)(a >> 32));
}

// Scores of a thread over the channels so far, parked in its local memory (PARK kernels).  A running sum over all C
// channels would round at every step at its full size: 1.25 times the error of a sum over the lanes of a warp
// (na2d_simt.cuh) at C = 128, 1.44 times at 256.  Instead the registers sum at most 32 channels (64 where a strip's channels
// lie over four threads); their sum then joins the parked one, and what that addition rounds off starts the next.  Error
// on normal rows against the lanes' sum: at most 0.99 times up to C = 96, 0.95 at 128, 0.86 at 256.  Registers or shared
// memory for both sums would take a block per SM.  In local memory they cost 4 to 12 % of a kernel's time, in tensor
// memory (allocated and freed by every block) 7 to 20 %.
// Where the lines lie: up to 32 channels (64 with four threads to a strip) the running sum rounds no more than the
// lanes' sum, 0.96 (0.99) times, and the kernels without parking are 1 to 5 % (8 to 11 %) faster there.
template <typename S>
constexpr int kParkAbove = S::kSplit > 1 ? 2 * kChunk : kChunk;
template <typename S, bool REGULAR>
__device__ __forceinline__ float& score(float (&acc)[kR][S::kU], int i) {      // a regular strip has a band of them
    return REGULAR ? acc[i / S::kKs][i / S::kKs + i % S::kKs] : acc[i / S::kU][i % S::kU];
}
template <typename S, bool REGULAR>
constexpr int kScores = kR * (REGULAR ? S::kKs : S::kU);
template <typename S, bool REGULAR>
__device__ __forceinline__ void park(float (&acc)[kR][S::kU], float4* parked, bool first) {
#pragma unroll
    for (int i = 0; i < kScores<S, REGULAR>; i += 4) {
        const float4 old = first ? make_float4(0.f, 0.f, 0.f, 0.f) : parked[i / 4];
        float sum[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float& a = score<S, REGULAR>(acc, i + e);
            const float total = __fadd_rn(sum[e], a);
            a = fabsf(total) <= FLT_MAX ? __fsub_rn(a, __fsub_rn(total, sum[e])) : 0.f;      // an infinite sum stays one
            sum[e] = total;
        }
        parked[i / 4] = make_float4(sum[0], sum[1], sum[2], sum[3]);
    }
}
template <typename S, bool REGULAR>
__device__ __forceinline__ void unpark(float (&acc)[kR][S::kU], const float4* parked) {
#pragma unroll
    for (int i = 0; i < kScores<S, REGULAR>; i += 4) {
        const float4 sum = parked[i / 4];
        score<S, REGULAR>(acc, i) += sum.x;
        score<S, REGULAR>(acc, i + 1) += sum.y;
        score<S, REGULAR>(acc, i + 2) += sum.z;
        score<S, REGULAR>(acc, i + 3) += sum.w;
    }
}
// Steps (of eight channels) of the chunk at channel c0 after which a PARK kernel parks, 0 for none: as few times as the error
// allows.  Up to 64 channels that is the middle of each chunk, since 16 + 32 + 16 round less than 32 + 32, beyond
// that its end; where a strip's channels lie over four threads, every other chunk from 128 on.
template <typename S>
constexpr int kSteps = kF / 2 / S::kSplit;
template <typename S>
__device__ __forceinline__ int park_after(int c0, int C) {
    if (C <= 2 * kChunk) return c0 + kChunk / 2 < C ? kSteps<S> / 2 : 0;
    const bool every = S::kSplit == 1 || C < 4 * kChunk;
    return c0 + kChunk < C && (every || c0 % (2 * kChunk) != 0) ? kSteps<S> : 0;
}

// acc[r][j] += own pixel r . halo column j over one staged chunk, eight channels at a time: their products are
// summed in packed pairs first and join acc as one number: six instructions where eight multiply-adds would stand, and
// one rounding of acc.
template <typename S, bool REGULAR, bool PARK>
__device__ __forceinline__ void dot_chunk(float (&acc)[kR][S::kU], const float4* own, int row, int strip,
                                          const float4* halo, int hy, int hx, int split, float4* parked, int park_at,
                                          bool first) {
    const ulonglong2* own2 = reinterpret_cast<const ulonglong2*>(own);
    const ulonglong2* halo2 = reinterpret_cast<const ulonglong2*>(halo);
#pragma unroll 1
    for (int i = 0; i < kSteps<S>; ++i) {
        const int f = 2 * (split * kSteps<S> + i);
        ulonglong2 q0[kR], q1[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            q0[r] = own2[r * kF + place_of<S::kTh>(f, row, kR * strip)];
            q1[r] = own2[r * kF + place_of<S::kTh>(f + 1, row, kR * strip)];
        }
#pragma unroll
        for (int j = 0; j < S::kU; ++j) {
            const ulonglong2 x0 = halo2[j * kF + place_of<S::kTh>(f, hy, hx + j)];
            const ulonglong2 x1 = halo2[j * kF + place_of<S::kTh>(f + 1, hy, hx + j)];
            unsigned long long part[kR];
#pragma unroll
            for (int r = 0; r < kR; ++r) part[r] = mul2(q0[r].x, x0.x);
#pragma unroll
            for (int r = 0; r < kR; ++r) part[r] = fma2(q0[r].y, x0.y, part[r]);
#pragma unroll
            for (int r = 0; r < kR; ++r) part[r] = fma2(q1[r].x, x1.x, part[r]);
#pragma unroll
            for (int r = 0; r < kR; ++r) part[r] = fma2(q1[r].y, x1.y, part[r]);
#pragma unroll
            for (int r = 0; r < kR; ++r)
                if (!REGULAR || (j >= r && j - r < S::kKs)) acc[r][j] += sum2(part[r]);
        }
        if (PARK && S::kSplit == 1 && i + 1 == park_at) park<S, REGULAR>(acc, parked, first);
    }
    if (PARK && S::kSplit > 1 && park_at != 0) park<S, REGULAR>(acc, parked, first);
}

// What a thread does in the dot loop: window row u of the strip `strip` of tile row `row`.
struct DotItem {
    int row, u, strip, split;
    bool active;
    int hy, hx;                   // first halo pixel
    Strip s;
};
// ky0, kx0: local row and column of halo pixel (0, 0).
template <typename S>
__device__ __forceinline__ DotItem dot_item(const Tile& t, const Na2dGeom& g, int ky0, int kx0) {
    DotItem d;
    int it = threadIdx.x;
    d.split = it % S::kSplit;
    it /= S::kSplit;
    d.row = it % S::kTh;
    it /= S::kTh;
    d.u = it % S::kKh;
    d.strip = it / S::kKh;
    d.active = threadIdx.x < S::kItems && d.row < t.rows && kR * d.strip < t.cols;
    if (!d.active) { d.row = 0; d.u = 0; d.strip = 0; }
    d.s = strip_at<S::kKs>(t.x0 + kR * d.strip, g.W);
    d.hy = na2d_ws(g.q_row0 + t.y0 + d.row, g.Hg, S::kKh) - g.kv_row0 - ky0 + d.u;
    d.hx = d.s.start - kx0;
    return d;
}
template <typename S>
__device__ __forceinline__ float4* weight_slots(float4* w, const DotItem& d) {
    return w + (d.strip * S::kKh + d.u) * S::kU * S::kTh + d.row;       // column j at [j * kTh]
}

// Scores of the whole tile: own tensor x (tile pixels) against tensor y (halo), all channel chunks.
// Ends with the halo holding y's last chunk and every thread past its reads.
template <typename T, typename S, bool PARK>
__device__ __forceinline__ void tile_dot(float (&acc)[kR][S::kU], const Operand& x, const Operand& y, float4* own,
                                         float4* halo, const Tile& t, const DotItem& d, const Na2dGeom& g, int ky0,
                                         int kx0, int halo_rows) {
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
        for (int j = 0; j < S::kU; ++j) acc[r][j] = 0.f;
    const T* xs = unit<T>(x, t);
    const T* ys = unit<T>(y, t);
    const float4* own_px = own + (d.row * S::kTw + kR * d.strip) * kF;
    const float4* halo_px = halo + (d.hy * S::kHaloW + d.hx) * kF;
    float4 local[PARK ? S::kU : 1];
    float4* parked = local;
    if constexpr (PARK) asm volatile("" : "+l"(parked));    // not in registers: those are needed for the loop
    bool first = true;
    for (int c0 = 0; c0 < g.C; c0 += kChunk) {
        stage<T, S::kTh, S::kThreads, S::kTw>(own, xs, x.st, t.y0, t.rows, t.x0, g.W, c0, g.C, x.vec);
        stage<T, S::kTh, S::kThreads, S::kHaloW>(halo, ys, y.st, ky0, halo_rows, kx0, g.W, c0, g.C, y.vec);
        copies_done();
        __syncthreads();
        if (d.active) {
            const int park_at = PARK ? park_after<S>(c0, g.C) : 0;
            if (d.s.regular) dot_chunk<S, true, PARK>(acc, own_px, d.row, d.strip, halo_px, d.hy, d.hx, d.split, parked, park_at, first);
            else dot_chunk<S, false, PARK>(acc, own_px, d.row, d.strip, halo_px, d.hy, d.hx, d.split, parked, park_at, first);
            first = first && park_at == 0;
        }
        __syncthreads();
    }
    if (PARK && !first) {
        if (d.s.regular) unpark<S, true>(acc, parked);
        else unpark<S, false>(acc, parked);
    }
    if constexpr (S::kSplit > 1) {
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int j = 0; j < S::kU; ++j)
#pragma unroll
                for (int m = 1; m < S::kSplit; m <<= 1) acc[r][j] += __shfl_xor_sync(0xffffffffu, acc[r][j], m);
    }
}

__device__ __forceinline__ void add_scaled(float4& acc, float w, float4 x) {
    acc.x = fmaf(w, x.x, acc.x);
    acc.y = fmaf(w, x.y, acc.y);
    acc.z = fmaf(w, x.z, acc.z);
    acc.w = fmaf(w, x.w, acc.w);
}
__device__ __forceinline__ float lane_of(const float4& v, int r) { return r == 0 ? v.x : r == 1 ? v.y : r == 2 ? v.z : v.w; }

// acc[r] += sum over halo columns of one window row; `w` column j at [j * kTh].
template <typename S, bool REGULAR>
__device__ __forceinline__ void apply_row(float4 (&acc)[kR], const float4* w, const float4* halo, int f, int hy, int hx,
                                          const Strip& s) {
#pragma unroll
    for (int j = 0; j < S::kU; ++j) {
        const float4 x = halo[j * kF + place_of<S::kTh>(f, hy, hx + j)];
        const float4 wt = w[j * S::kTh];
#pragma unroll
        for (int r = 0; r < kR; ++r)
            if (REGULAR ? (j >= r && j - r < S::kKs) : in_window<S::kKs>(s, r, j)) add_scaled(acc[r], lane_of(wt, r), x);
    }
}

// The window's rows, odd and even ones in sums of their own: two short sums round less than a long one.
template <typename S, bool REGULAR>
__device__ __forceinline__ void apply_rows(float4 (&acc)[kR], const float4* w, const float4* halo, int f, int hy, int hx,
                                           const Strip& s) {
    float4 odd[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) odd[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int kW = S::kU * S::kTh, kH = S::kHaloW * kF;
#pragma unroll 1
    for (int u = 0; u + 1 < S::kKh; u += 2) {
        apply_row<S, REGULAR>(acc, w + u * kW, halo + u * kH, f, hy + u, hx, s);
        apply_row<S, REGULAR>(odd, w + (u + 1) * kW, halo + (u + 1) * kH, f, hy + u + 1, hx, s);
    }
    apply_row<S, REGULAR>(acc, w + (S::kKh - 1) * kW, halo + (S::kKh - 1) * kH, f, hy + S::kKh - 1, hx, s);
#pragma unroll
    for (int r = 0; r < kR; ++r)
        acc[r] = make_float4(acc[r].x + odd[r].x, acc[r].y + odd[r].y, acc[r].z + odd[r].z, acc[r].w + odd[r].w);
}

// out = sum over the window of weight * y: all channel chunks, last chunk first (it may be in the halo
// already: `staged`).  inv: per-pixel factors (float4 over a strip's pixels at [strip * kTh + row]) or null.
template <typename T, typename S>
__device__ __forceinline__ void tile_apply(const Operand& out, const Operand& y, const float4* w, const float4* inv,
                                           float4* halo, const Tile& t, const Na2dGeom& g, int ky0, int kx0,
                                           int halo_rows, bool staged) {
    const T* ys = unit<T>(y, t);
    T* os = unit<T>(out, t);
    for (int c0 = (g.C - 1) / kChunk * kChunk; c0 >= 0; c0 -= kChunk) {
        if (!staged) {
            __syncthreads();
            stage<T, S::kTh, S::kThreads, S::kHaloW>(halo, ys, y.st, ky0, halo_rows, kx0, g.W, c0, g.C, y.vec);
            copies_done();
        }
        staged = false;
        __syncthreads();
        for (int it = threadIdx.x; it < S::kApply; it += S::kThreads) {
            const int f = it % kF, row = it / kF % S::kTh, strip = it / (kF * S::kTh);
            if (row >= t.rows || kR * strip >= t.cols) continue;
            const Strip s = strip_at<S::kKs>(t.x0 + kR * strip, g.W);
            const int hx = s.start - kx0;
            const int hy0 = na2d_ws(g.q_row0 + t.y0 + row, g.Hg, S::kKh) - g.kv_row0 - ky0;
            float4 acc[kR];
#pragma unroll
            for (int r = 0; r < kR; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4* wr = w + strip * S::kKh * S::kU * S::kTh + row;
            const float4* hr = halo + (hy0 * S::kHaloW + hx) * kF;
            if (s.regular) apply_rows<S, true>(acc, wr, hr, f, hy0, hx, s);
            else apply_rows<S, false>(acc, wr, hr, f, hy0, hx, s);
            const float4 fac = inv ? inv[strip * S::kTh + row] : make_float4(1.f, 1.f, 1.f, 1.f);
            T* o = os + (t.y0 + row) * out.st.h + (t.x0 + kR * strip) * out.st.w;
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                const float m = lane_of(fac, r);
                if (t.x0 + kR * strip + r < g.W)
                    store_channels<T>(o + r * out.st.w, make_float4(acc[r].x * m, acc[r].y * m, acc[r].z * m, acc[r].w * m),
                                      c0 + 4 * f, g.C, out.vec);
            }
        }
    }
}

// Calls f(index into a dense (units, H, W, kh * ks) array that starts at unit `unit0`, index into the tile's weights as floats)
// for every weight of the tile: a warp takes a query, its lanes neighbouring window members.
template <typename S, typename F>
__device__ __forceinline__ void for_each_weight(const Tile& t, const Na2dGeom& g, int unit0, F&& f) {
    constexpr int kTaps = S::kKh * S::kKs, kWarps = S::kThreads / 32, kPerLane = (kTaps + 31) / 32;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    int slot[kPerLane];
#pragma unroll
    for (int e = 0; e < kPerLane; ++e) {
        const int tap = lane + 32 * e, u = tap / S::kKs;
        slot[e] = (u * S::kU + tap - u * S::kKs) * S::kTh * kR;
    }
    for (int i = warp; i < t.rows * S::kTw; i += kWarps) {
        const int row = i / S::kTw, q = i % S::kTw, strip = q / kR;
        if (q >= t.cols) continue;
        const int off = na2d_ws(t.x0 + q, g.W, S::kKs) - na2d_ws(t.x0 + kR * strip, g.W, S::kKs);
        const int at = ((strip * S::kKh * S::kU + off) * S::kTh + row) * kR + q % kR;
        const long long base = (((long long)(t.bn - unit0) * g.Hq + t.y0 + row) * g.W + t.x0 + q) * kTaps + lane;
#pragma unroll
        for (int e = 0; e < kPerLane; ++e)
            if (lane + 32 * e < kTaps) f(base + 32 * e, at + slot[e]);
    }
}

// Sum of a strip's per-window-row values, in four partial sums.
template <typename S>
__device__ __forceinline__ float4 sum_rows(const float4* v) {
    float4 s[4] = {};
    auto add = [](float4 a, float4 x) { return make_float4(a.x + x.x, a.y + x.y, a.z + x.z, a.w + x.w); };
#pragma unroll
    for (int u = 0; u < S::kKh; ++u) s[u & 3] = add(s[u & 3], v[u * S::kTh]);
    return add(add(s[0], s[1]), add(s[2], s[3]));
}

// Rows and columns of the halo of a tile of queries.
template <typename S>
__device__ __forceinline__ void query_halo(const Tile& t, const Na2dGeom& g, int& ky0, int& kx0, int& rows) {
    ky0 = na2d_ws(g.q_row0 + t.y0, g.Hg, S::kKh) - g.kv_row0;
    rows = na2d_ws(g.q_row0 + t.y0 + t.rows - 1, g.Hg, S::kKh) + S::kKh - g.kv_row0 - ky0;
    kx0 = na2d_ws(t.x0, g.W, S::kKs);
}

// ------------------------------------------------------------------------------------ forward
template <typename T, int KS, bool ONE_D, bool PARK>
__global__ void __launch_bounds__(Shape<KS, ONE_D>::kThreads, Shape<KS, ONE_D>::kBlocks)
fwd_kernel(const __grid_constant__ Operand q, const __grid_constant__ Operand k, const __grid_constant__ Operand v,
           const __grid_constant__ Operand o, float* __restrict__ lse, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS, ONE_D>;
    extern __shared__ float4 smem[];
    float4 *w = smem, *own = w + S::kWeights, *halo = own + S::kOwn;
    const Tile t = tile_of_block<S>(g, g.Hq);
    int ky0, kx0, halo_rows;
    query_halo<S>(t, g, ky0, kx0, halo_rows);
    const DotItem d = dot_item<S>(t, g, ky0, kx0);
    float s[kR][S::kU];
    tile_dot<T, S, PARK>(s, q, k, own, halo, t, d, g, ky0, kx0, halo_rows);

    // Softmax over the kKh threads that share a strip, through the own-pixel buffer: row maxima and sums.
    float4 *mx = own, *sum = own + S::kTh * S::kStrips * S::kKh, *inv = sum + S::kTh * S::kStrips * S::kKh;
    const int slot = (d.strip * S::kKh + d.u) * S::kTh + d.row;
    if (d.active) {
        float m[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            m[r] = -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < S::kU; ++j) {
                s[r][j] *= g.scale;
                if (in_window<KS>(d.s, r, j)) m[r] = fmaxf(m[r], s[r][j]);
            }
        }
        if (d.split == 0) mx[slot] = make_float4(m[0], m[1], m[2], m[3]);
    }
    __syncthreads();
    float4 m4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (d.active) {
        m4 = mx[d.strip * S::kKh * S::kTh + d.row];
        for (int u = 1; u < S::kKh; ++u) {
            const float4 x = mx[(d.strip * S::kKh + u) * S::kTh + d.row];
            m4 = make_float4(fmaxf(m4.x, x.x), fmaxf(m4.y, x.y), fmaxf(m4.z, x.z), fmaxf(m4.w, x.w));
        }
        float l[4][kR] = {};                                // four short sums instead of a long one
        float4* slots = weight_slots<S>(w, d);
#pragma unroll
        for (int j = 0; j < S::kU; ++j) {
            float e[kR];
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                e[r] = in_window<KS>(d.s, r, j) ? expf(s[r][j] - lane_of(m4, r)) : 0.f;
                l[j & 3][r] += e[r];
            }
            if (j % S::kSplit == d.split) slots[j * S::kTh] = make_float4(e[0], e[1], e[2], e[3]);
        }
        auto total = [&](int r) { return (l[0][r] + l[1][r]) + (l[2][r] + l[3][r]); };
        if (d.split == 0) sum[slot] = make_float4(total(0), total(1), total(2), total(3));
    }
    __syncthreads();
    if (d.active && d.u == 0 && d.split == 0) {
        const float4 l4 = sum_rows<S>(sum + d.strip * S::kKh * S::kTh + d.row);
        inv[d.strip * S::kTh + d.row] = make_float4(1.f / l4.x, 1.f / l4.y, 1.f / l4.z, 1.f / l4.w);
        const int c0 = t.x0 + kR * d.strip;
        float* dst = lse + ((long long)t.bn * g.Hq + t.y0 + d.row) * g.W + c0;
#pragma unroll
        for (int r = 0; r < kR; ++r)
            if (c0 + r < g.W) dst[r] = lane_of(m4, r) + logf(lane_of(l4, r));
    }
    tile_apply<T, S>(o, v, w, inv, halo, t, g, ky0, kx0, halo_rows, false);
}

}  // namespace na2d_tile
