// CUDA-core kernels of the 1D operator (a 1 x KS window on one-row images) for rows of whole 16-byte pieces, at most 256 bytes
// long: fused forward, the query half of the backward (dQ, delta, and the P / dS weights the key half reads), and the key half.
// fp32 arithmetic throughout; fp32, bf16 and fp16 tensors.
//
// A block owns kTile tokens of one (batch, head) sequence.  The rows its windows reach lie in shared memory as they come,
// all channels, copied asynchronously in one go.  A strip of four neighbouring tokens belongs to four neighbouring lanes,
// which share its channels, 16-byte pieces in turn: a lane keeps its part of the strip's 4 x (KS + 3) scores in registers, a
// halo piece is read once for four tokens, and a transposing butterfly (3 (KS + 3) shuffles) leaves each lane the whole
// scores of one token.  Softmax, delta and dS of a token are then one lane's, without a barrier or an exchange; its weights go
// through shared memory to the strip's other lanes, which all are in the same warp.  The only block barriers are those behind the
// copies: two in the forward and the query half, whose halos are waited for one by one, one in the key half.
//
// What bounds them: issue slots of the two (query half: three) loops, and the latency of the copies, of which the blocks of an SM
// overlap: three or four at rows of up to 128 bytes, two at 256 bytes from window 5 on, where shared memory holds no more (the register
// bounds below are for the shorter rows; 16-bit rows spill up to 130 bytes a thread under them at window 13).
// The tiled kernels (na2d_tile.cuh) stage 32 channels at a time as fp32 with two barriers each, and repeat a strip's
// softmax on all of its lanes.  Measured against those on one B200: 4 x 8 x 4096 x 64, window 13,
// bf16: forward 70 -> 29 us, both halves of the backward 195 -> 84; 4 x 4 x 32768 x 128, window 7, bf16: 393 -> 153, 859 -> 337;
// 4 x 8 x 4096 x 32, window 13, fp32: 33 -> 23, 101 -> 64.
//
// Windows are clamped at the borders; a strip away from them ("regular") takes loops whose band is known at compile time, any other
// takes loops that test each pair.  Pairs outside a window never enter a sum.
#pragma once

#include "na2d_ptx.cuh"
#include "na2d_tile_bwd.cuh"

namespace na2d_line {

using na2d_ptx::add2;
using na2d_ptx::fma2;
using na2d_ptx::hi2;
using na2d_ptx::lo2;
using na2d_ptx::mul2;
using na2d_ptx::pair2;
using na2d_tile::kR;
using na2d_tile::Operand;

constexpr int kTile = 128, kStrips = kTile / kR, kLanes = 4, kThreads = kStrips * kLanes;
// Bytes of a row at most.  fp32 rows of 256 bytes are no faster here than in the tiled kernels (4 x 8 x 4096 x 64, window 3 / 7:
// forward 37 / 43 against 33 / 38 us, window 13 50 against 54), of 192 bytes they are (window 7 29 against 35 us, window 13 35
// against 52).  16-bit rows gain throughout, and would beyond this line too: 8 x 16384 tokens, window 7, 272 bytes forward 149 -> 59 and
// backward 308 -> 128 us, 336 bytes 183 -> 70 and 377 -> 148 (window 13 at 336 bytes 278 -> 82 and 560 -> 262); two blocks fit an SM there.
constexpr int max_row(int element_bytes) { return element_bytes == 4 ? 192 : 256; }

template <int KS> constexpr int kU = KS + kR - 1;     // halo rows a regular strip reaches
template <int KS> constexpr int kRows = kTile + KS - 1 + kR - 1;      // halo rows of a tile, and what strips at its end may touch
template <int KS> constexpr int kSlots = kU<KS> * kR + kR;            // floats of a strip's weights, padded against bank conflicts
// Query rows that the keys of a tile meet at most: a key within KS of a border is seen by up to KS / 2 more.
template <int KS> constexpr int kKeyRows = kTile + KS + KS / 2;
// Query rows that four neighbouring keys meet at most: all of a sequence whose ends both are within KS of them.
template <int KS> constexpr int kMet = 2 * KS + kR - 2;

// 16-byte pieces of a row in shared memory: an odd number, which puts the two strips of a quarter warp on different banks.
__host__ __device__ constexpr int pitch_of(int row_bytes) { return row_bytes / 16 | 1; }
template <int KS> constexpr int forward_smem(int row_bytes) { return (2 * kRows<KS> * pitch_of(row_bytes) + kStrips * kSlots<KS> / 4) * 16; }
template <int KS> constexpr int key_smem(int row_bytes) { return (2 * kKeyRows<KS> * pitch_of(row_bytes) + 2 * kStrips * (kMet<KS> + 1)) * 16; }

// A piece as fp32 pairs.
template <typename T> struct Pairs { static constexpr int N = 8 / sizeof(T); };
__device__ __forceinline__ void unpack(uint4 x, uint64_t (&p)[2], float) {
    p[0] = pair2(x.x, x.y);
    p[1] = pair2(x.z, x.w);
}
__device__ __forceinline__ uint64_t unpack_pair(uint32_t w, __nv_bfloat16) { return pair2(w << 16, w & 0xffff0000u); }
__device__ __forceinline__ uint64_t unpack_pair(uint32_t w, __half) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    return pair2(f.x, f.y);
}
template <typename T>
__device__ __forceinline__ void unpack(uint4 x, uint64_t (&p)[4], T) {
    p[0] = unpack_pair(x.x, T{});
    p[1] = unpack_pair(x.y, T{});
    p[2] = unpack_pair(x.z, T{});
    p[3] = unpack_pair(x.w, T{});
}
__device__ __forceinline__ uint4 pack(const uint64_t (&p)[2], float) {
    return make_uint4((uint32_t)p[0], (uint32_t)(p[0] >> 32), (uint32_t)p[1], (uint32_t)(p[1] >> 32));
}
__device__ __forceinline__ uint32_t pack_pair(uint64_t p, __nv_bfloat16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo2(p), hi2(p));
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_pair(uint64_t p, __half) {
    const __half2 h = __floats2half2_rn(lo2(p), hi2(p));
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <typename T>
__device__ __forceinline__ uint4 pack(const uint64_t (&p)[4], T) {
    return make_uint4(pack_pair(p[0], T{}), pack_pair(p[1], T{}), pack_pair(p[2], T{}), pack_pair(p[3], T{}));
}

// Where a thread works: sequence, tile, strip and lane of the strip.
struct Place {
    int bn, b, n, x0, strip, lane, t0;           // t0: the strip's first token
};
__device__ __forceinline__ Place place_of_block(const Na2dGeom& g, int unit0) {
    const unsigned tiles = (unsigned)(g.W + kTile - 1) / kTile;
    Place p;
    p.bn = unit0 + (int)(blockIdx.x / tiles);
    p.x0 = (int)(blockIdx.x % tiles) * kTile;
    p.b = p.bn / g.N;
    p.n = p.bn - p.b * g.N;
    p.strip = threadIdx.x / kLanes;
    p.lane = threadIdx.x % kLanes;
    p.t0 = p.x0 + kR * p.strip;
    return p;
}
template <typename T>
__device__ __forceinline__ T* sequence(const Operand& o, const Place& p) {
    return static_cast<T*>(o.ptr) + p.b * o.st.b + p.n * o.st.n;
}

// Copies rows [first, first + rows) of N sequences, all of them inside, to shared memory.  A thread's next piece lies kThreads pieces on; it
// steps there by rows and pieces, so that it divides once: with a division for each piece copying was a tenth of the forward at window 3
// (4 x 8 x 4096 x 64, bf16, window 3 / 13: forward 16.4 / 30.8 -> 15.1 / 28.9 us, dQ alone 21.8 / 45.4 -> 20.5 / 43.3).
template <typename T, int N>
__device__ __forceinline__ void copy_rows(uint4* const (&dst)[N], const T* const (&src)[N], const Na2dStride* const (&st)[N], int first, int rows,
                                          int pieces, int pitch) {
    constexpr int kN = 16 / sizeof(T);
    const int down = kThreads / pieces, across = kThreads - down * pieces;
    int row = (int)threadIdx.x / pieces, piece = (int)threadIdx.x - row * pieces, to = row * pitch + piece;
    const T* from[N];
#pragma unroll
    for (int i = 0; i < N; ++i) from[i] = src[i] + (long long)(first + row) * st[i]->w + piece * kN;
    while (row < rows) {
        row += down;
        piece += across;
        const bool wrap = piece >= pieces;
        if (wrap) piece -= pieces, ++row;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            na2d_tile::copy16(reinterpret_cast<float4*>(dst[i]) + to, from[i], true);
            from[i] += (long long)down * st[i]->w + across * kN;
            if (wrap) from[i] += st[i]->w - pieces * kN;
        }
        to += down * pitch + across + (wrap ? pitch - pieces : 0);
    }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void arrived() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One piece of each of a strip's four rows, as it lies in global memory.
template <typename T>
__device__ __forceinline__ void load_strip(uint4 (&raw)[kR], const T* x, const Na2dStride& st, int t0, int W, int piece) {
#pragma unroll
    for (int r = 0; r < kR; ++r)
        raw[r] = __ldg(reinterpret_cast<const uint4*>(x + (long long)min(t0 + r, W - 1) * st.w + piece * (16 / (int)sizeof(T))));
}
// This lane's pieces of the strip's rows x against its pieces of the halo rows at `halo` (the strip's first):
// acc[r][j] += x[r] . halo[j].  raw: the lane's first piece of x; the next is loaded under the arithmetic of one.
template <typename T, int KS, bool REGULAR>
__device__ __forceinline__ void dot(float (&acc)[kR][kU<KS>], uint4 (&raw)[kR], const T* x, const Na2dStride& st, int t0, int W,
                                    const uint4* halo, int pieces, int pitch, int lane) {
    constexpr int NP = Pairs<T>::N;
#pragma unroll 1
    for (int piece = lane; piece < pieces; piece += kLanes) {
        uint64_t q[kR][NP];
#pragma unroll
        for (int r = 0; r < kR; ++r) unpack(raw[r], q[r], T{});
        if (piece + kLanes < pieces) load_strip<T>(raw, x, st, t0, W, piece + kLanes);
#pragma unroll
        for (int j = 0; j < kU<KS>; ++j) {
            uint64_t y[NP];
            unpack(halo[j * pitch + piece], y, T{});
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                if (REGULAR && !(j >= r && j - r < KS)) continue;
                uint64_t part = mul2(q[r][0], y[0]);
#pragma unroll
                for (int c = 1; c < NP; ++c) part = fma2(q[r][c], y[c], part);
                acc[r][j] += lo2(part) + hi2(part);
            }
        }
    }
}
// Scores of token t0 + lane against the halo rows from the strip's start on, summed over the strip's lanes.
template <typename T, int KS>
__device__ __forceinline__ void scores(float (&s)[kU<KS>], uint4 (&raw)[kR], const Operand& x, const Place& p, const na2d_tile::Strip& w,
                                       int W, const uint4* halo, int pieces, int pitch) {
    float acc[kR][kU<KS>];
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
        for (int j = 0; j < kU<KS>; ++j) acc[r][j] = 0.f;
    const T* xs = sequence<T>(x, p);
    if (w.regular) dot<T, KS, true>(acc, raw, xs, x.st, p.t0, W, halo, pieces, pitch, p.lane);
    else dot<T, KS, false>(acc, raw, xs, x.st, p.t0, W, halo, pieces, pitch, p.lane);
    __syncwarp();
    const bool high = p.lane & 2, odd = p.lane & 1;
#pragma unroll
    for (int j = 0; j < kU<KS>; ++j) {
        // lanes 0, 1 keep tokens 0, 1, lanes 2, 3 tokens 2, 3; then the even lane the even one
        const float a = (high ? acc[2][j] : acc[0][j]) + __shfl_xor_sync(0xffffffffu, high ? acc[0][j] : acc[2][j], 2);
        const float b = (high ? acc[3][j] : acc[1][j]) + __shfl_xor_sync(0xffffffffu, high ? acc[1][j] : acc[3][j], 2);
        s[j] = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
    }
}

// out[r] = factor[r] * sum over the window of weight * halo row, this lane's pieces; weights of halo row j at w[j] (four tokens).
template <typename T, int KS, bool REGULAR>
__device__ __forceinline__ void apply(T* out, const Na2dStride& st, int t0, int W, const float4* w, const uint4* halo, int pieces,
                                      int pitch, int lane, const na2d_tile::Strip& s, float4 factor) {
    constexpr int kN = 16 / sizeof(T), NP = Pairs<T>::N;
    for (int piece = lane; piece < pieces; piece += kLanes) {
        uint64_t acc[kR][NP];
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int c = 0; c < NP; ++c) acc[r][c] = 0;
#pragma unroll
        for (int j = 0; j < kU<KS>; ++j) {
            uint64_t y[NP];
            unpack(halo[j * pitch + piece], y, T{});
            const float4 wt = w[j];
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                if (!(REGULAR ? (j >= r && j - r < KS) : na2d_tile::in_window<KS>(s, r, j))) continue;
                const float x = na2d_tile::lane_of(wt, r);
#pragma unroll
                for (int c = 0; c < NP; ++c) acc[r][c] = fma2(pair2(x, x), y[c], acc[r][c]);
            }
        }
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const float f = na2d_tile::lane_of(factor, r);
#pragma unroll
            for (int c = 0; c < NP; ++c) acc[r][c] = mul2(pair2(f, f), acc[r][c]);
            if (t0 + r < W) *reinterpret_cast<uint4*>(out + (long long)(t0 + r) * st.w + piece * kN) = pack(acc[r], T{});
        }
    }
}

// ------------------------------------------------------------------------------------ forward
template <typename T, int KS>
__global__ void __launch_bounds__(kThreads, KS >= 11 ? 3 : 4)
fwd_kernel(const __grid_constant__ Operand q, const __grid_constant__ Operand k, const __grid_constant__ Operand v,
           const __grid_constant__ Operand o, float* __restrict__ lse, const __grid_constant__ Na2dGeom g) {
    extern __shared__ uint4 smem16[];
    const int pieces = g.C * (int)sizeof(T) / 16, pitch = pitch_of(g.C * (int)sizeof(T));
    uint4 *sk = smem16, *sv = sk + kRows<KS> * pitch;
    float* weights = reinterpret_cast<float*>(sv + kRows<KS> * pitch);
    const Place p = place_of_block(g, 0);
    const int h0 = na2d_ws(p.x0, g.W, KS), rows = na2d_ws(min(p.x0 + kTile, g.W) - 1, g.W, KS) + KS - h0;
    copy_rows<T, 1>({sk}, {sequence<T>(k, p)}, {&k.st}, h0, rows, pieces, pitch);
    commit();
    copy_rows<T, 1>({sv}, {sequence<T>(v, p)}, {&v.st}, h0, rows, pieces, pitch);
    commit();
    const na2d_tile::Strip w = na2d_tile::strip_at<KS>(p.t0, g.W);
    const int hx = w.start - h0;
    uint4 raw[kR];
    if (p.lane < pieces) load_strip<T>(raw, sequence<T>(q, p), q.st, p.t0, g.W, p.lane);
    arrived<1>();
    __syncthreads();
    float s[kU<KS>];
    scores<T, KS>(s, raw, q, p, w, g.W, sk + hx * pitch, pieces, pitch);
    // softmax of token t0 + lane
    const int t = p.t0 + p.lane, off = p.lane == 0 ? w.off[0] : p.lane == 1 ? w.off[1] : p.lane == 2 ? w.off[2] : w.off[3];
    float m = -CUDART_INF_F;
#pragma unroll
    for (int j = 0; j < kU<KS>; ++j) {
        s[j] *= g.scale;
        if ((unsigned)(j - off) < (unsigned)KS) m = fmaxf(m, s[j]);
    }
    float l[4] = {0.f, 0.f, 0.f, 0.f};                     // four short sums instead of a long one
    float* mine = weights + p.strip * kSlots<KS>;
#pragma unroll
    for (int j = 0; j < kU<KS>; ++j) {
        const float e = (unsigned)(j - off) < (unsigned)KS ? expf(s[j] - m) : 0.f;
        l[j & 3] += e;
        mine[j * kR + p.lane] = e;
    }
    const float total = (l[0] + l[1]) + (l[2] + l[3]), inv = 1.f / total;
    if (t < g.W) lse[(long long)p.bn * g.W + t] = m + logf(total);
    mine[kU<KS> * kR + p.lane] = inv;
    arrived<0>();
    __syncthreads();
    const float4* wt = reinterpret_cast<const float4*>(mine);
    T* out = sequence<T>(o, p);
    if (w.regular) apply<T, KS, true>(out, o.st, p.t0, g.W, wt, sv + hx * pitch, pieces, pitch, p.lane, w, wt[kU<KS>]);
    else apply<T, KS, false>(out, o.st, p.t0, g.W, wt, sv + hx * pitch, pieces, pitch, p.lane, w, wt[kU<KS>]);
}

// ------------------------------------------------------------------------------------ dQ (+ delta, P, dS)
// As na2d_tile::dq_kernel; the weights go out in that kernel's layout, a tile's slots one after another.
template <typename T, int KS>
__global__ void __launch_bounds__(kThreads, KS >= 11 ? 3 : 4)
dq_kernel(const __grid_constant__ Operand q, const __grid_constant__ Operand k, const __grid_constant__ Operand v,
          const __grid_constant__ Operand d_o, const __grid_constant__ Operand d_q, const float* __restrict__ lse,
          float* __restrict__ delta, float* __restrict__ row_factor, float4* __restrict__ p_out, float4* __restrict__ ds_out,
          const int unit0, const __grid_constant__ Na2dGeom g) {
    extern __shared__ uint4 smem16[];
    const int pieces = g.C * (int)sizeof(T) / 16, pitch = pitch_of(g.C * (int)sizeof(T));
    uint4 *sk = smem16, *sv = sk + kRows<KS> * pitch;
    float* weights = reinterpret_cast<float*>(sv + kRows<KS> * pitch);
    const Place p = place_of_block(g, unit0);
    const int h0 = na2d_ws(p.x0, g.W, KS), rows = na2d_ws(min(p.x0 + kTile, g.W) - 1, g.W, KS) + KS - h0;
    copy_rows<T, 1>({sv}, {sequence<T>(v, p)}, {&v.st}, h0, rows, pieces, pitch);
    commit();
    copy_rows<T, 1>({sk}, {sequence<T>(k, p)}, {&k.st}, h0, rows, pieces, pitch);
    commit();
    const na2d_tile::Strip w = na2d_tile::strip_at<KS>(p.t0, g.W);
    const int hx = w.start - h0;
    const int t = p.t0 + p.lane, off = p.lane == 0 ? w.off[0] : p.lane == 1 ? w.off[1] : p.lane == 2 ? w.off[2] : w.off[3];
    const long long stat = (long long)p.bn * g.W + t;
    const float row_lse = t < g.W ? lse[stat] : 0.f;
    uint4 raw[kR];
    if (p.lane < pieces) load_strip<T>(raw, sequence<T>(d_o, p), d_o.st, p.t0, g.W, p.lane);
    arrived<1>();
    __syncthreads();
    float dp[kU<KS>], s[kU<KS>];
    scores<T, KS>(dp, raw, d_o, p, w, g.W, sv + hx * pitch, pieces, pitch);
    if (p.lane < pieces) load_strip<T>(raw, sequence<T>(q, p), q.st, p.t0, g.W, p.lane);
    arrived<0>();
    __syncthreads();
    scores<T, KS>(s, raw, q, p, w, g.W, sk + hx * pitch, pieces, pitch);
    float l[2] = {0.f, 0.f}, dl[2] = {0.f, 0.f};           // two short sums instead of a long one
#pragma unroll
    for (int j = 0; j < kU<KS>; ++j) {
        const bool in = (unsigned)(j - off) < (unsigned)KS;
        s[j] = in ? expf(s[j] * g.scale - row_lse) : 0.f;
        dp[j] = in ? dp[j] : 0.f;
        l[j & 1] += s[j];
        if (in) dl[j & 1] = fmaf(s[j], dp[j], dl[j & 1]);
    }
    const float factor = na2d_row_factor(l[0] + l[1], row_lse), total = (dl[0] + dl[1]) * factor;
    if (t < g.W) {
        delta[stat] = total;
        if (row_factor) row_factor[stat] = factor;
    }
    float* mine = weights + p.strip * kSlots<KS>;
    const float4* wt = reinterpret_cast<const float4*>(mine);
    const long long place = ((long long)(p.bn - unit0) * ((g.W + kTile - 1) / kTile) + p.x0 / kTile) * (kStrips * kU<KS>) + p.strip * kU<KS>;
#pragma unroll
    for (int j = 0; j < kU<KS>; ++j) s[j] *= factor;
    if (p_out) {
#pragma unroll
        for (int j = 0; j < kU<KS>; ++j) mine[j * kR + p.lane] = s[j];
        __syncwarp();
        for (int j = p.lane; j < kU<KS>; j += kLanes) p_out[place + j] = wt[j];
        __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < kU<KS>; ++j) {
        const bool in = (unsigned)(j - off) < (unsigned)KS;
        mine[j * kR + p.lane] = in ? g.scale * s[j] * (dp[j] - total) : 0.f;
    }
    __syncwarp();
    if (ds_out)
        for (int j = p.lane; j < kU<KS>; j += kLanes) ds_out[place + j] = wt[j];
    if (d_q.ptr) {
        const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
        T* out = sequence<T>(d_q, p);
        if (w.regular) apply<T, KS, true>(out, d_q.st, p.t0, g.W, wt, sk + hx * pitch, pieces, pitch, p.lane, w, one);
        else apply<T, KS, false>(out, d_q.st, p.t0, g.W, wt, sk + hx * pitch, pieces, pitch, p.lane, w, one);
    }
}

// ------------------------------------------------------------------------------------ dK, dV
// What a strip of four keys sums over: query rows [first, first + met), of which key r meets [lo[r], hi[r]).
struct Met {
    int first, met, lo[kR], hi[kR];
    bool regular;
};
template <int KS>
__device__ __forceinline__ Met met_by(int t0, int W) {
    Met m;
    m.first = na2d_bws(min(t0, W - 1), KS);
    m.met = 0;
    m.regular = true;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
        m.lo[r] = t0 + r < W ? na2d_bws(t0 + r, KS) - m.first : 0;
        m.hi[r] = t0 + r < W ? na2d_bwe(t0 + r, W, KS) - m.first : 0;
        m.met = max(m.met, m.hi[r]);
        m.regular = m.regular && m.lo[r] == r && m.hi[r] == r + KS;
    }
    return m;
}
template <typename T, int KS, bool REGULAR>
__device__ __forceinline__ void key_sums(T* out_k, T* out_v, const Na2dStride& st_k, const Na2dStride& st_v, int t0, int W, const float4* ds,
                                         const float4* pw, const uint4* xq, const uint4* xg, int pieces, int pitch, int lane, const Met& m) {
    constexpr int kN = 16 / sizeof(T), NP = Pairs<T>::N;
    for (int piece = lane; piece < pieces; piece += kLanes) {
        uint64_t dk[kR][NP], dv[kR][NP];
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int c = 0; c < NP; ++c) dk[r][c] = dv[r][c] = 0;
        auto row = [&](int i) {
            uint64_t yq[NP], yg[NP];
            unpack(xq[i * pitch + piece], yq, T{});
            unpack(xg[i * pitch + piece], yg, T{});
            const float4 a = ds[i], b = pw[i];
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                if (!(REGULAR ? (i >= r && i - r < KS) : (i >= m.lo[r] && i < m.hi[r]))) continue;
                const float wa = na2d_tile::lane_of(a, r), wb = na2d_tile::lane_of(b, r);
#pragma unroll
                for (int c = 0; c < NP; ++c) {
                    dk[r][c] = fma2(pair2(wa, wa), yq[c], dk[r][c]);
                    dv[r][c] = fma2(pair2(wb, wb), yg[c], dv[r][c]);
                }
            }
        };
        if constexpr (REGULAR) {
#pragma unroll
            for (int i = 0; i < kU<KS>; ++i) row(i);
        } else {
            for (int i = 0; i < m.met; ++i) row(i);
        }
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            if (t0 + r >= W) continue;
            *reinterpret_cast<uint4*>(out_k + (long long)(t0 + r) * st_k.w + piece * kN) = pack(dk[r], T{});
            *reinterpret_cast<uint4*>(out_v + (long long)(t0 + r) * st_v.w + piece * kN) = pack(dv[r], T{});
        }
    }
}

template <typename T, int KS>
__global__ void __launch_bounds__(kThreads, 3)
key_kernel(const __grid_constant__ Operand q, const __grid_constant__ Operand d_o, const __grid_constant__ Operand d_k,
           const __grid_constant__ Operand d_v, const float4* __restrict__ p_in, const float4* __restrict__ ds_in, const int unit0,
           const __grid_constant__ Na2dGeom g) {
    extern __shared__ uint4 smem16[];
    const int pieces = g.C * (int)sizeof(T) / 16, pitch = pitch_of(g.C * (int)sizeof(T));
    uint4 *sq = smem16, *sg = sq + kKeyRows<KS> * pitch;
    constexpr int kStrip = (kMet<KS> + 1) * kR;             // floats, padded against bank conflicts
    float *weights_ds = reinterpret_cast<float*>(sg + kKeyRows<KS> * pitch), *weights_p = weights_ds + kStrips * kStrip;
    const Place p = place_of_block(g, unit0);
    const int h0 = na2d_bws(p.x0, KS), rows = na2d_bwe(min(p.x0 + kTile, g.W) - 1, g.W, KS) - h0;
    copy_rows<T, 2>({sq, sg}, {sequence<T>(q, p), sequence<T>(d_o, p)}, {&q.st, &d_o.st}, h0, rows, pieces, pitch);
    commit();
    // This lane's key t: its weights from the strips of queries that see it, a float4 (four queries) each.
    const Met m = met_by<KS>(p.t0, g.W);
    const int t = p.t0 + p.lane;
    if (t < g.W) {
        const int lo = na2d_bws(t, KS), hi = na2d_bwe(t, g.W, KS);
        const long long unit = (long long)(p.bn - unit0) * ((g.W + kTile - 1) / kTile) * (kStrips * kU<KS>);
        for (int s4 = lo / kR; s4 <= (hi - 1) / kR; ++s4) {          // (strip kStrips * tile + s has its slots at that place)
            const int j = t - na2d_ws(kR * s4, g.W, KS);
            const float4 a = __ldg(ds_in + unit + (long long)s4 * kU<KS> + j), b = __ldg(p_in + unit + (long long)s4 * kU<KS> + j);
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                const int i = kR * s4 + r;
                if (i < lo || i >= hi) continue;
                const int at = p.strip * kStrip + (i - m.first) * kR + p.lane;
                weights_ds[at] = na2d_tile::lane_of(a, r);
                weights_p[at] = na2d_tile::lane_of(b, r);
            }
        }
    }
    arrived<0>();
    __syncthreads();
    const float4 *ds = reinterpret_cast<const float4*>(weights_ds + p.strip * kStrip), *pw = reinterpret_cast<const float4*>(weights_p + p.strip * kStrip);
    const uint4 *xq = sq + (m.first - h0) * pitch, *xg = sg + (m.first - h0) * pitch;
    if (m.regular) key_sums<T, KS, true>(sequence<T>(d_k, p), sequence<T>(d_v, p), d_k.st, d_v.st, p.t0, g.W, ds, pw, xq, xg, pieces, pitch, p.lane, m);
    else key_sums<T, KS, false>(sequence<T>(d_k, p), sequence<T>(d_v, p), d_k.st, d_v.st, p.t0, g.W, ds, pw, xq, xg, pieces, pitch, p.lane, m);
}

}  // namespace na2d_line
