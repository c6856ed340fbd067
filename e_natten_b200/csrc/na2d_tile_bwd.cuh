// Tiled CUDA-core kernels of the backward: the query half, which hands the weights P and dS on, and the
// key-side sum over the inverse neighbourhood.
//
// What bounds them: the shared-memory pipe and block barriers in the query half (three loops of the forward's kind),
// issue slots in the key sums.  Keeping P and dS (2 ks * (ks + 3) floats per pixel) costs less than the two score loops
// that would form them again.  Measured on one B200 against the warp-per-pixel kernels, 4 x 4 x 256 x 256 x 128,
// window 5, fp32: both halves 27.6 -> 2.24 ms; 4 x 8 x 4096 x 64, window 13, bf16, 1D: step 1.72 -> 0.29 ms.
// (fp32 in 2D goes to na2d_box.cuh and 1D rows to na2d_line.cuh where rows start on 16-byte boundaries; these kernels keep the rest.)
#pragma once

#include "na2d_tile.cuh"

namespace na2d_tile {

// ------------------------------------------------------------------------------------ dQ (+ delta, P, dS)
// delta = sum_j p_j dp_j, which equals dO . o exactly and does not depend on how o was rounded when it
// was stored.  d_q may be null: then only delta (and the weights) are produced.  p_out / ds_out, both or
// neither: the tiles' weight slots for the key half, as they lie in shared memory, tile after tile in the rows of
// `band`'s ring.  row_factor (or null): what each row's exp(s - lse) is multiplied by to be P.
template <typename T, int KS, bool ONE_D, bool PARK>
__global__ void __launch_bounds__(Shape<KS, ONE_D>::kThreads, Shape<KS, ONE_D>::kBlocks)
dq_kernel(const __grid_constant__ Operand q, const __grid_constant__ Operand k, const __grid_constant__ Operand v,
          const __grid_constant__ Operand d_o, const __grid_constant__ Operand d_q, const float* __restrict__ lse,
          float* __restrict__ delta, float* __restrict__ row_factor, float4* __restrict__ p_out, float4* __restrict__ ds_out,
          const __grid_constant__ Band band, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS, ONE_D>;
    extern __shared__ float4 smem[];
    float4 *w = smem, *own = w + S::kWeights, *halo = own + S::kOwn;
    const Tile t = tile_of_block<S>(g, g.Hq, band.unit0, band.row0, band.rows);
    int ky0, kx0, halo_rows;
    query_halo<S>(t, g, ky0, kx0, halo_rows);
    const DotItem d = dot_item<S>(t, g, ky0, kx0);
    float4* slots = weight_slots<S>(w, d);
    const int c0 = t.x0 + kR * d.strip;
    const long long stat = ((long long)t.bn * g.Hq + t.y0 + d.row) * g.W + c0;
    float s[kR][S::kU];
    // dP first, parked in the thread's own weight slots; the scores second, so that the halo ends up
    // holding a chunk of k, which dQ needs next
    tile_dot<T, S, PARK>(s, d_o, v, own, halo, t, d, g, ky0, kx0, halo_rows);
    if (d.active) {
#pragma unroll
        for (int j = 0; j < S::kU; ++j)
            if (j % S::kSplit == d.split) slots[j * S::kTh] = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
    }
    tile_dot<T, S, PARK>(s, q, k, own, halo, t, d, g, ky0, kx0, halo_rows);
    float4 *part = own, *total = own + S::kTh * S::kStrips * S::kKh;
    if (d.active) {
        float dl[2][kR], l[2][kR];                          // two short sums instead of a long one
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            dl[0][r] = dl[1][r] = l[0][r] = l[1][r] = 0.f;
            const float row_lse = c0 + r < g.W ? lse[stat + r] : 0.f;
#pragma unroll
            for (int j = 0; j < S::kU; ++j) s[r][j] = in_window<KS>(d.s, r, j) ? expf(s[r][j] * g.scale - row_lse) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < S::kU; ++j) {
            const float4 dp = slots[j * S::kTh];
#pragma unroll
            for (int r = 0; r < kR; ++r)
                if (in_window<KS>(d.s, r, j)) {
                    l[j & 1][r] += s[r][j];
                    dl[j & 1][r] = fmaf(s[r][j], lane_of(dp, r), dl[j & 1][r]);
                }
        }
        if (d.split == 0) {
            const int slot = (d.strip * S::kKh + d.u) * S::kTh + d.row;
            part[slot] = make_float4(dl[0][0] + dl[1][0], dl[0][1] + dl[1][1], dl[0][2] + dl[1][2], dl[0][3] + dl[1][3]);
            total[slot] = make_float4(l[0][0] + l[1][0], l[0][1] + l[1][1], l[0][2] + l[1][2], l[0][3] + l[1][3]);
        }
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
            for (int j = 0; j < S::kU; ++j) s[r][j] *= lane_of(inv, r);
        if (d.u == 0 && d.split == 0) {
#pragma unroll
            for (int r = 0; r < kR; ++r)
                if (c0 + r < g.W) {
                    delta[stat + r] = lane_of(dl4, r);
                    if (row_factor) row_factor[stat + r] = lane_of(inv, r);
                }
        }
        // the slots turn from dP into P, the registers from P into dS
#pragma unroll
        for (int j = 0; j < S::kU; ++j) {
            const float4 dp = slots[j * S::kTh];
            if constexpr (S::kSplit > 1) __syncwarp(0xfu << (threadIdx.x & 28));      // a strip's four lanes share its slots
            if (p_out && j % S::kSplit == d.split) slots[j * S::kTh] = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
#pragma unroll
            for (int r = 0; r < kR; ++r) s[r][j] = g.scale * s[r][j] * (lane_of(dp, r) - lane_of(dl4, r));
        }
    }
    const long long place = (((long long)(t.bn - band.unit0) * band.ring + t.y0 / S::kTh % band.ring) *
                                 ((g.W + S::kTw - 1) / S::kTw) + t.x0 / S::kTw) * S::kWeights;
    if (p_out) {
        __syncthreads();
        for (int i = threadIdx.x; i < S::kWeights; i += S::kThreads) p_out[place + i] = w[i];
        __syncthreads();
    }
    if (d.active) {
#pragma unroll
        for (int j = 0; j < S::kU; ++j)
            if (j % S::kSplit == d.split) slots[j * S::kTh] = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
    }
    if (ds_out) {
        __syncthreads();
        for (int i = threadIdx.x; i < S::kWeights; i += S::kThreads) ds_out[place + i] = w[i];
    }
    if (d_q.ptr) tile_apply<T, S>(d_q, k, w, nullptr, halo, t, g, ky0, kx0, halo_rows, true);
}

// ------------------------------------------------------------------------------------ key side
// out[key] = sum over the queries i whose window holds the key of attn[i, position of the key in i's window]
// * x[i]: dK (attn = dS, x = q) and dV (attn = P, x = dO).  Two such sums run in one launch (blockIdx.y).
// Whole images only; attn starts at the launch's first unit: the dense (units, H, W, kh * ks) array of the
// unfused pair, or (TILED) the weight slots of query tiles that dq_kernel wrote, in the rows of `band`'s ring.
//
// The queries that see a key are a product of a row range and a column range: ks x ks away from the
// borders, up to (3 * ks / 2) on a side near them.  A strip of four keys away from the borders meets a band
// of ks + 3 query columns, as in the apply loop above.  Query rows are taken in groups that fit the shared
// memory, the weights being gathered into the apply loop's layout.
constexpr int max_of(int a, int b) { return a > b ? a : b; }

template <typename S>
struct KeyShape {
    static constexpr int KS = S::kKs;
    static constexpr int kThreads = S::kApply;
    // Query columns of one strip, at most: a strip that starts below KS meets column 0, and up to KS columns past it.
    static constexpr int kMaxUnion = max_of((KS - 1) / kR * kR + kR - 1 + KS, kR - 1 + KS + KS / 2);
    static constexpr int kWeights = max_of(S::kWeights, S::kTh * S::kStrips * kMaxUnion);
    // Room for the query columns of any tile and for at least two query rows of each of its key rows.  A
    // tile whose first key column x0 lies below KS starts at query column 0 and may end KS columns past its last
    // key; one whose first row lies below KS and its last does not has first query rows up to kSpan apart.
    static constexpr int kBelow = (KS - 1) / S::kTw * S::kTw;              // last tile column start below KS
    static constexpr int kMaxCols = max_of(kBelow + S::kTw - 1 + KS, S::kTw - 1 + KS + KS / 2);
    static constexpr int kLast = S::kOneD ? 0 : (KS - 1) / S::kTh * S::kTh + S::kTh - 1;
    static constexpr int kSpan = S::kOneD ? 0 : max_of(S::kTh - 1, kLast < KS ? 0 : kLast - KS / 2);
    static constexpr int kHalo = max_of(S::kHalo, kMaxCols * (kSpan + 2) * kF);
    static constexpr int kSmem = (kWeights + kHalo) * 16;
    static constexpr int kBlocksSmem = kSmemPerSm / (kSmem + 1024);
    // With the dense weights of the unfused pair three blocks of 256 threads, 80 registers each, are faster than four with 64 from window 5
    // on (both spill: 4 to 48 bytes a thread with 80, 36 to 120 with 64): 4 x 4 x 64 x 64 x 128, window 5, fp32, both calls' backwards 287 -> 254 us (4 x 8 x 64 x 96 x 48, window 3,
    // fp16 237 -> 242).  With tiled ones four are (4 x 4 x 256 x 256 x 128, fp32: 1.0 against 1.1 ms).
    static constexpr int kBlocksTiled = kBlocksSmem * kThreads > 1024 ? 1024 / kThreads : kBlocksSmem;
    static constexpr int kBlocksDense = KS > 3 && kBlocksSmem * kThreads > 768 ? 768 / kThreads : kBlocksTiled;
};

// stage() for a halo of `cols` columns, all of them inside the image.
template <typename T, int TH, int THREADS>
__device__ __forceinline__ void stage_columns(float4* dst, const T* src, const Na2dStride& st, int y0, int rows, int x0,
                                              int cols, int c0, int C, bool vec) {
    constexpr int kPx = THREADS / kF;
    const int f = threadIdx.x % kF, c = c0 + 4 * f, first = threadIdx.x / kF;
    const bool in = c < C;
    int y = first / cols, x = first - y * cols;
    const T* p = src + (y0 + y) * st.h + (x0 + x) * st.w + c;
    const long long wrap = st.h - cols * st.w;
    const int n = rows * cols;
#pragma unroll 2
    for (int px = first; px < n; px += kPx) {
        stage_quad<T>(dst + px * kF + place_of<TH>(f, y, x), in ? p : src, in, c, C, vec);
        x += kPx;
        p += kPx * st.w;
        while (x >= cols) { x -= cols; ++y; p += wrap; }
    }
}

struct KeySum {
    const void* attn;
    Operand x, out;
};

template <typename T, typename TW, bool TILED, int KS, bool ONE_D>
__global__ void __launch_bounds__(KeyShape<Shape<KS, ONE_D>>::kThreads, TILED ? KeyShape<Shape<KS, ONE_D>>::kBlocksTiled : KeyShape<Shape<KS, ONE_D>>::kBlocksDense)
key_sum_kernel(const __grid_constant__ KeySum first, const __grid_constant__ KeySum second,
               const __grid_constant__ Band band, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS, ONE_D>;
    using K = KeyShape<S>;
    constexpr int kTaps = S::kKh * KS;
    extern __shared__ float4 smem[];
    float4 *w = smem, *halo = w + K::kWeights;
    const KeySum& job = blockIdx.y == 0 ? first : second;
    const Tile t = tile_of_block<S>(g, g.Hkv, band.unit0, band.row0, band.rows);
    const int H = g.Hg, W = g.W;
    // query rows and columns the tile's keys meet
    const int qy0 = na2d_bws(t.y0, S::kKh), qx0 = na2d_bws(t.x0, KS);
    const int cols = na2d_bwe(t.x0 + t.cols - 1, W, KS) - qx0;
    const int row_span = na2d_bws(t.y0 + t.rows - 1, S::kKh) - qy0;      // how far the keys' first query rows lie apart
    int nu = 0, nj = 0;
    for (int y = 0; y < t.rows; ++y) nu = max(nu, na2d_bwe(t.y0 + y, H, S::kKh) - na2d_bws(t.y0 + y, S::kKh));
    for (int x = 0; x < t.cols; x += kR)
        nj = max(nj, na2d_bwe(min(t.x0 + x + kR, W) - 1, W, KS) - na2d_bws(t.x0 + x, KS));
    const int group = min(nu, min(K::kWeights / (S::kTh * S::kStrips * nj), K::kHalo / (kF * cols) - row_span));

    const int f = threadIdx.x % kF, row = threadIdx.x / kF % S::kTh, strip = threadIdx.x / (kF * S::kTh);
    const bool active = row < t.rows && kR * strip < t.cols;
    const int c0 = t.x0 + kR * strip;
    Strip s;                                               // off: first query column; hi: one past the last
    int hi[kR];
    s.start = na2d_bws(min(c0, W - 1), KS);
    s.regular = true;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
        s.off[r] = c0 + r < W ? na2d_bws(c0 + r, KS) - s.start : 0;
        hi[r] = c0 + r < W ? na2d_bwe(c0 + r, W, KS) - s.start : 0;
        s.regular = s.regular && s.off[r] == r && hi[r] == r + KS;
    }
    const int my_nj = max(max(hi[0], hi[1]), max(hi[2], hi[3]));
    const int my_u0 = na2d_bws(t.y0 + min(row, t.rows - 1), S::kKh), my_nu = na2d_bwe(t.y0 + min(row, t.rows - 1), H, S::kKh) - my_u0;
    const int hx = s.start - qx0;

    const int tiles_w = (W + S::kTw - 1) / S::kTw;
    const unsigned first_tile_row = (unsigned)qy0 / S::kTh, first_place = first_tile_row % (unsigned)band.ring;
    const TW* attn = static_cast<const TW*>(job.attn) +
                     (t.bn - band.unit0) * (TILED ? (long long)band.ring * tiles_w * S::kWeights * kR : (long long)H * W * kTaps);
    const T* xs = unit<T>(job.x, t);
    T* os = unit<T>(job.out, t);
    for (int ch = 0; ch < g.C; ch += kChunk) {
        float4 acc[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int g0 = 0; g0 < nu; g0 += group) {
            const int gn = min(group, nu - g0);
            __syncthreads();
            const int rows = min(row_span + gn, H - qy0 - g0);
            if (cols == S::kHaloW)                          // away from the column borders
                stage<T, S::kTh, K::kThreads, S::kHaloW>(halo, xs, job.x.st, qy0 + g0, rows, qx0, W, ch, g.C, job.x.vec);
            else
                stage_columns<T, S::kTh, K::kThreads>(halo, xs, job.x.st, qy0 + g0, rows, qx0, cols, ch, g.C, job.x.vec);
            if (ch == 0 || group < nu) {
                // weights of the group: element (strip, u, j, row, r), four pixels r of eight rows to a warp.  Lane
                // (row, r) takes the d-th query column of its key, so that a warp's queries lie on a block of
                // neighbouring pixels, as its keys do: the slots of a query tile hold their weights side by side.
                const int lr = threadIdx.x % kR, ly = threadIdx.x / kR % S::kTh;
                constexpr int kPar = K::kThreads / (kR * S::kTh);
                const int y = t.y0 + ly;
                const int first_row = na2d_bws(min(y, H - 1), S::kKh) + g0;
                const int rows_here = ly < t.rows ? min(gn, na2d_bwe(y, H, S::kKh) - first_row) : 0;
                float* wf = reinterpret_cast<float*>(w);
                for (int k = threadIdx.x / (kR * S::kTh); k < S::kStrips * gn; k += kPar) {
                    const int st = k % S::kStrips, u = k / S::kStrips, col = t.x0 + kR * st + lr;
                    if (u >= rows_here || col >= W) continue;
                    const int lo = na2d_bws(col, KS), n = na2d_bwe(col, W, KS) - lo;
                    const int qy = first_row + u, uq = y - na2d_ws(qy, H, S::kKh);
                    float* to = wf + (((st * gn + u) * nj + lo - na2d_bws(t.x0 + kR * st, KS)) * S::kTh + ly) * kR + lr;
                    if constexpr (TILED) {
                        // query (qy, qx): tile (qy / kTh, qx / kTw), strip and pixel r of its column, row qy % kTh;
                        // the key is column col - (window start of the strip) of its halo
                        const unsigned in_row = (unsigned)qy % S::kTh;
                        unsigned place = first_place + (unsigned)qy / S::kTh - first_tile_row;
                        if (place >= (unsigned)band.ring) place -= band.ring;
                        const TW* line = attn + ((long long)(place * (unsigned)tiles_w) * S::kWeights + uq * (S::kU * S::kTh) + in_row) * kR;
#pragma unroll 4
                        for (int i = 0; i < n; ++i, to += S::kTh * kR) {
                            const unsigned qx = lo + i, strip_q = qx % S::kTw / kR;
                            const int j = col - na2d_ws(qx & ~(kR - 1u), W, KS);
                            copy4(to, line + (long long)(qx / S::kTw) * (S::kWeights * kR) +
                                          (int)((strip_q * (S::kKh * S::kU) + j) * (S::kTh * kR) + qx % kR));
                        }
                    } else {
                        const TW* line = attn + (long long)qy * W * kTaps + uq * KS + col;
#pragma unroll 4
                        for (int i = 0; i < n; ++i, to += S::kTh * kR)
                            *to = to_f<TW>(__ldg(line + (long long)(lo + i) * kTaps - na2d_ws(lo + i, W, KS)));
                    }
                }
            }
            copies_done();
            __syncthreads();
            if (active) {
                const int n_rows = min(gn, my_nu - g0);
                for (int u = 0; u < n_rows; ++u) {
                    const int hy = my_u0 - qy0 + u;
                    const float4* wr = w + (strip * gn + u) * nj * S::kTh + row;
                    const float4* hr = halo + (hy * cols + hx) * kF;
                    if (s.regular) {
                        apply_row<S, true>(acc, wr, hr, f, hy, hx, s);
                    } else {
                        for (int j = 0; j < my_nj; ++j) {
                            const float4 x = hr[j * kF + place_of<S::kTh>(f, hy, hx + j)];
                            const float4 wt = wr[j * S::kTh];
#pragma unroll
                            for (int r = 0; r < kR; ++r)
                                if (j >= s.off[r] && j < hi[r]) add_scaled(acc[r], lane_of(wt, r), x);
                        }
                    }
                }
            }
        }
        if (active) {
            T* o = os + (t.y0 + row) * job.out.st.h + c0 * job.out.st.w;
#pragma unroll
            for (int r = 0; r < kR; ++r)
                if (c0 + r < W) store_channels<T>(o + r * job.out.st.w, acc[r], ch + 4 * f, g.C, job.out.vec);
        }
    }
}

}  // namespace na2d_tile
