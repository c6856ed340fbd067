// Key half of the backward and of the unfused pair on the boxes of na2d_box.cuh:
// out[key] = sum over the queries i whose window holds the key of attn[i, position of the key in i's window] * x[i]: dK (attn = dS,
// x = q) and dV (attn = P, x = dO).  Two such sums run in one launch (blockIdx.y).  Whole images only; attn starts at the launch's
// first unit: the dense (units, H, W, KS * KS) array of the unfused pair, or (TILED) the slots of query tiles that dq_kernel wrote, in
// the rows of `band`'s ring.
//
// The queries that see a key are a product of a row range and a column range: KS x KS away from the borders, up to (3 * KS / 2)
// on a side near them.  The four keys of a strip meet strips of four queries each: the weights of a query strip for one key are one
// float4 (a slot of dq_kernel as it is), and that times the strip's four rows of x is what the query strip adds to the key.
// A thread holds such sums for the keys of kRows image rows, and reads a row of x once for all of them.  Query rows are taken in
// groups that fit the shared memory.
//
// Columns near the left and right border take one of two forms.
//   edges (windows 3 and 5)   A query at most KS / 2 columns from the key (the "band") sees it wherever the two lie: a clamped window
//          still holds whatever is that near.  The rest are queries nearer to the border than KS / 2 with a key further than that
//          from it, 1 or 3 pairs of columns a border: the band loop, known at compile time, runs for all strips (columns
//          outside the image are zeros, and so are their weights), and those pairs are added one by one.
//   strips (the other windows, of which 6 to 21 such pairs a border would wait for each other)   A strip whose keys all are a window's
//          width from the borders ("regular") runs the band loop; any other tests each pair of a query and a key, and so
//          do its weights take a slot for every pair of a query strip and a key.
// Measured on one B200, both sums of 32 x 128 x 64 pixels (half of the tiles at a border), 128 channels, edges / strips, us: window 3 165 / 207, 5
// 248 / 334, 7 462 / 466, 9 832 / 794, 13 2214 / 1713.
#pragma once

#include "na2d_box.cuh"

namespace na2d_box {

template <typename S>
struct KeyShape {
    static constexpr int KS = S::kKs, kHalf = KS / 2;
    static constexpr bool kEdges = KS <= 5;
    static constexpr int kRows = KS <= 5 ? 2 : 1;                        // image rows of a thread
    static constexpr int kThreads = S::kTh / kRows * S::kStrips * kF;
    static constexpr int kLeft = (kHalf + kR - 1) / kR;                  // query strips that a regular strip meets to its left
    // How far the first query rows of a tile's key rows lie apart: a tile may start below KS and end beyond it.
    static constexpr int kLast = (KS - 1) / S::kTh * S::kTh + S::kTh - 1;
    static constexpr int kSpan = max_of(S::kTh - 1, kLast < KS ? 0 : kLast - kHalf);
    // Edge pairs of a border: key KS / 2 + 1 + i from it (i < KS / 2) with the i + 1 queries next to it.  Float4 of a query row's.
    static constexpr int kPairs = kHalf * (kHalf + 1) / 2, kRowEdge = S::kTh * 2 * kPairs / 4;
    // Query strips that one strip of keys meets, at most: one that starts below KS meets column 0, and up to KS - 1 columns past it.
    static constexpr int kMaxStrips = max_of(((KS - 1) / kR * kR + KS + 2) / kR, (KS + 2) / kR + kLeft) + 1;
    static constexpr int kRowSlots = S::kTh * S::kStrips * S::kU;
    static constexpr int kSlots = kEdges ? KS * (kRowSlots + kRowEdge) : max_of(KS * kRowSlots, S::kTh * S::kStrips * kMaxStrips * kR);
    // Boxes: that of a tile away from the borders, and a wide one for those that meet more columns: edge pairs to the right
    // of the band, or whole query strips.  As many rows of it as fit the same room, and one more than kSpan at least.
    static constexpr int kMaxCols = (max_of((KS - 1) / S::kTw * S::kTw, kLeft * kR) + S::kTw + KS - 1 + kR - 1) / kR * kR;
    static constexpr int kWideW = (kEdges ? kHalf + S::kTw + KS - 1 : kMaxCols) | 1;
    static constexpr int kFit = S::kHaloH * S::kBoxW / kWideW, kWideH = max_of(kSpan + 1, kFit < S::kHaloH ? kFit : S::kHaloH);
    static constexpr int kWeightsAt = whole_kb(max_of(S::kHaloH * S::kBoxW, kWideH * kWideW) * kPixel);
    static constexpr int kBarriersAt = kWeightsAt + kSlots * 16, kSmem = kBarriersAt + S::kBarriers;
    static constexpr int kBlocksSmem = na2d_tile::kSmemPerSm / (kSmem + 1024);
    static constexpr int kBlocks = kBlocksSmem * kThreads > 512 ? 512 / kThreads : kBlocksSmem;
    static_assert(S::kHaloH > kSpan && kWideH > kSpan && kBlocks >= 1, "a query row of each key row fits");
    static_assert(!kEdges || S::kTw >= KS, "keys below KS lie in a row's first tile");
};

// A query row meets a row of a strip's keys: x the KS + 3 columns that it reaches, weights at wr[slot * kTh], slots those of the band or
// (PAIRS) of (query strip, key) pairs.
template <typename S, bool PAIRS>
__device__ __forceinline__ void key_band(Channels (&acc)[kR], const float4* wr, const ulonglong2 (&x)[S::kU]) {
    constexpr int kHalf = S::kKs / 2;
#pragma unroll
    for (int j = 0; j < S::kU; ++j) {
        const int d = (j + 4 * S::kKs - kHalf) / kR - S::kKs, r = j - kHalf - kR * d;      // floor((j - kHalf) / 4), and the rest
        const float4 wt = wr[(PAIRS ? (KeyShape<S>::kLeft - d) * kR + r : j) * S::kTh];
#pragma unroll
        for (int c = 0; c < kR; ++c) {
            const int q = c - kR * d;                      // query column, from the strip's
            if (q >= r - kHalf && q <= r + kHalf) add_scaled(acc[r], lane_of(wt, c), x[q + kHalf < 0 ? 0 : q + kHalf >= S::kU ? 0 : q + kHalf]);
        }
    }
}

struct KeyOut {
    const void* attn;
    Operand out;
};

// tm_x0, tm_x1: boxes of the two jobs' x, 32 channels, tm_w0, tm_w1: wide ones.
template <bool TILED, int KS>
__global__ void __launch_bounds__(KeyShape<Shape<KS>>::kThreads, KeyShape<Shape<KS>>::kBlocks)
key_sum_kernel(const __grid_constant__ CUtensorMap tm_x0, const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_x1,
               const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ KeyOut first, const __grid_constant__ KeyOut second,
               const ErrorState* __restrict__ errors, const __grid_constant__ Band band, const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS>;
    using K = KeyShape<S>;
    constexpr int kHalf = KS / 2, kGroups = S::kTh / K::kRows;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (!starts_right(smem, errors)) return;
    float4* w = reinterpret_cast<float4*>(smem + K::kWeightsAt);
    Loads loads(smem + K::kBarriersAt, errors);
    const Tile t = tile_of_block<S>(g, g.Hkv, band.unit0, band.row0, band.rows);
    const int H = g.Hg, W = g.W;
    // all strips of queries that the band meets are in the image, and their windows not shifted
    const bool inner = t.x0 >= KS && t.x0 + S::kTw <= W - KS;
    // (edges) the tile has edge pairs of the left, of the right border
    const bool left = t.x0 < KS && t.x0 + t.cols > kHalf + 1, right = t.x0 + t.cols > W - KS && t.x0 < W - 1 - kHalf;
    const bool wide = K::kEdges ? right && W > t.x0 + S::kTw + kHalf : !inner;
    // first query row that the tile's keys meet, and first column of the box: where the band begins, or the first query strip
    const int qy0 = na2d_bws(t.y0, KS), qx0 = K::kEdges || inner ? t.x0 - kHalf : na2d_bws(t.x0, KS) / kR * kR;
    const int box_w = wide ? K::kWideW : S::kBoxW, box_h = wide ? K::kWideH : S::kHaloH;
    auto load = [&](int c0, int row) {
        uint64_t* bar = loads.expect(0, box_w * box_h * kPixel);
        // (each map by its name: one chosen through a pointer may be copied to where TMA cannot read it)
        if (blockIdx.y == 0) {
            if (!wide) na2d_ptx::tma_load_5d(smem, &tm_x0, bar, c0, qx0, row, t.n, t.b);
            else na2d_ptx::tma_load_5d(smem, &tm_w0, bar, c0, qx0, row, t.n, t.b);
        } else {
            if (!wide) na2d_ptx::tma_load_5d(smem, &tm_x1, bar, c0, qx0, row, t.n, t.b);
            else na2d_ptx::tma_load_5d(smem, &tm_w1, bar, c0, qx0, row, t.n, t.b);
        }
    };
    if (threadIdx.x == 0) load(0, qy0);
    const KeyOut& job = blockIdx.y == 0 ? first : second;
    const int row_span = na2d_bws(t.y0 + t.rows - 1, KS) - qy0;          // how far the keys' first query rows lie apart
    int nu = 0, nj = S::kU;                                // query rows of a key row, weight slots of a strip, at most
#pragma unroll
    for (int y = 0; y < S::kTh; ++y)
        if (y < t.rows) nu = max(nu, na2d_bwe(t.y0 + y, H, KS) - na2d_bws(t.y0 + y, KS));
    if (!K::kEdges && !inner) {
        nj = 0;
#pragma unroll
        for (int x = 0; x < S::kTw; x += kR)
            if (x < t.cols) nj = max(nj, ((na2d_bwe(min(t.x0 + x + kR, W) - 1, W, KS) - 1) / kR - na2d_bws(t.x0 + x, KS) / kR + 1) * kR);
    }
    const int group = min(nu, min(K::kEdges || inner ? KS : K::kSlots / (S::kTh * S::kStrips * nj), box_h - row_span));

    const int f = threadIdx.x % kF, row0 = threadIdx.x / kF % kGroups * K::kRows, strip = threadIdx.x / (kF * kGroups);
    const bool active = row0 < t.rows && kR * strip < t.cols;
    const int c0 = t.x0 + kR * strip;
    // (strips) query columns of each key: the first one from the first query strip's, and how many
    const bool regular = K::kEdges || (c0 >= KS && c0 + kR <= W - KS);
    const int strip0 = na2d_bws(min(c0, W - 1), KS) / kR;
    int lo[kR], n_of[kR], strips = 0;
    if constexpr (!K::kEdges) {
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            lo[r] = c0 + r < W ? na2d_bws(c0 + r, KS) - strip0 * kR : 0;
            const int hi = c0 + r < W ? na2d_bwe(c0 + r, W, KS) - strip0 * kR : 0;
            n_of[r] = hi - lo[r];
            strips = max(strips, (hi + kR - 1) / kR);
        }
    }
    int u0[K::kRows], rows_of[K::kRows];                   // query rows of each key row
#pragma unroll
    for (int p = 0; p < K::kRows; ++p) {
        const int y = t.y0 + row0 + p;
        u0[p] = na2d_bws(min(y, H - 1), KS);
        rows_of[p] = row0 + p < t.rows ? na2d_bwe(y, H, KS) - u0[p] : 0;
    }
    const int last = row0 + K::kRows <= t.rows ? K::kRows - 1 : 0;       // the last of them in the tile

    const int tiles_w = (W + S::kTw - 1) / S::kTw;
    const unsigned first_tile_row = (unsigned)qy0 / S::kTh, first_place = first_tile_row % (unsigned)band.ring;
    const float* attn = static_cast<const float*>(job.attn) +
                        (t.bn - band.unit0) * (TILED ? (long long)band.ring * tiles_w * S::kBand * kR : (long long)H * W * kTaps<KS>);
    float* os = unit<float>(job.out, t) + (t.y0 + row0) * job.out.st.h + c0 * job.out.st.w + 4 * f;

    // Weights of query row qy for key row y.
    auto row_at = [&](int qy, int y) {
        const int uq = y - na2d_ws(qy, H, KS);
        if constexpr (TILED) {
            unsigned place = first_place + (unsigned)qy / S::kTh - first_tile_row;
            if (place >= (unsigned)band.ring) place -= band.ring;
            return attn + ((long long)(place * (unsigned)tiles_w) * S::kBand + uq * (S::kU * S::kTh) + (unsigned)qy % S::kTh) * kR;
        } else {
            return attn + (long long)qy * W * kTaps<KS> + uq * KS;
        }
    };
    // In such a row: the slot of query strip sq for column `slot` of its halo band, and a query's weight for key column `key`.
    auto slot_at = [&](const float* row, int sq, int slot) {
        return reinterpret_cast<const float4*>(row) + (long long)((unsigned)sq / S::kStrips) * S::kBand +
               ((unsigned)sq % S::kStrips * (KS * S::kU) + slot) * S::kTh;
    };
    auto weight = [&](const float* row, int q, int key) {
        if constexpr (TILED) return __ldg(reinterpret_cast<const float*>(slot_at(row, q / kR, key - na2d_ws(q / kR * kR, W, KS))) + q % kR);
        else return __ldg(row + (long long)q * kTaps<KS> + key - na2d_ws(q, W, KS));
    };
    // The weights of query strip sq for key column `key` of the image, to shared memory; zeros where a query is outside the image.  PAIRS:
    // nothing is written, and nothing will be read, where none of the strip's windows holds the key.
    auto fetch = [&](float4* to, const float* row, int sq, int key, bool pairs) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (sq >= 0 && kR * sq < W) {
            if constexpr (TILED) {
                const int slot = key - na2d_ws(kR * sq, W, KS);
                const bool in = (unsigned)slot < (unsigned)S::kU;
                if (pairs) {
                    if (in) copy16(to, slot_at(row, sq, slot), true);
                    return;
                }
                if (in) v = __ldg(slot_at(row, sq, slot));
                if (kR * sq + 1 >= W) v.y = 0.f;           // (not written where the query is outside the image)
                if (kR * sq + 2 >= W) v.z = 0.f;
                if (kR * sq + 3 >= W) v.w = 0.f;
            } else {
                float e[kR];
#pragma unroll
                for (int c = 0; c < kR; ++c) {
                    const int member = kR * sq + c < W ? key - na2d_ws(kR * sq + c, W, KS) : -1;
                    e[c] = (unsigned)member < (unsigned)KS ? weight(row, kR * sq + c, key) : 0.f;
                }
                v = make_float4(e[0], e[1], e[2], e[3]);
            }
        }
        *to = v;
    };
    // The group's weights: slots [strip][query row][slot][key row], a thread keeps its slot and key row and goes over the rest (eight key
    // rows of a slot lie side by side, as their query rows do in a query tile's weights); then edge pairs [query row][border][pair][key row].
    auto gather = [&](int g0, int gn) {
        constexpr int kLines = K::kThreads / S::kTh, kPar = kLines / S::kU;            // query rows at a time
        static_assert(kPar > 0, "a line a slot");
        const int ly = threadIdx.x % S::kTh, y = t.y0 + ly, line = threadIdx.x / S::kTh;
        const int first_row = na2d_bws(min(y, H - 1), KS) + g0;
        const int rows_here = ly < t.rows ? min(gn, na2d_bwe(y, H, KS) - first_row) : 0;
        if (K::kEdges || inner) {
            const int j = line % S::kU, d = (j + 4 * KS - kHalf) / kR - KS;            // floor((j - kHalf) / 4): the query strip lies d before the key's
            const int key0 = t.x0 + j - kHalf - kR * d, sq0 = t.x0 / kR - d;
            for (int u = line / S::kU; u < rows_here; u += kPar) {
                if (line >= kPar * S::kU) break;
                const float* row = row_at(first_row + u, y);
#pragma unroll (TILED ? S::kStrips : 1)
                for (int st = 0; st < S::kStrips; ++st) {
                    float4* to = w + ((st * gn + u) * S::kU + j) * S::kTh + ly;
                    if (TILED && inner) copy16(to, slot_at(row, sq0 + st, j), true);
                    else if (key0 + kR * st < W) fetch(to, row, sq0 + st, key0 + kR * st, false);
                }
            }
        } else {
            for (int i = line; i < gn * nj; i += kLines) {
                const int u = i / nj, j = i - u * nj;
                if (u >= rows_here) break;
                const float* row = row_at(first_row + u, y);
#pragma unroll (TILED ? S::kStrips : 1)
                for (int st = 0; st < S::kStrips; ++st) {
                    const int key = t.x0 + kR * st + j % kR;
                    if (key < W) fetch(w + ((st * gn + u) * nj + j) * S::kTh + ly, row, na2d_bws(t.x0 + kR * st, KS) / kR + j / kR, key, true);
                }
            }
        }
        if (!K::kEdges || !(left || right)) return;
        float* edge = reinterpret_cast<float*>(w + gn * K::kRowSlots);
        for (int i = line; i < rows_here * (2 * K::kPairs); i += kLines) {
            const int u = i / (2 * K::kPairs), border = i % (2 * K::kPairs) / K::kPairs, pair = i % K::kPairs;
            int k = 0;
            while ((k + 1) * (k + 2) / 2 <= pair) ++k;
            const int from = kHalf + 1 + k, q = pair - k * (k + 1) / 2, key = border ? W - 1 - from : from;
            if (key < t.x0 || key >= t.x0 + t.cols) continue;
            edge[i * S::kTh + ly] = weight(row_at(first_row + u, y), border ? W - 1 - q : q, key);
        }
    };

    __syncthreads();                                       // the barriers are set up
    for (int ch = 0; ch < g.C; ch += kChunk) {
        Channels acc[K::kRows][kR];
#pragma unroll
        for (int i = 0; i < K::kRows * kR; ++i) acc[i / kR][i % kR] = Channels{0, 0};
        for (int g0 = 0; g0 < nu; g0 += group) {
            const int gn = min(group, nu - g0);
            if (ch == 0 || group < nu) {
                gather(g0, gn);
                copies_done();
                __syncthreads();
            }
            loads.wait(0);
            if (active) {
                int n[K::kRows];                           // query rows in this group
#pragma unroll
                for (int p = 0; p < K::kRows; ++p) n[p] = max(0, min(gn, rows_of[p] - g0));
                const int end = u0[last] - u0[0] + n[last];
                const int first_px = (u0[0] - qy0) * box_w - qx0;        // box place of column 0 of the first query row
                const float4* ws = w + strip * gn * nj * S::kTh + row0;
#pragma unroll 1
                for (int h = 0; h < end; ++h) {
                    const int at = first_px + h * box_w;
                    if (regular) {
                        ulonglong2 x[S::kU];
#pragma unroll
                        for (int j = 0; j < S::kU; ++j) x[j] = quad_at(smem, pixel(at + c0 - kHalf + j) ^ 16 * f);
#pragma unroll
                        for (int p = 0; p < K::kRows; ++p) {
                            const int u = h - (u0[p] - u0[0]);
                            if ((unsigned)u >= (unsigned)n[p]) continue;
                            if (K::kEdges || inner) key_band<S, false>(acc[p], ws + u * (S::kU * S::kTh) + p, x);
                            else key_band<S, true>(acc[p], ws + u * nj * S::kTh + p, x);
                        }
                    } else if constexpr (!K::kEdges) {
                        for (int m = 0; m < strips; ++m) {
                            ulonglong2 x[kR];
#pragma unroll
                            for (int c = 0; c < kR; ++c) x[c] = quad_at(smem, pixel(at + (strip0 + m) * kR + c) ^ 16 * f);
#pragma unroll
                            for (int p = 0; p < K::kRows; ++p) {
                                const int u = h - (u0[p] - u0[0]);
                                if ((unsigned)u >= (unsigned)n[p]) continue;
                                const float4* wr = ws + (u * nj + kR * m) * S::kTh + p;
#pragma unroll
                                for (int r = 0; r < kR; ++r) {
                                    const float4 wt = wr[r * S::kTh];
#pragma unroll
                                    for (int c = 0; c < kR; ++c)
                                        if ((unsigned)(kR * m + c - lo[r]) < (unsigned)n_of[r]) add_scaled(acc[p][r], lane_of(wt, c), x[c]);
                                }
                            }
                        }
                    }
                }
                if (K::kEdges && (left || right)) {
                    const float* edge = reinterpret_cast<const float*>(w + gn * K::kRowSlots) + row0;
#pragma unroll
                    for (int r = 0; r < kR; ++r) {
                        const int key = c0 + r;
                        if (key >= W) break;
#pragma unroll 1
                        for (int border = 0; border < 2; ++border) {
                            const int from = border ? W - 1 - key : key, k = from - kHalf - 1;
                            if (k < 0 || from >= KS) continue;
#pragma unroll 1
                            for (int q = 0; q <= k; ++q) {
                                const float* we = edge + (border * K::kPairs + k * (k + 1) / 2 + q) * S::kTh;
                                const int at = first_px + (border ? W - 1 - q : q);
#pragma unroll
                                for (int p = 0; p < K::kRows; ++p)
#pragma unroll 2
                                    for (int u = 0; u < n[p]; ++u)
                                        add_scaled(acc[p][r], we[u * (2 * K::kPairs * S::kTh) + p],
                                                   quad_at(smem, pixel(at + (u0[p] - u0[0] + u) * box_w) ^ 16 * f));
                            }
                        }
                    }
                }
            }
            const bool more = g0 + group < nu;
            if (more || ch + kChunk < g.C) {
                __syncthreads();
                if (threadIdx.x == 0) load(more ? ch : ch + kChunk, more ? qy0 + g0 + group : qy0);
            }
        }
        if (active && ch + 4 * f < g.C) {
#pragma unroll
            for (int p = 0; p < K::kRows; ++p) {
                if (row0 + p >= t.rows) break;
#pragma unroll
                for (int r = 0; r < kR; ++r)
                    if (c0 + r < W) *reinterpret_cast<float4*>(os + p * job.out.st.h + r * job.out.st.w + ch) = channels(acc[p][r]);
            }
        }
    }
    loads.drain();
}

}  // namespace na2d_box
