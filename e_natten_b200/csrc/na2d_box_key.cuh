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
//
// What bounds it: latencies (eight to sixteen warps an SM issue in half of the cycles) and the FMA pipe.  Against the tiled key sums,
// both sums, us: 4 x 8 x 28 x 30 x 64, window 5 49 -> 32, 9 107 -> 87, 13 211 -> 186; 2 x 200 x 260 x 64, window 5 82 -> 59, 9 164 -> 140, 13 363 -> 290;
// with the dense weights of the pair, 4 x 4 x 64 x 64 x 128, window 5, each 72 -> 55.
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
    // of the band, or whole query strips.  As many rows of that as the room allows that is left beside the blocks an SM holds: with one
    // or two query rows at a time, each with its loads and its gather, a border tile took up to 17 turns at window 9.
    static constexpr int kMaxCols = (max_of((KS - 1) / S::kTw * S::kTw, kLeft * kR) + S::kTw + KS - 1 + kR - 1) / kR * kR;
    static constexpr int kWideW = (kEdges ? kHalf + S::kTw + KS - 1 : kMaxCols) | 1;
    // Tables of the gather: where the group's rows of weights lie, for each key row, and the slots in a row.
    static constexpr int kMaxSlots = S::kStrips * max_of(S::kU, kEdges ? 0 : kMaxStrips * kR);
    static constexpr int kBesides = kSlots * 16 + KS * S::kTh * 8 + kMaxSlots * 8 + S::kBarriers + 1024;
    static constexpr int kBox = S::kHaloH * S::kBoxW * kPixel;
    static constexpr int kFitting = na2d_tile::kSmemPerSm / (whole_kb(kBox) + kBesides);
    static constexpr int kBlocks = kFitting * kThreads > 512 ? 512 / kThreads : kFitting;
    static constexpr int kRoom = (na2d_tile::kSmemPerSm / kBlocks - kBesides) / 1024 * 1024, kFit = kRoom / (kWideW * kPixel);
    static constexpr int kWideH = kFit < S::kHaloH ? kFit : S::kHaloH;
    static constexpr int kWeightsAt = whole_kb(max_of(kBox, kWideH * kWideW * kPixel));
    static constexpr int kRowsAt = kWeightsAt + kSlots * 16, kSlotsAt = kRowsAt + KS * S::kTh * 8;
    static constexpr int kBarriersAt = kSlotsAt + kMaxSlots * 8, kSmem = kBarriersAt + S::kBarriers;
    static_assert(S::kHaloH > kSpan && kWideH > kSpan && kBlocks * (kSmem + 1024) <= na2d_tile::kSmemPerSm, "a query row of each key row fits");
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

// tm_x0, tm_x1: boxes of the two jobs' x, 32 channels, tm_w0, tm_w1: wide ones.  A block sums `span` channels (whole chunks), blockIdx.z
// the how manieth.
template <bool TILED, int KS>
__global__ void __launch_bounds__(KeyShape<Shape<KS>>::kThreads, KeyShape<Shape<KS>>::kBlocks)
key_sum_kernel(const __grid_constant__ CUtensorMap tm_x0, const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_x1,
               const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ KeyOut first, const __grid_constant__ KeyOut second,
               const int span, const ErrorState* __restrict__ errors, const __grid_constant__ Band band, const __grid_constant__ Na2dGeom g) {
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
        if (!bar) return;
        // (each map by its name: one chosen through a pointer may be copied to where TMA cannot read it)
        if (blockIdx.y == 0) {
            if (!wide) na2d_ptx::tma_load_5d(smem, &tm_x0, bar, c0, qx0, row, t.n, t.b);
            else na2d_ptx::tma_load_5d(smem, &tm_w0, bar, c0, qx0, row, t.n, t.b);
        } else {
            if (!wide) na2d_ptx::tma_load_5d(smem, &tm_x1, bar, c0, qx0, row, t.n, t.b);
            else na2d_ptx::tma_load_5d(smem, &tm_w1, bar, c0, qx0, row, t.n, t.b);
        }
    };
    const int ch0 = blockIdx.z * span, ch_end = min(g.C, ch0 + span);
    if (threadIdx.x == 0) load(ch0, qy0);
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
    const int group = min(nu, min(min(KS, K::kSlots / (S::kTh * S::kStrips * nj)), box_h - row_span));

    const int f = threadIdx.x % kF, row0 = threadIdx.x / kF % kGroups * K::kRows, strip = threadIdx.x / (kF * kGroups);
    const bool active = row0 < t.rows && kR * strip < t.cols;
    const int c0 = t.x0 + kR * strip;
    // (strips) query columns of each key: the first one from the first query strip's, and how many
    const bool regular = K::kEdges || (c0 >= KS && c0 + kR <= W - KS);
    const int strip0 = na2d_bws(min(c0, W - 1), KS) / kR;
    int lo[kR], n_of[kR], strips = 0, lo_all = 0, hi_all = 1 << 20;      // every key meets the queries lo_all to hi_all
    if constexpr (!K::kEdges) {
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            lo[r] = c0 + r < W ? na2d_bws(c0 + r, KS) - strip0 * kR : 0;
            const int hi = c0 + r < W ? na2d_bwe(c0 + r, W, KS) - strip0 * kR : 0;
            n_of[r] = hi - lo[r];
            lo_all = max(lo_all, lo[r]);
            hi_all = min(hi_all, hi);
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
    // (dense weights) The slots of the four keys of strip st in query row u, one lane a key and key row: the four keys' weights of a query
    // lie side by side.  As in fetch, zeros where the band leaves the image, and nothing where a pair has no weight.
    auto fetch_strip = [&](int st, int u, int gn, const float* row, int ly, int r) {
        const bool in_band = K::kEdges || inner;
        const int first = t.x0 + kR * st, key = first + r;
        if (key >= W) return;
        const int sq0 = in_band ? first / kR : na2d_bws(first, KS) / kR;               // slots count from this query strip
        const int q0 = in_band ? first - kHalf : kR * sq0;
        const int n = in_band ? S::kU : na2d_bwe(min(first + kR, W) - 1, W, KS) - q0;
        const uint32_t to = na2d_ptx::smem_u32(w + ((st * gn + u) * nj + r) * S::kTh + ly);
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
            const int q = q0 + i, member = key - na2d_ws(q, W, KS);
            const bool pair = in_band ? (unsigned)(i - r) < (unsigned)KS : (unsigned)member < (unsigned)KS, in = q >= 0 && q < W;
            const int slot = in_band ? kHalf - kR * ((q >> 2) - sq0) : kR * ((q >> 2) - sq0);
            const float* from = in ? row + (long long)q * kTaps<KS> + member : row;
            if (pair)                                      // (a copy of no bytes leaves zeros)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + (slot * (S::kTh * kR) + (q & 3)) * 4), "l"(from), "r"(in ? 4 : 0) : "memory");
        }
    };
    // The group's weights: slots [strip][query row][slot][key row] (eight key rows of a slot lie side by side, as their query rows do in a
    // query tile's weights); then edge pairs [query row][border][pair][key row].  Places are worked out once, into tables:
    // worked out for each copy they took a third of the kernel's instructions at windows 9 to 13.
    long long* row_table = reinterpret_cast<long long*>(smem + K::kRowsAt);            // [query row][key row]: from attn, -1 for none
    long long* slot_table = reinterpret_cast<long long*>(smem + K::kSlotsAt);          // [strip][slot]: 8 * (float4 from the row) + its queries in the image
    const int ly = threadIdx.x % S::kTh, line = threadIdx.x / S::kTh;
    constexpr int kLines = K::kThreads / S::kTh;
    auto find_slots = [&] {
        for (int i = threadIdx.x; TILED && i < S::kStrips * nj; i += K::kThreads) {
            const int st = i / nj, j = i - st * nj, first = t.x0 + kR * st;
            int key, sq;
            if (K::kEdges || inner) {
                const int d = (j + 4 * KS - kHalf) / kR - KS;            // floor((j - kHalf) / 4): the query strip lies d before the key's
                key = first + j - kHalf - kR * d;
                sq = first / kR - d;
            } else {
                key = first + j % kR;
                sq = na2d_bws(min(first, W - 1), KS) / kR + j / kR;
            }
            const int slot = key < W && sq >= 0 && kR * sq < W ? key - na2d_ws(kR * sq, W, KS) : -1;
            slot_table[i] = (unsigned)slot < (unsigned)S::kU ? (slot_at(attn, sq, slot) - reinterpret_cast<const float4*>(attn)) * 8 + min(kR, W - kR * sq) : 0;
        }
    };
    auto gather = [&](int g0, int gn) {
        for (int i = threadIdx.x; i < gn * S::kTh; i += K::kThreads) {
            const int y = t.y0 + i % S::kTh, qy = na2d_bws(min(y, H - 1), KS) + g0 + i / S::kTh;
            row_table[i] = y < t.y0 + t.rows && qy < na2d_bwe(y, H, KS) ? row_at(qy, y) - attn : -1;
        }
        __syncthreads();
        if constexpr (TILED) {
            for (int i = line; i < S::kStrips * nj; i += kLines) {
                const long long place = slot_table[i];
                const float* from = attn + (place >> 3) * kR;
                const int queries = (int)place & 7, st = i / nj;
                float4* to = w + (st * gn * nj + i - st * nj) * S::kTh + ly;
                if (!K::kEdges && queries == 0) continue;  // (a pair without weights is not read)
#pragma unroll 4
                for (int u = 0; u < gn; ++u) {
                    const long long row = row_table[u * S::kTh + ly];
                    if (row < 0) break;
                    if (!K::kEdges || queries == kR) {
                        copy16(to + u * nj * S::kTh, from + row, true);
                    } else {                               // zeros where a query is outside the image: nothing was written there
                        float4 v = queries > 0 ? __ldg(reinterpret_cast<const float4*>(from + row)) : make_float4(0.f, 0.f, 0.f, 0.f);
                        if (queries < 2) v.y = 0.f;
                        if (queries < 3) v.z = 0.f;
                        v.w = 0.f;
                        to[u * nj * S::kTh] = v;
                    }
                }
            }
        } else {
            constexpr int kPer = kLines / kR;
            for (int i = line / kR; i < gn * S::kStrips; i += kPer) {
                const long long row = row_table[i / S::kStrips * S::kTh + ly];
                if (row >= 0) fetch_strip(i % S::kStrips, i / S::kStrips, gn, attn + row, ly, line % kR);
            }
        }
        if (!K::kEdges || !(left || right)) return;
        float* edge = reinterpret_cast<float*>(w + gn * K::kRowSlots);
        for (int i = line; i < gn * (2 * K::kPairs); i += kLines) {
            const int u = i / (2 * K::kPairs), border = i % (2 * K::kPairs) / K::kPairs, pair = i % K::kPairs;
            int k = 0;
            while ((k + 1) * (k + 2) / 2 <= pair) ++k;
            const int from = kHalf + 1 + k, q = pair - k * (k + 1) / 2, key = border ? W - 1 - from : from;
            const long long row = row_table[u * S::kTh + ly];
            if (key < t.x0 || key >= t.x0 + t.cols || row < 0) continue;
            edge[i * S::kTh + ly] = weight(attn + row, border ? W - 1 - q : q, key);
        }
    };

    find_slots();
    __syncthreads();                                       // the barriers are set up
    for (int ch = ch0; ch < ch_end; ch += kChunk) {
        Channels acc[K::kRows][kR];
#pragma unroll
        for (int i = 0; i < K::kRows * kR; ++i) acc[i / kR][i % kR] = Channels{0, 0};
        for (int g0 = 0; g0 < nu; g0 += group) {
            const int gn = min(group, nu - g0);
            if (ch == ch0 || group < nu) {
                gather(g0, gn);                            // (waits for the slots' table, too)
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
                                auto add = [&](auto all) {
#pragma unroll
                                    for (int r = 0; r < kR; ++r) {
                                        const float4 wt = wr[r * S::kTh];
#pragma unroll
                                        for (int c = 0; c < kR; ++c)
                                            if (decltype(all)::value || (unsigned)(kR * m + c - lo[r]) < (unsigned)n_of[r])
                                                add_scaled(acc[p][r], lane_of(wt, c), x[c]);
                                    }
                                };
                                if (kR * m >= lo_all && kR * m + kR <= hi_all) add(std::true_type{});
                                else add(std::false_type{});
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
            if (more || ch + kChunk < ch_end) {
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
