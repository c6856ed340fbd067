// Column strips of a query tile's halo box, for the kernels of the larger windows.
//
// The halo box of a TH x TW query tile is cut into strips of STRIP columns and all box rows.  A warp's 32 queries (four image
// rows) see ks + 3 of the box rows: the same part of every strip.  Of chunks of whole box rows some warps see everything
// and others nothing, and as a chunk's MMAs wait for all of its warps it lasts as long as the busiest one.  The rows of a
// strip that a query sees are one range of columns of S, and STRIP divides 16, so a mask is a few operations per 16
// columns.
#pragma once

namespace na2d_tc {

// The last strip starts earlier where the strips would reach past the box; it takes no part of the columns it shares with
// the one before.
template <int D, int KS, int STRIP>
struct StripCfg {
    static_assert(STRIP == 2 || STRIP == 4 || STRIP == 8, "the column pattern of a strip must divide 16");
    static constexpr int HH = TH + KS - 1, BOX_W = TW + KS - 1;    // halo box
    static constexpr int HW = STRIP;                               // columns of a strip
    static constexpr int NCH = (BOX_W + STRIP - 1) / STRIP;        // strips of a tile
    static constexpr int NK = HH * STRIP;                          // keys of a strip, key (r, c) at r * STRIP + c
    static constexpr int NKP = (NK + 15) / 16 * 16;                // padded to the UMMA granularity
    static constexpr int NS = (D + 63) / 64;                       // channel slabs
    static constexpr int SLAB_C = D < 64 ? D : 64;
    static constexpr int ROWB = SLAB_C * 2;
    static constexpr uint32_t SWZ = ROWB == 128 ? 2u : 4u;         // descriptor swizzle code
    static constexpr int ATOM = 8 * ROWB;
    static constexpr int Q_SLAB = TM * ROWB, Q_BYTES = NS * Q_SLAB;
    static constexpr int KV_SLAB = NKP * ROWB, KV_BYTES = NS * KV_SLAB;
    static constexpr uint32_t REP = STRIP == 8 ? 0x0101u : STRIP == 4 ? 0x1111u : 0x5555u;   // column 0 of every row in 16 columns
    static_assert(KV_SLAB % 1024 == 0 && Q_SLAB % 1024 == 0, "slabs must keep the swizzle alignment");

    static __device__ __forceinline__ int first_col(int c) { return min(c * STRIP, BOX_W - STRIP); }
    // Columns of strip c (bit i: column i) that a query sees whose window columns are the bits of `window` (of the box).
    static __device__ __forceinline__ uint32_t seen_cols(uint32_t window, int c) {
        return ((window >> (c * STRIP)) << (c * STRIP - first_col(c))) & ((1u << STRIP) - 1u);
    }
};

}  // namespace na2d_tc
