// Host entry points of the box kernels (na2d_box.cuh, na2d_box_key.cuh): fp32 tensors of the 2D operator and the unfused pair.
#pragma once

#include <initializer_list>

#include "na2d_ptx.cuh"
#include "na2d_tile_entry.h"
#include "na2d_tile_rule.h"

namespace na2d_box {

// What a launch gets besides its tensors.
struct Call {
    const Na2dGeom& g;
    int device;
    cudaStream_t st;
    const na2d_ptx::ErrorState* errors;
};

// A launcher's status besides those of na2d.h: no tensor map describes an operand; nothing was launched, and the tiled kernels, which
// take any strides and hand the same weights on, take the launch.
constexpr int kNoMap = 1;

// Whether these operands are rows that start on 16-byte boundaries, as tensor maps and float4 stores want them.
inline bool takes(const Na2dGeom& g, std::initializer_list<const na2d_tile::Tensor*> operands) {
    if (g.kh == 1 || g.C % 4 != 0) return false;
    for (const na2d_tile::Tensor* t : operands) {
        if (t->ptr == nullptr) continue;
        if (reinterpret_cast<uintptr_t>(t->ptr) % 16 != 0) return false;
        for (long long s : {t->st.b, t->st.n, t->st.h, t->st.w})
            if (s <= 0 || s % 4 != 0 || s >= (1ll << 38)) return false;
    }
    return true;
}

// Whether these kernels pay.  By the whole image's rows, so that a band of them is computed as the image is.
// Where every tile meets a border they do little less than the tiled ones: forward /
// dQ of 16 x 8 x 14 x 14 x 64, window 11, 70 -> 72 / 104 -> 106 us, window 13 100 -> 116 / 147 -> 175 (4 x 8 x 28 x 30 x 64 102 -> 103 / 152 -> 163),
// key sums at window 7 74 -> 77 (17 columns 49 -> 48).
// At window 13 one image row per thread is all that fits the registers, and what the boxes gain shows with many tiles to a SM only, sooner with
// one chunk of channels or where half of each row's last tile is idle (the boxes' threads skip it).  Speed against the tiled kernels, one
// B200, 64 and 128 channels, by tiles (whole: 64 x 64, 28 x 40, 30 x 128, 39 x 45, 256 x 256; half: 50 x 52, 100 x 90, 200 x 260):
//                           64 - 256       300 - 640      720 - 1440     1536 - 2475
//   forward, whole          0.90 - 1.02    0.93 - 1.05    0.99 - 1.10    1.01 - 1.10
//   forward, half           0.98 - 1.07    1.03 - 1.11    1.04 - 1.11    1.08 - 1.13
//   dQ alone, whole         0.83 - 1.00    0.86 - 1.03    0.95 - 1.14    0.99 - 1.03
//   dQ alone, half          0.93 - 0.97    0.97 - 1.07    1.02 - 1.10    1.05 - 1.16
// and 32 channels 0.92 - 1.02 up to 256 tiles, beyond forward 1.00 - 1.20, dQ 0.98 - 1.17.  The whole backward, where the query half writes
// P and dS as well (and which dQ alone has to agree with bit for bit), is at 1.02 to 1.21 with the boxes' halves from 300 tiles on.
// The pair's scores 0.93 to 1.34 everywhere; its apply 1.00 to 2.2 up to 98 tiles, whose channels are split over blocks, from 120 on
// 0.82 to 1.03 (147 tiles of 50 x 52 1.07 and 1.18).  At window 11 the forward is at 0.96 to 1.00 where 192 to 256 tiles, two blocks for
// some SMs and no second wave, are all whole, and at 1.01 to 1.2 elsewhere.
using na2d_tile::Work;
inline bool pays(Work work, const Na2dGeom& g) {
    if (work == Work::kKeySum) return g.ks != 7 || g.W >= 16;
    if (g.ks < 11) return true;
    const long long tiles = (long long)g.BN * ((g.Hg + 7) / 8) * ((g.W + 7) / 8);
    if (g.ks == 11) return g.W >= 16 && (work != Work::kForward || g.Hg % 8 != 0 || g.W % 8 != 0 || tiles <= 148 || tiles > 296);
    if (g.W < 36) return false;
    if (work == Work::kDot) return true;
    if (work == Work::kApply) return tiles <= 100;
    const bool soon = g.C <= 32 || (g.W % 8 >= 1 && g.W % 8 <= 4);
    return tiles > (soon ? 2 : 5) * 148;
}

// Query tiles a launch covers, and where it puts their weights: na2d_tile::Band.
struct Rows {
    int unit0, row0, rows, ring;
};
int forward(const Call& c, const na2d_tile::Tensor& q, const na2d_tile::Tensor& k, const na2d_tile::Tensor& v, const na2d_tile::Tensor& o,
            float* lse);
// units: (batch, head) units of the launch, from rows.unit0 on; p, ds: where the weights go (or null).
int query_half(const Call& c, const na2d_tile::Tensor& q, const na2d_tile::Tensor& k, const na2d_tile::Tensor& v, const na2d_tile::Tensor& d_o,
               const na2d_tile::Tensor& d_q, const float* lse, float* delta, float* row_factor, float4* p, float4* ds, int units, const Rows& rows);
// dK of q and ds, dV of d_o and p.
int key_half(const Call& c, const na2d_tile::Tensor& q, const na2d_tile::Tensor& d_o, const na2d_tile::Tensor& d_k, const na2d_tile::Tensor& d_v,
             const float4* p, const float4* ds, int units, const Rows& rows);
int pair_dot(const Call& c, const na2d_tile::Tensor& x, const na2d_tile::Tensor& y, float* attn);
int pair_apply(const Call& c, const float* attn, const na2d_tile::Tensor& y, const na2d_tile::Tensor& out);
int pair_inverse(const Call& c, const float* attn, const na2d_tile::Tensor& x, const na2d_tile::Tensor& out);

}  // namespace na2d_box
