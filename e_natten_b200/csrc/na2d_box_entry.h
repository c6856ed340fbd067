// Host entry points of the box kernels (na2d_box.cuh, na2d_box_key.cuh): fp32 tensors of the 2D operator and the unfused pair.
#pragma once

#include <initializer_list>

#include "na2d_ptx.cuh"
#include "na2d_tile_entry.h"

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

// Whether these kernels pay for an image's width.  Where every tile meets a border they do little less than the tiled ones: forward /
// dQ of 16 x 8 x 14 x 14 x 64, window 11, 70 -> 72 / 104 -> 106 us, window 13 100 -> 116 / 147 -> 175 (4 x 8 x 28 x 30 x 64 102 -> 103 / 152 -> 163; 4 x 33 x 40 x 32
// 22.5 -> 20.5 / 30 -> 29), key sums at window 7 74 -> 77 (17 columns 49 -> 48).
inline bool query_side_pays(const Na2dGeom& g) { return g.W >= (g.ks == 13 ? 36 : g.ks == 11 ? 16 : 0); }
inline bool key_side_pays(const Na2dGeom& g) { return g.ks != 7 || g.W >= 16; }

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
