// Host entry points of the tiled CUDA-core kernels, compiled in one translation unit per element type
// (na2d_tile.cu with -DNA2D_TILE_DT=0 fp32, 1 bf16, 2 fp16).
#pragma once

#include <cuda_runtime.h>

#include "na2d_index.cuh"
#include "na2d_ptx.cuh"

namespace na2d_tile {

// A tensor as the caller describes it, strides resolved.
struct Tensor {
    void* ptr;
    Na2dStride st;
};

// Kernel sizes the tiled kernels are built for; na2d_tile_rule.h says which calls of these they take.  From 15 on a tile
// would take 139 KB and leave one block per SM: that wants another shape, which is not built.
inline bool supported(int ks) { return ks == 3 || ks == 5 || ks == 7 || ks == 9 || ks == 11 || ks == 13; }

// How the backward hands P and dS from its query half to its key half: `units` (batch, head) units at a time, for each of
// which a workspace has room for `rows` rows of tiles.  Where that is not the whole image, units is 1, and the halves
// take turns, the rows of the workspace being used again as the key half is done with them.
struct Turns {
    int units, rows;
};
// fp32 values of workspace that the backward asks for: all of P and dS up to `limit` values, else as many whole
// units, or whole rows of tiles of one unit, as fit (but no fewer than a row of key tiles reads: the weights of at most
// 32 image rows; a one-row image cannot be cut).
long long workspace_floats(const Na2dGeom& g, long long limit);
// The turns a workspace of so many values allows; units is 0 if it is too small for any.
Turns workspace_turns(const Na2dGeom& g, long long floats);

// Where a launch runs: fp32 kernels fed by TMA report waits that gave up to `errors`.
struct Place {
    int device;
    cudaStream_t st;
    const na2d_ptx::ErrorState* errors;
};

// backward_dq: row_factor (or null) takes what the key half multiplies each row's exp(s - lse) by.
// backward: both halves, for whole images.
// Status: 0, NA2D_ERR_TOO_LARGE (grid), or NA2D_ERR_CUDA (the launch's error is left for cudaGetLastError).
#define NA2D_TILE_ENTRIES(suffix)                                                                                     \
    int forward_##suffix(const Na2dGeom& g, const Place& at, const Tensor& q, const Tensor& k, const Tensor& v,       \
                         const Tensor& o, float* lse);                                                                \
    int backward_dq_##suffix(const Na2dGeom& g, const Place& at, const Tensor& q, const Tensor& k, const Tensor& v,   \
                             const Tensor& d_o, const Tensor& d_q, const float* lse, float* delta, float* row_factor);                   \
    int backward_##suffix(const Na2dGeom& g, const Place& at, const Tensor& q, const Tensor& k, const Tensor& v,      \
                          const Tensor& d_o, const Tensor& d_q, const Tensor& d_k, const Tensor& d_v,                 \
                          const float* lse, float* delta, float* workspace, Turns turns, int* launches);                \
    int pair_dot_##suffix(const Na2dGeom& g, const Place& at, const Tensor& x, const Tensor& y, void* attn);          \
    int pair_apply_##suffix(const Na2dGeom& g, const Place& at, const void* attn, const Tensor& y, const Tensor& out); \
    int pair_inverse_##suffix(const Na2dGeom& g, const Place& at, const void* attn, const Tensor& x, const Tensor& out);
NA2D_TILE_ENTRIES(f32)
NA2D_TILE_ENTRIES(bf16)
NA2D_TILE_ENTRIES(f16)
#undef NA2D_TILE_ENTRIES

}  // namespace na2d_tile
