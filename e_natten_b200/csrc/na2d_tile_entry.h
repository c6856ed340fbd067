// Host entry points of the tiled CUDA-core kernels, compiled in one translation unit per element type
// (na2d_tile.cu with -DNA2D_TILE_DT=0 fp32, 1 bf16, 2 fp16).
#pragma once

#include <cuda_runtime.h>

#include "na2d_index.cuh"

namespace na2d_tile {

// A tensor as the caller describes it, strides resolved.
struct Tensor {
    void* ptr;
    Na2dStride st;
};

// Kernel sizes the tiled kernels are built for.  They are the faster ones at every size of these, down to a few tiles
// (1 x 2 x 16 x 16 x 32, window 5, fp32: forward 23 -> 19 us).  From 15 on a tile would take 139 KB and leave one block per SM: that
// wants another shape, which is not built.
inline bool supported(int ks) { return ks == 3 || ks == 5 || ks == 7 || ks == 9 || ks == 11 || ks == 13; }

// fp32 values of P and dS that the backward of one unit hands from its query half to its key half.
long long workspace_floats(const Na2dGeom& g);

// backward: both halves, for whole images; the workspace holds workspace_floats() of `units` units, which
// are taken that many at a time.
// Status: 0, NA2D_ERR_TOO_LARGE (grid), or NA2D_ERR_CUDA (the launch's error is left for cudaGetLastError).
#define NA2D_TILE_ENTRIES(suffix)                                                                                     \
    int forward_##suffix(const Na2dGeom& g, cudaStream_t st, const Tensor& q, const Tensor& k, const Tensor& v,       \
                         const Tensor& o, float* lse);                                                                \
    int backward_dq_##suffix(const Na2dGeom& g, cudaStream_t st, const Tensor& q, const Tensor& k, const Tensor& v,   \
                             const Tensor& d_o, const Tensor& d_q, const float* lse, float* delta);                   \
    int backward_##suffix(const Na2dGeom& g, cudaStream_t st, const Tensor& q, const Tensor& k, const Tensor& v,      \
                          const Tensor& d_o, const Tensor& d_q, const Tensor& d_k, const Tensor& d_v,                 \
                          const float* lse, float* delta, float* workspace, int units, int* launches);                \
    int pair_dot_##suffix(const Na2dGeom& g, cudaStream_t st, const Tensor& x, const Tensor& y, void* attn);          \
    int pair_apply_##suffix(const Na2dGeom& g, cudaStream_t st, const void* attn, const Tensor& y, const Tensor& out); \
    int pair_inverse_##suffix(const Na2dGeom& g, cudaStream_t st, const void* attn, const Tensor& x, const Tensor& out);
NA2D_TILE_ENTRIES(f32)
NA2D_TILE_ENTRIES(bf16)
NA2D_TILE_ENTRIES(f16)
#undef NA2D_TILE_ENTRIES

}  // namespace na2d_tile
