// Tiled CUDA-core kernels of the unfused pair (scores, apply); its key-side gradients are key sums.
// Measured on one B200 against the warp-per-pixel kernels: step of 4 x 4 x 64 x 64 x 128, window 5, fp32
// 0.80 -> 0.43 ms, the softmax between the two calls included.  (fp32 rows that start on 16-byte boundaries go to na2d_box.cuh: 0.28 ms.)
#pragma once

#include "na2d_tile.cuh"

namespace na2d_tile {

// ------------------------------------------------------------------------------------ unfused pair
// attn[pixel, member] = x[pixel] . y[member of the pixel's window]
template <typename T, int KS, bool PARK>
__global__ void __launch_bounds__(Shape<KS, false>::kThreads, Shape<KS, false>::kBlocks)
window_dot_kernel(const __grid_constant__ Operand x, const __grid_constant__ Operand y, T* __restrict__ attn,
                  const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS, false>;
    extern __shared__ float4 smem[];
    float4 *w = smem, *own = w + S::kWeights, *halo = own + S::kOwn;
    const Tile t = tile_of_block<S>(g, g.Hq);
    int ky0, kx0, halo_rows;
    query_halo<S>(t, g, ky0, kx0, halo_rows);
    const DotItem d = dot_item<S>(t, g, ky0, kx0);
    float s[kR][S::kU];
    tile_dot<T, S, PARK>(s, x, y, own, halo, t, d, g, ky0, kx0, halo_rows);
    if (d.active) {
        float4* slots = weight_slots<S>(w, d);
#pragma unroll
        for (int j = 0; j < S::kU; ++j)
            if (j % S::kSplit == d.split) slots[j * S::kTh] = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
    }
    __syncthreads();
    const float* wf = reinterpret_cast<const float*>(w);
    for_each_weight<S>(t, g, 0, [&](long long e, int i) { attn[e] = from_f<T>(wf[i]); });
}

// out[pixel] = sum over the window of attn[pixel, member] * y[member]
template <typename T, int KS>
__global__ void __launch_bounds__(Shape<KS, false>::kThreads, Shape<KS, false>::kBlocks)
window_apply_kernel(const T* __restrict__ attn, const __grid_constant__ Operand y, const __grid_constant__ Operand out,
                    const __grid_constant__ Na2dGeom g) {
    using S = Shape<KS, false>;
    extern __shared__ float4 smem[];
    float4 *w = smem, *halo = w + S::kWeights + S::kOwn;
    const Tile t = tile_of_block<S>(g, g.Hq);
    int ky0, kx0, halo_rows;
    query_halo<S>(t, g, ky0, kx0, halo_rows);
    float* wf = reinterpret_cast<float*>(w);
    for_each_weight<S>(t, g, 0, [&](long long e, int i) { wf[i] = to_f<T>(__ldg(attn + e)); });
    tile_apply<T, S>(out, y, w, nullptr, halo, t, g, ky0, kx0, halo_rows, false);
}

}  // namespace na2d_tile
