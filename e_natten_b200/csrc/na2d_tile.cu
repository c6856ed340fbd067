// Launchers of the tiled CUDA-core kernels for one element type.
#include "na2d_tile_entry.h"

#include "../../include/na2d.h"
#include "na2d_tile.cuh"
#include "na2d_tile_bwd.cuh"
#include "na2d_tile_pair.cuh"

#if NA2D_TILE_DT == 0
using Elem = float;
#define NA2D_NAME(f) f##_f32
#elif NA2D_TILE_DT == 1
using Elem = __nv_bfloat16;
#define NA2D_NAME(f) f##_bf16
#else
using Elem = __half;
#define NA2D_NAME(f) f##_f16
#endif

namespace na2d_tile {
namespace {

// Four neighbouring channels can be moved at once: rows start on a boundary of four elements and hold a
// multiple of four.
Operand operand(const Tensor& t, int C) {
    const size_t quad = 4 * sizeof(Elem);
    const bool vec = reinterpret_cast<uintptr_t>(t.ptr) % quad == 0 && C % 4 == 0 && t.st.b % 4 == 0 && t.st.n % 4 == 0 &&
                     t.st.h % 4 == 0 && t.st.w % 4 == 0;
    return Operand{t.ptr, t.st, vec ? 1 : 0};
}

// Calls f(Shape) for the window size, of the 2D operator and the pair or of one-row images.
template <bool ONE_D, typename F>
int by_size(const Na2dGeom& g, F&& f) {
    switch (g.ks) {
        case 3: return f(Shape<3, ONE_D>{});
        case 5: return f(Shape<5, ONE_D>{});
        case 7: return f(Shape<7, ONE_D>{});
        case 9: return f(Shape<9, ONE_D>{});
        case 11: return f(Shape<11, ONE_D>{});
        case 13: return f(Shape<13, ONE_D>{});
        default: return NA2D_ERR_UNSUPPORTED;
    }
}
template <typename F>
int by_window(const Na2dGeom& g, F&& f) {
    return g.kh == 1 ? by_size<true>(g, f) : by_size<false>(g, f);
}

template <typename S>
int tiles(const Na2dGeom& g, int units, int H, unsigned* n) {
    const long long t = (long long)units * ((H + S::kTh - 1) / S::kTh) * ((g.W + S::kTw - 1) / S::kTw);
    if (t > 0x7fffffffLL) return NA2D_ERR_TOO_LARGE;
    *n = (unsigned)t;
    return NA2D_OK;
}

template <typename... P, typename... A>
int launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return NA2D_ERR_CUDA;
    kernel<<<grid, threads, smem, st>>>(static_cast<P>(args)...);
    return cudaPeekAtLastError() == cudaSuccess ? NA2D_OK : NA2D_ERR_CUDA;
}

}  // namespace

#if NA2D_TILE_DT == 0
long long workspace_floats(const Na2dGeom& g) {
    long long floats = 0;
    by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        floats = 2ll * ((g.Hq + S::kTh - 1) / S::kTh) * ((g.W + S::kTw - 1) / S::kTw) * S::kWeights * kR;
        return NA2D_OK;
    });
    return floats;
}
#endif

int NA2D_NAME(forward)(const Na2dGeom& g, cudaStream_t st, const Tensor& q, const Tensor& k, const Tensor& v,
                       const Tensor& o, float* lse) {
    return by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? fwd_kernel<Elem, S::kKs, S::kOneD, true> : fwd_kernel<Elem, S::kKs, S::kOneD, false>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        return launch(kernel, n, S::kThreads, S::kSmem, st, operand(q, g.C), operand(k, g.C),
                      operand(v, g.C), operand(o, g.C), lse, g);
    });
}

int NA2D_NAME(backward_dq)(const Na2dGeom& g, cudaStream_t st, const Tensor& q, const Tensor& k, const Tensor& v,
                           const Tensor& d_o, const Tensor& d_q, const float* lse, float* delta) {
    return by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? dq_kernel<Elem, S::kKs, S::kOneD, true> : dq_kernel<Elem, S::kKs, S::kOneD, false>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        return launch(kernel, n, S::kThreads, S::kSmem, st, operand(q, g.C), operand(k, g.C),
                      operand(v, g.C), operand(d_o, g.C), operand(d_q, g.C), lse, delta, (float4*)nullptr,
                      (float4*)nullptr, 0, g);
    });
}

int NA2D_NAME(backward)(const Na2dGeom& g, cudaStream_t st, const Tensor& q, const Tensor& k, const Tensor& v,
                        const Tensor& d_o, const Tensor& d_q, const Tensor& d_k, const Tensor& d_v, const float* lse,
                        float* delta, float* workspace, int units, int* launches) {
    return by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? dq_kernel<Elem, S::kKs, S::kOneD, true> : dq_kernel<Elem, S::kKs, S::kOneD, false>;
        using K = KeyShape<S>;
        for (int unit0 = 0; unit0 < g.BN; unit0 += units) {
            const int here = g.BN - unit0 < units ? g.BN - unit0 : units;
            float4 *p = reinterpret_cast<float4*>(workspace), *ds = p + workspace_floats(g) / 8 * here;
            unsigned n = 0;
            if (int rc = tiles<S>(g, here, g.Hq, &n)) return rc;
            if (int rc = launch(kernel, n, S::kThreads, S::kSmem, st, operand(q, g.C),
                                operand(k, g.C), operand(v, g.C), operand(d_o, g.C), operand(d_q, g.C), lse, delta, p, ds,
                                unit0, g))
                return rc;
            ++*launches;
            const KeySum for_dk{ds, operand(q, g.C), operand(d_k, g.C)}, for_dv{p, operand(d_o, g.C), operand(d_v, g.C)};
            if (int rc = launch(key_sum_kernel<Elem, float, true, S::kKs, S::kOneD>, dim3(n, 2), K::kThreads, K::kSmem, st, for_dk,
                                for_dv, unit0, g))
                return rc;
            ++*launches;
        }
        return NA2D_OK;
    });
}

int NA2D_NAME(pair_dot)(const Na2dGeom& g, cudaStream_t st, const Tensor& x, const Tensor& y, void* attn) {
    return by_size<false>(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? window_dot_kernel<Elem, S::kKs, true> : window_dot_kernel<Elem, S::kKs, false>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        return launch(kernel, n, S::kThreads, S::kSmem, st, operand(x, g.C),
                      operand(y, g.C), (Elem*)attn, g);
    });
}

int NA2D_NAME(pair_apply)(const Na2dGeom& g, cudaStream_t st, const void* attn, const Tensor& y, const Tensor& out) {
    return by_size<false>(g, [&](auto shape) -> int {
        using S = decltype(shape);
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        return launch(window_apply_kernel<Elem, S::kKs>, n, S::kThreads, S::kSmem, st, (const Elem*)attn,
                      operand(y, g.C), operand(out, g.C), g);
    });
}

int NA2D_NAME(pair_inverse)(const Na2dGeom& g, cudaStream_t st, const void* attn, const Tensor& x, const Tensor& out) {
    return by_size<false>(g, [&](auto shape) -> int {
        using S = decltype(shape);
        using K = KeyShape<S>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hkv, &n)) return rc;
        const KeySum sum{attn, operand(x, g.C), operand(out, g.C)};
        return launch(key_sum_kernel<Elem, Elem, false, S::kKs, false>, n, K::kThreads, K::kSmem, st, sum, sum, 0, g);
    });
}

}  // namespace na2d_tile
