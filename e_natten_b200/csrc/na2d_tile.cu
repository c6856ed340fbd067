// Launchers of the tiled CUDA-core kernels for one element type.
#include "na2d_tile_entry.h"

#include <initializer_list>

#include "../../include/na2d.h"
#include "na2d_tile.cuh"
#include "na2d_tile_bwd.cuh"
#include "na2d_tile_pair.cuh"
#include "na2d_line.cuh"
#if NA2D_TILE_DT == 0
#include "na2d_box_entry.h"
#endif

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

template <typename S>
Band whole_images(const Na2dGeom& g, int H) {
    const int rows = (H + S::kTh - 1) / S::kTh;
    return Band{0, 0, rows, rows};
}

template <typename... P, typename... A>
int launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return NA2D_ERR_CUDA;
    kernel<<<grid, threads, smem, st>>>(static_cast<P>(args)...);
    return cudaPeekAtLastError() == cudaSuccess ? NA2D_OK : NA2D_ERR_CUDA;
}

// Whether the kernels of na2d_line.cuh take these operands: rows of whole 16-byte pieces that start on 16-byte boundaries and
// are short enough.
bool in_line(const Na2dGeom& g, std::initializer_list<const Tensor*> operands) {
    constexpr long long n = 16 / sizeof(Elem);
    if (g.C % n != 0 || g.C * (int)sizeof(Elem) > na2d_line::max_row(sizeof(Elem))) return false;
    for (const Tensor* t : operands)
        if (reinterpret_cast<uintptr_t>(t->ptr) % 16 != 0 || t->st.b % n != 0 || t->st.n % n != 0 || t->st.w % n != 0) return false;
    return true;
}

#if NA2D_TILE_DT == 0
// fp32 operands that na2d_box.cuh takes go there: run(call) launches.  True with the status, or false where the tiled kernels are to
// take the launch.
template <typename F>
bool in_boxes(const Na2dGeom& g, const Place& at, bool pays, std::initializer_list<const Tensor*> operands, int* rc, F&& run) {
    if (!pays || !na2d_box::takes(g, operands)) return false;
    *rc = run(na2d_box::Call{g, at.device, at.st, at.errors});
    return *rc != na2d_box::kNoMap;
}
#endif

}  // namespace

// ---- how the backward's workspace is shared out -------------------------------------------------------
namespace {

template <typename S> int tile_rows(const Na2dGeom& g) { return (g.Hq + S::kTh - 1) / S::kTh; }
// fp32 values of P and dS of a row of tiles.
template <typename S> long long row_floats(const Na2dGeom& g) {
    return 2ll * ((g.W + S::kTw - 1) / S::kTw) * S::kWeights * kR;
}
// First and last row of query tiles that a row of key tiles reads.
template <typename S> int first_query_row(int row) { return na2d_bws(row * S::kTh, S::kKh) / S::kTh; }
template <typename S> int last_query_row(const Na2dGeom& g, int row) {
    const int last_key = (row + 1) * S::kTh < g.Hkv ? (row + 1) * S::kTh - 1 : g.Hkv - 1;
    return (na2d_bwe(last_key, g.Hg, S::kKh) - 1) / S::kTh;
}
// Tile rows that the weights need at least, one unit at a time.
template <typename S> int least_rows(const Na2dGeom& g) {
    int least = 1;
    for (int row = 0; row < tile_rows<S>(g); ++row) {
        const int n = last_query_row<S>(g, row) - first_query_row<S>(row) + 1;
        if (n > least) least = n;
    }
    return least;
}

}  // namespace

#if NA2D_TILE_DT == 0
long long workspace_floats(const Na2dGeom& g, long long limit) {
    long long floats = 0;
    by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const long long row = row_floats<S>(g), unit = row * tile_rows<S>(g);
        const long long units = limit / unit < g.BN ? limit / unit : g.BN;
        if (units > 0) {
            floats = units * unit;
        } else {
            const long long rows = limit / row, least = least_rows<S>(g);
            floats = row * (rows > least ? rows : least);
        }
        return NA2D_OK;
    });
    return floats;
}

Turns workspace_turns(const Na2dGeom& g, long long floats) {
    Turns t{0, 0};
    by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const long long row = row_floats<S>(g), unit = row * tile_rows<S>(g);
        if (floats >= unit) {
            t = Turns{(int)(floats / unit < g.BN ? floats / unit : g.BN), tile_rows<S>(g)};
        } else if (floats / row >= least_rows<S>(g)) {
            t = Turns{1, (int)(floats / row)};
        }
        return NA2D_OK;
    });
    return t;
}
#endif

int NA2D_NAME(forward)(const Na2dGeom& g, const Place& at, const Tensor& q, const Tensor& k, const Tensor& v,
                       const Tensor& o, float* lse) {
#if NA2D_TILE_DT == 0
    if (int rc = 0; in_boxes(g, at, na2d_box::pays(na2d_box::Work::kForward, g), {&q, &k, &v, &o}, &rc, [&](const na2d_box::Call& c) { return na2d_box::forward(c, q, k, v, o, lse); })) return rc;
#endif
    return by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? fwd_kernel<Elem, S::kKs, S::kOneD, true> : fwd_kernel<Elem, S::kKs, S::kOneD, false>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        if constexpr (S::kOneD) {
            if (in_line(g, {&q, &k, &v, &o}))
                return launch(na2d_line::fwd_kernel<Elem, S::kKs>, n, na2d_line::kThreads, na2d_line::forward_smem<S::kKs>(g.C * sizeof(Elem)),
                              at.st, operand(q, g.C), operand(k, g.C), operand(v, g.C), operand(o, g.C), lse, g);
        }
        return launch(kernel, n, S::kThreads, S::kSmem, at.st, operand(q, g.C), operand(k, g.C),
                      operand(v, g.C), operand(o, g.C), lse, g);
    });
}

int NA2D_NAME(backward_dq)(const Na2dGeom& g, const Place& at, const Tensor& q, const Tensor& k, const Tensor& v,
                           const Tensor& d_o, const Tensor& d_q, const float* lse, float* delta, float* row_factor) {
#if NA2D_TILE_DT == 0
    if (int rc = 0; in_boxes(g, at, na2d_box::pays(na2d_box::Work::kQueryHalf, g), {&q, &k, &v, &d_o, &d_q}, &rc, [&](const na2d_box::Call& c) {
            const int rows = (g.Hq + 7) / 8;
            return na2d_box::query_half(c, q, k, v, d_o, d_q, lse, delta, row_factor, nullptr, nullptr, g.BN, na2d_box::Rows{0, 0, rows, rows});
        }))
        return rc;
#endif
    return by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? dq_kernel<Elem, S::kKs, S::kOneD, true> : dq_kernel<Elem, S::kKs, S::kOneD, false>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        if constexpr (S::kOneD) {
            if (in_line(g, {&q, &k, &v, &d_o, &d_q}))
                return launch(na2d_line::dq_kernel<Elem, S::kKs>, n, na2d_line::kThreads, na2d_line::forward_smem<S::kKs>(g.C * sizeof(Elem)),
                              at.st, operand(q, g.C), operand(k, g.C), operand(v, g.C), operand(d_o, g.C), operand(d_q, g.C), lse, delta,
                              row_factor, (float4*)nullptr, (float4*)nullptr, 0, g);
        }
        return launch(kernel, n, S::kThreads, S::kSmem, at.st, operand(q, g.C), operand(k, g.C),
                      operand(v, g.C), operand(d_o, g.C), operand(d_q, g.C), lse, delta, row_factor, (float4*)nullptr,
                      (float4*)nullptr, whole_images<S>(g, g.Hq), g);
    });
}

int NA2D_NAME(backward)(const Na2dGeom& g, const Place& at, const Tensor& q, const Tensor& k, const Tensor& v,
                        const Tensor& d_o, const Tensor& d_q, const Tensor& d_k, const Tensor& d_v, const float* lse,
                        float* delta, float* workspace, Turns turns, int* launches) {
    return by_window(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? dq_kernel<Elem, S::kKs, S::kOneD, true> : dq_kernel<Elem, S::kKs, S::kOneD, false>;
        using K = KeyShape<S>;
        const int all_rows = tile_rows<S>(g), tiles_w = (g.W + S::kTw - 1) / S::kTw;
        for (long long unit0 = 0; unit0 < g.BN; unit0 += turns.units) {
            const int units = (int)(g.BN - unit0 < turns.units ? g.BN - unit0 : turns.units);
            float4 *p = reinterpret_cast<float4*>(workspace), *ds = p + (long long)units * turns.rows * tiles_w * S::kWeights;
            if constexpr (S::kOneD) {
                static_assert(S::kTw == na2d_line::kTile && S::kWeights == na2d_line::kStrips * na2d_line::kU<S::kKs>, "one layout of the weights");
                if (in_line(g, {&q, &k, &v, &d_o, &d_q, &d_k, &d_v})) {
                    unsigned n = 0;
                    if (int rc = tiles<S>(g, units, 1, &n)) return rc;
                    const int row_bytes = g.C * (int)sizeof(Elem);
                    if (int rc = launch(na2d_line::dq_kernel<Elem, S::kKs>, n, na2d_line::kThreads, na2d_line::forward_smem<S::kKs>(row_bytes), at.st,
                                        operand(q, g.C), operand(k, g.C), operand(v, g.C), operand(d_o, g.C), operand(d_q, g.C), lse, delta,
                                        (float*)nullptr, p, ds, (int)unit0, g))
                        return rc;
                    ++*launches;
                    if (int rc = launch(na2d_line::key_kernel<Elem, S::kKs>, n, na2d_line::kThreads, na2d_line::key_smem<S::kKs>(row_bytes), at.st,
                                        operand(q, g.C), operand(d_o, g.C), operand(d_k, g.C), operand(d_v, g.C), p, ds, (int)unit0, g))
                        return rc;
                    ++*launches;
                    continue;
                }
            }
            const KeySum for_dk{ds, operand(q, g.C), operand(d_k, g.C)}, for_dv{p, operand(d_o, g.C), operand(d_v, g.C)};
            // Query tiles as far as the ring has room without losing a row that the next key tiles read, then the
            // key tiles that have all their queries; in one go where the ring holds the whole image.
            for (int keys = 0, queries = 0; keys < all_rows;) {
                const int room = first_query_row<S>(keys) + turns.rows, query_end = room < all_rows ? room : all_rows;
                int key_end = keys;
                while (key_end < all_rows && last_query_row<S>(g, key_end) < query_end) ++key_end;
                if (key_end == keys) return NA2D_ERR_BAD_ARG;              // a ring below least_rows()
                const Band query_band{(int)unit0, queries, query_end - queries, turns.rows};
                const Band key_band{(int)unit0, keys, key_end - keys, turns.rows};
                unsigned n = 0;
                const auto query_half = [&]() -> int {
#if NA2D_TILE_DT == 0
                    const na2d_box::Rows rows{query_band.unit0, query_band.row0, query_band.rows, query_band.ring};
                    if (int rc = 0; in_boxes(g, at, na2d_box::pays(na2d_box::Work::kQueryHalf, g), {&q, &k, &v, &d_o, &d_q}, &rc, [&](const na2d_box::Call& c) {
                            return na2d_box::query_half(c, q, k, v, d_o, d_q, lse, delta, nullptr, p, ds, units, rows);
                        }))
                        return rc;
#endif
                    if (int rc = tiles<S>(g, units, query_band.rows * S::kTh, &n)) return rc;
                    return launch(kernel, n, S::kThreads, S::kSmem, at.st, operand(q, g.C), operand(k, g.C), operand(v, g.C),
                                  operand(d_o, g.C), operand(d_q, g.C), lse, delta, (float*)nullptr, p, ds, query_band, g);
                };
                const auto key_half = [&]() -> int {
#if NA2D_TILE_DT == 0
                    const na2d_box::Rows rows{key_band.unit0, key_band.row0, key_band.rows, key_band.ring};
                    if (int rc = 0; in_boxes(g, at, na2d_box::pays(na2d_box::Work::kKeySum, g), {&q, &d_o, &d_k, &d_v}, &rc, [&](const na2d_box::Call& c) {
                            return na2d_box::key_half(c, q, d_o, d_k, d_v, p, ds, units, rows);
                        }))
                        return rc;
#endif
                    if (int rc = tiles<S>(g, units, key_band.rows * S::kTh, &n)) return rc;
                    return launch(key_sum_kernel<Elem, float, true, S::kKs, S::kOneD>, dim3(n, 2), K::kThreads, K::kSmem, at.st,
                                  for_dk, for_dv, key_band, g);
                };
                if (query_band.rows > 0) {
                    if (int rc = query_half()) return rc;
                    ++*launches;
                }
                if (int rc = key_half()) return rc;
                ++*launches;
                keys = key_end;
                queries = query_end;
            }
        }
        return NA2D_OK;
    });
}

int NA2D_NAME(pair_dot)(const Na2dGeom& g, const Place& at, const Tensor& x, const Tensor& y, void* attn) {
#if NA2D_TILE_DT == 0
    if (int rc = 0; in_boxes(g, at, na2d_box::pays(na2d_box::Work::kDot, g), {&x, &y}, &rc, [&](const na2d_box::Call& c) { return na2d_box::pair_dot(c, x, y, (float*)attn); })) return rc;
#endif
    return by_size<false>(g, [&](auto shape) -> int {
        using S = decltype(shape);
        const auto kernel = g.C > kParkAbove<S> ? window_dot_kernel<Elem, S::kKs, true> : window_dot_kernel<Elem, S::kKs, false>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        return launch(kernel, n, S::kThreads, S::kSmem, at.st, operand(x, g.C),
                      operand(y, g.C), (Elem*)attn, g);
    });
}

int NA2D_NAME(pair_apply)(const Na2dGeom& g, const Place& at, const void* attn, const Tensor& y, const Tensor& out) {
#if NA2D_TILE_DT == 0
    if (int rc = 0; in_boxes(g, at, na2d_box::pays(na2d_box::Work::kApply, g), {&y, &out}, &rc, [&](const na2d_box::Call& c) { return na2d_box::pair_apply(c, (const float*)attn, y, out); })) return rc;
#endif
    return by_size<false>(g, [&](auto shape) -> int {
        using S = decltype(shape);
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hq, &n)) return rc;
        return launch(window_apply_kernel<Elem, S::kKs>, n, S::kThreads, S::kSmem, at.st, (const Elem*)attn,
                      operand(y, g.C), operand(out, g.C), g);
    });
}

int NA2D_NAME(pair_inverse)(const Na2dGeom& g, const Place& at, const void* attn, const Tensor& x, const Tensor& out) {
#if NA2D_TILE_DT == 0
    if (int rc = 0; in_boxes(g, at, na2d_box::pays(na2d_box::Work::kKeySum, g), {&x, &out}, &rc, [&](const na2d_box::Call& c) { return na2d_box::pair_inverse(c, (const float*)attn, x, out); })) return rc;
#endif
    return by_size<false>(g, [&](auto shape) -> int {
        using S = decltype(shape);
        using K = KeyShape<S>;
        unsigned n = 0;
        if (int rc = tiles<S>(g, g.BN, g.Hkv, &n)) return rc;
        const KeySum sum{attn, operand(x, g.C), operand(out, g.C)};
        return launch(key_sum_kernel<Elem, Elem, false, S::kKs, false>, n, K::kThreads, K::kSmem, at.st, sum, sum, whole_images<S>(g, g.Hkv), g);
    });
}

}  // namespace na2d_tile
