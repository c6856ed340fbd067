// C ABI of libna2d.so (declared in include/na2d.h): argument checking, device selection and
// dispatch to the tcgen05, tiled CUDA-core or warp-per-pixel (SIMT) kernels.  No framework headers; plain pointers and sizes.
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "../../include/na2d.h"
#include "na2d_delta.cuh"
#include "na2d_index.cuh"
#include "na2d_simt.cuh"
#include "na2d_tc_entry.h"
#include "na2d_tile_entry.h"
#include "na2d_tile_rule.h"

namespace {

std::atomic<long long> g_launches{0};
thread_local char t_cuda_err[256] = "";

int cuda_fail(cudaError_t e, const char* what) {
    snprintf(t_cuda_err, sizeof(t_cuda_err), "%s: %s", what, cudaGetErrorString(e));
    return NA2D_ERR_CUDA;
}

// Failure of a tcgen05 launcher: either a runtime error or a failed tensor-map encode (a driver call).
int tc_fail(const char* what) {
    int& drv = na2d_tc::last_driver_result();
    if (drv != 0) {
        snprintf(t_cuda_err, sizeof(t_cuda_err), "%s: cuTensorMapEncodeTiled failed with CUresult %d", what, drv);
        drv = 0;
        return NA2D_ERR_CUDA;
    }
    return cuda_fail(cudaGetLastError(), what);
}

#define NA2D_CUDA(call)                                        \
    do {                                                       \
        cudaError_t e__ = (call);                              \
        if (e__ != cudaSuccess) return cuda_fail(e__, #call);  \
    } while (0)

// Makes `device` current for the scope and restores the previous device afterwards.
// cudaSetDevice is called even when `device` already is the thread's current device: a thread that
// has made no runtime call yet (an autograd worker thread, for one) reports device 0 as current
// without having its context bound, and the driver call that encodes tensor maps needs a bound
// context.
struct DeviceScope {
    int prev = -1;
    cudaError_t err = cudaSuccess;
    explicit DeviceScope(int device) {
        err = cudaGetDevice(&prev);
        if (err == cudaSuccess) err = cudaSetDevice(device);
    }
    ~DeviceScope() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

constexpr int kMaxDevices = 64;

// Compute-capability check, cached per device.
int check_device(int device) {
    static std::mutex mu;
    static int state[kMaxDevices];   // 0 unknown, 1 ok, 2 not sm_100
    if (device < 0 || device >= kMaxDevices) return NA2D_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(mu);
    if (state[device] == 0) {
        int major = 0;
        cudaError_t e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
        if (e != cudaSuccess) { cuda_fail(e, "cudaDeviceGetAttribute"); return NA2D_ERR_NO_DEVICE; }
        state[device] = (major == 10) ? 1 : 2;
    }
    return state[device] == 1 ? NA2D_OK : NA2D_ERR_NO_DEVICE;
}

// ---- error state ---------------------------------------------------------------------------------
// What the waits of a device's kernels report to, and their limit; kernels get its address as an argument.  A wait that
// gives up marks its kind in a pinned host word, a byte for each: na2d_poll looks there, which costs no CUDA call (a copy of a device
// word and an event per backward took 8 us of a small call, and a slot between its kernels).  The limit, in microseconds, 0 =
// the built-in 4 s, comes from the environment variable NA2D_WAIT_LIMIT_US: a profiler pass that instruments every instruction
// can stretch a healthy hand-over past the built-in limit (seen under `ncu --set full`).
__device__ na2d_ptx::ErrorState g_errors;

struct Errors {
    const na2d_ptx::ErrorState* device = nullptr;
    volatile unsigned int* word = nullptr;
};
std::atomic<volatile unsigned int*> g_error_words[kMaxDevices];     // null until the device's state is set up

// The kinds in a device's error word, which it clears: bit i for byte i.  Each is seen by one caller, and one that is written
// meanwhile by the next.
unsigned int take_errors(volatile unsigned int* word) {
    if (*word == 0) return 0;
    const unsigned int bytes = __atomic_exchange_n(word, 0u, __ATOMIC_ACQ_REL);
    unsigned int kinds = 0;
    for (int i = 0; i < 4; ++i) kinds |= ((bytes >> (8 * i)) & 1u) << i;
    return kinds;
}

// The error state of `device` (which must be current), set up once per device; that may happen while a stream is being captured,
// so it stays off the streams of others.
int error_state(int device, Errors* out) {
    static std::mutex mu;
    static Errors cache[kMaxDevices];
    if (device < 0 || device >= kMaxDevices) return NA2D_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(mu);
    if (cache[device].device == nullptr) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        NA2D_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        const int rc = [&]() -> int {
            void *state = nullptr, *host = nullptr;
            cudaStream_t st = nullptr;
            na2d_ptx::ErrorState init{nullptr, 0u, 0u};
            if (const char* env = getenv("NA2D_WAIT_LIMIT_US")) {
                const unsigned long long v = strtoull(env, nullptr, 10);
                if (v > 0 && v <= 0xffffffffull) init.limit_us = (unsigned int)v;
            }
            NA2D_CUDA(cudaGetSymbolAddress(&state, g_errors));
            NA2D_CUDA(cudaHostAlloc(&host, sizeof(unsigned int), cudaHostAllocMapped | cudaHostAllocPortable));
            *static_cast<unsigned int*>(host) = 0;
            cudaError_t e = cudaHostGetDevicePointer((void**)&init.error_bytes, host, 0);
            if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
            if (e == cudaSuccess) {
                e = cudaMemcpyAsync(state, &init, sizeof(init), cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                cudaStreamDestroy(st);
            }
            if (e != cudaSuccess) {
                cudaFreeHost(host);
                return cuda_fail(e, "setting up the error state");
            }
            cache[device] = Errors{static_cast<const na2d_ptx::ErrorState*>(state), static_cast<unsigned int*>(host)};
            g_error_words[device].store(cache[device].word, std::memory_order_release);
            return NA2D_OK;
        }();
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (rc != NA2D_OK) return rc;
    }
    *out = cache[device];
    return NA2D_OK;
}

// The kernel of na2d_selftest_wait_timeout: one thread waits on a barrier nothing completes, once for each kind of wait; the first
// wait lasts its limit, the others end soon.
__global__ void wait_timeout_kernel(const na2d_ptx::ErrorState* errors, unsigned long long limit_ns) {
    __shared__ uint64_t bar;
    __shared__ na2d_ptx::WaitState state;
    if (threadIdx.x == 0) {
        na2d_ptx::wait_state_init(&state, errors, limit_ns);
        state.limit_us = static_cast<uint32_t>(limit_ns / 1000ull);        // the self-test's own limit, whatever is configured
        na2d_ptx::mbar_init(&bar, 1);
        na2d_ptx::mbar_fence_init();
        const na2d_ptx::WaitCtx wctx{&state};
        na2d_ptx::mbar_wait(&bar, 0, wctx, na2d_ptx::kErrLoadWait);
        na2d_ptx::mbar_wait(&bar, 0, wctx, na2d_ptx::kErrMmaWait);
        na2d_ptx::mbar_wait(&bar, 0, wctx, na2d_ptx::kErrOther);
    }
}

// ---- problem description --------------------------------------------------------------------------
struct Tensor {
    void* ptr = nullptr;
    Na2dStride st{0, 0, 0, 0};
};

struct Problem {
    Na2dGeom g;
    int B = 0;
    int dtype = 0;
    bool tensor = false;      // run the tcgen05 kernels
    bool dkdv_f32 = false;    // dK / dV are fp32 tensors
    int sm_margin = 0;        // SMs the persistent kernels leave free
    int device = 0;
    cudaStream_t st = nullptr;
    Tensor q, k, v, o, d_o, d_q, d_k, d_v;
    float* lse = nullptr;
    float* delta = nullptr;
    float* row_factor = nullptr;   // CUDA-core backward: factors of exp(s - lse) on their way to the key half
};

// Strides of one operand: the caller's, or dense (B, N, rows, W, C) when all four are zero.  The
// stride of a dimension of extent 1 never reaches an address, so whatever the caller passed for
// it is replaced by the dense value (frameworks report arbitrary strides there).
Tensor resolve(const na2d_tensor& t, int B, int N, int rows, int W, int C, bool one_d) {
    Tensor r;
    r.ptr = t.ptr;
    const bool dense = t.stride_b == 0 && t.stride_n == 0 && t.stride_h == 0 && t.stride_w == 0;
    r.st.w = (dense || W == 1) ? C : t.stride_w;
    r.st.h = (dense || rows == 1 || one_d) ? (long long)W * r.st.w : t.stride_h;
    r.st.n = (dense || N == 1) ? (long long)rows * r.st.h : t.stride_n;
    r.st.b = (dense || B == 1) ? (long long)N * r.st.n : t.stride_b;
    return r;
}

// What a TMA tensor map needs of an operand: a 16-byte aligned base, strides that are multiples of
// 16 bytes (8 elements of 16 bits) and below 2^40 bytes.
bool tma_compatible(const Tensor& t) {
    if (t.ptr == nullptr) return true;
    if (reinterpret_cast<uintptr_t>(t.ptr) & 15u) return false;
    const long long s[4] = {t.st.b, t.st.n, t.st.h, t.st.w};
    for (long long x : s)
        if (x <= 0 || (x & 7) != 0 || x >= (1ll << 39)) return false;
    return true;
}

// Pixels per block for the SIMT kernels: 64 (eight per warp, neighbouring windows share L1) unless
// that gives fewer than two blocks per SM, where one pixel per warp fills the GPU better.
int simt_patch(long long BN, int H, int W) {
    return na2d_simt::patch_count(BN, H, W, na2d_simt::kPatch) < 2 * 148 ? na2d_simt::kPatchSmall : na2d_simt::kPatch;
}

// na2d_args without the workspace fields, which callers built against an earlier header do not have.
constexpr size_t kArgsBase = offsetof(na2d_args, workspace);

// `key_side`: the call is the key half of the backward, whose key band may be any part of the image
// (each key sums over whichever local queries see it); the other calls need a key band that holds
// every window of the query band.
int make_problem(const na2d_args* a, Problem* out, bool key_side = false) {
    if (!a || a->struct_size < kArgsBase) return NA2D_ERR_BAD_ARG;
    const int B = a->B, N = a->N, H = a->H, W = a->W, C = a->C, ks = a->kernel_size, dtype = a->dtype, path = a->path;
    if (B <= 0 || N <= 0 || H <= 0 || W <= 0 || C <= 0) return NA2D_ERR_BAD_ARG;
    if (ks <= 0 || (ks & 1) == 0) return NA2D_ERR_BAD_ARG;
    if (dtype != NA2D_F32 && dtype != NA2D_BF16 && dtype != NA2D_F16) return NA2D_ERR_UNSUPPORTED;
    if (path != NA2D_PATH_AUTO && path != NA2D_PATH_SIMT && path != NA2D_PATH_TENSOR) return NA2D_ERR_BAD_ARG;
    if (a->op != NA2D_OP_2D && a->op != NA2D_OP_1D) return NA2D_ERR_BAD_ARG;
    if (!(a->scale > 0.f) || !(a->scale < 3.0e38f)) return NA2D_ERR_BAD_ARG;
    if ((long long)B * N > 0x7fffffffLL) return NA2D_ERR_TOO_LARGE;
    const bool one_d = a->op == NA2D_OP_1D;
    Na2dGeom g;
    g.BN = B * N; g.N = N; g.W = W; g.C = C; g.ks = ks; g.kh = one_d ? 1 : ks;
    g.n_magic = na2d_heads_magic(g.BN, N);
    g.scale = a->scale;
    g.sl2 = a->scale * 1.4426950408889634f;
    if (one_d) {
        if (H != 1 || a->rows) return NA2D_ERR_BAD_ARG;
        g.q_row0 = 0; g.Hq = 1; g.kv_row0 = 0; g.Hkv = 1; g.Hg = 1;
        // the reference reads out of range when the sequence is shorter than the window
        // (e_natten/pytorch.py:7-11 goes negative); here that is an error
        if (W < ks) return NA2D_ERR_WINDOW;
    } else {
        const na2d_rows* rows = a->rows;
        if (rows) {
            g.q_row0 = rows->q_row0; g.Hq = rows->Hq; g.kv_row0 = rows->kv_row0; g.Hkv = rows->Hkv;
            g.Hg = rows->H_global;
            if (g.Hq <= 0 || g.Hkv <= 0 || g.Hg <= 0 || g.q_row0 < 0 || g.kv_row0 < 0) return NA2D_ERR_BAD_ARG;
            if (g.q_row0 + g.Hq > g.Hg || g.kv_row0 + g.Hkv > g.Hg) return NA2D_ERR_BAD_ARG;
        } else {
            g.q_row0 = 0; g.Hq = H; g.kv_row0 = 0; g.Hkv = H; g.Hg = H;
        }
        // The reference silently reads garbage when a grid side is below the kernel size
        // (e_natten/pytorch.py:7-11 goes negative); here that is an error.
        if (g.Hg < ks || W < ks) return NA2D_ERR_WINDOW;
        // the key band must hold every window of the query band
        if (!key_side) {
            if (na2d_ws(g.q_row0, g.Hg, ks) < g.kv_row0) return NA2D_ERR_WINDOW;
            if (na2d_ws(g.q_row0 + g.Hq - 1, g.Hg, ks) + ks > g.kv_row0 + g.Hkv) return NA2D_ERR_WINDOW;
        }
    }
    Problem& p = *out;
    p.q = resolve(a->q, B, N, g.Hq, W, C, one_d);
    p.o = resolve(a->o, B, N, g.Hq, W, C, one_d);
    p.d_o = resolve(a->d_o, B, N, g.Hq, W, C, one_d);
    p.d_q = resolve(a->d_q, B, N, g.Hq, W, C, one_d);
    p.k = resolve(a->k, B, N, g.Hkv, W, C, one_d);
    p.v = resolve(a->v, B, N, g.Hkv, W, C, one_d);
    p.d_k = resolve(a->d_k, B, N, g.Hkv, W, C, one_d);
    p.d_v = resolve(a->d_v, B, N, g.Hkv, W, C, one_d);

    bool tc_ok = !one_d && na2d_tc::supported(dtype, C, ks);
    if (tc_ok) {
        for (const Tensor* t : {&p.q, &p.k, &p.v, &p.o, &p.d_o, &p.d_q, &p.d_k, &p.d_v})
            tc_ok = tc_ok && tma_compatible(*t);
    }
    bool tensor = false;
    if (path == NA2D_PATH_TENSOR) {
        if (!tc_ok) return NA2D_ERR_UNSUPPORTED;
        tensor = true;
    } else if (path == NA2D_PATH_AUTO) {
        tensor = tc_ok;
    }
    if (!tensor && (C > na2d_simt::kMaxC || ks > na2d_simt::kMaxKs)) return NA2D_ERR_UNSUPPORTED;
    g.patch = simt_patch(g.BN, g.Hq, W);
    p.g = g; p.B = B; p.dtype = dtype; p.tensor = tensor;
    p.device = a->device; p.st = (cudaStream_t)a->stream;
    p.lse = a->lse; p.delta = a->delta;
    p.dkdv_f32 = (a->flags & NA2D_FLAG_DKDV_F32) != 0 && dtype != NA2D_F32;
    p.sm_margin = (a->flags >> 8) & 0xff;
    if (a->flags & ~(NA2D_FLAG_DKDV_F32 | NA2D_FLAG_SM_MARGIN(0xff))) return NA2D_ERR_BAD_ARG;
    return NA2D_OK;
}

// ---- dispatch helpers -------------------------------------------------------------------------------
template <int V> using IntTag = std::integral_constant<int, V>;
template <typename T> struct TypeTag { using type = T; };

// Calls f(TypeTag<element type>, IntTag<channels per lane>) for the problem's dtype and head dim.
template <typename F>
int simt_dispatch(int dtype, int C, F&& f) {
    auto by_cpl = [&](auto type_tag) -> int {
        if (C <= 32) return f(type_tag, IntTag<1>{});
        if (C <= 64) return f(type_tag, IntTag<2>{});
        if (C <= 128) return f(type_tag, IntTag<4>{});
        return f(type_tag, IntTag<8>{});
    };
    switch (dtype) {
        case NA2D_F32: return by_cpl(TypeTag<float>{});
        case NA2D_BF16: return by_cpl(TypeTag<__nv_bfloat16>{});
        default: return by_cpl(TypeTag<__half>{});
    }
}

// One block per patch of a (BN, H, W) pixel grid.
int grid_for(long long BN, int H, int W, int patch, unsigned* grid) {
    const long long nb = na2d_simt::patch_count(BN, H, W, patch);
    if (nb > 0x7fffffffLL) return NA2D_ERR_TOO_LARGE;
    *grid = (unsigned)nb;
    return NA2D_OK;
}

constexpr int kSimtThreads = na2d_simt::kWarps * 32;

int after_launch() {
    g_launches.fetch_add(1);
    NA2D_CUDA(cudaGetLastError());
    return NA2D_OK;
}

// Whether the tiled kernels take this part of a CUDA-core call.  It goes by the whole image's rows, so that a band of them
// is computed as the image is, bit for bit.
bool in_tiles(na2d_tile::Work work, const Na2dGeom& g, int dtype) {
    return na2d_tile::supported(g.ks) &&
           na2d_tile::faster_in_tiles(work, g.kh == 1, dtype != NA2D_F32, (long long)g.BN * g.Hg * g.W, g.C, g.ks);
}
// The query half by itself; in 2D as the whole backward runs it, for the same reason.
bool query_half_in_tiles(const Na2dGeom& g, int dtype) {
    return in_tiles(na2d_tile::Work::kQueryHalf, g, dtype) || (g.kh > 1 && in_tiles(na2d_tile::Work::kBackward, g, dtype));
}

na2d_tile::Tensor tile(const Tensor& t) { return na2d_tile::Tensor{t.ptr, t.st}; }
// Calls run(place) with where a tiled call's launches run; the fp32 kernels of the 2D operator and the pair get the error state.
template <typename F>
int at_place(int device, cudaStream_t st, int dtype, const Na2dGeom& g, F&& run) {
    Errors err;
    if (dtype == NA2D_F32 && g.kh > 1)
        if (int rc = error_state(device, &err)) return rc;
    return run(na2d_tile::Place{device, st, err.device});
}

// The launcher of the element type.
#define NA2D_TILE_PICK(dtype, name) \
    ((dtype) == NA2D_F32 ? na2d_tile::name##_f32 : (dtype) == NA2D_BF16 ? na2d_tile::name##_bf16 : na2d_tile::name##_f16)

// Status of a tiled-kernel launcher that makes `launches` launches.
int after_tile(int rc, int launches) {
    if (rc == NA2D_OK) g_launches.fetch_add(launches);
    if (rc == NA2D_ERR_CUDA) return cuda_fail(cudaGetLastError(), "tiled kernel launch");
    return rc;
}

na2d_tc::TensorArg targ(const Tensor& t) { return na2d_tc::TensorArg{t.ptr, t.st}; }

// Whether the kernels of a tensor-core call are launched to overlap the end of the kernel before them.  Blocks that wait hold SMs, so not
// for calls that leave some to other streams' kernels (a margin, a band of rows beside its exchange).  And up to kOverlapPixels alone, from
// window 7 on: a launch hides about 2 us, a quarter of the smallest calls' time, 1 to 3 % at the line and at most 1 % at twice as many
// pixels, but kernels of some rounds of tiles last up to 4 us longer when their blocks start as SMs fall free (their places on the
// chip change, so L2's far half is the likely reason).  A step, one B200, bf16, cold L2, us without and with:
//   pixels            8 K - 64 K    125 K - 131 K   200 K         262 K - 280 K   520 K
//   28 x 28 x 64, 13  166.9 157.7   287.7 276.5     398.3 385.0   525.2 510.1     986.1 976.9
//   100^2 x 64, 9     109.6 102.3   152.6 145.4     224.3 221.2   298.0 294.9     513.0 511.9
//   56 x 56 x 32, 7   74.8 67.6     117.5 110.5     164.9 161.8   203.6 196.7     369.7 366.7
//   48 x 48 x 128, 13 171.0 165.9   281.6 278.5     414.9 414.7   510.9 506.0     951.4 950.2
// Replayed from a graph launches lie closer, and the line is at half: 100^2 x 64, window 9, L2 warm 92.4 90.4, 132.1 131.8, 202.9 209.1.
// Windows 3 and 5 in a stream, cold L2, 1.00 to 1.04 times as fast, but 5 as a graph loses from 64 K pixels on (64 x 64 x 128: 72.2 82.5,
// 122.3 136.8), and 1024^2 x 128, window 13, 17.3 17.6 ms.  What it costs: four streams at once, each with steps of its own of 100 K to 175 K
// pixels, are 1 to 2 % slower in all (236.1 241.6, 334.5 339.7 us a step), since a block that waits takes the place of another stream's.
constexpr long long kOverlapPixels = 1 << 18;
bool overlaps(const Problem& p) {
    const Na2dGeom& g = p.g;
    if (g.ks < 7 || p.sm_margin != 0 || g.Hq != g.Hg || g.Hkv != g.Hg) return false;
    const long long pixels = (long long)g.BN * g.Hg * g.W;
    if (pixels > kOverlapPixels) return false;
    if (pixels <= kOverlapPixels / 2) return true;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(p.st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
}

int launch_ctx(const Problem& p, int* launched, na2d_tc::LaunchCtx* lc) {
    Errors err;
    int rc = error_state(p.device, &err);
    if (rc != NA2D_OK) return rc;
    *lc = na2d_tc::LaunchCtx{p.g, p.dtype, p.B, p.device, p.st, err.device, launched, p.dkdv_f32, p.sm_margin, overlaps(p)};
    return NA2D_OK;
}

// ---- the three compute steps ---------------------------------------------------------------------------
int run_forward(const Problem& p) {
    const Na2dGeom& g = p.g;
    if (p.tensor) {
        int launched = 0;
        na2d_tc::LaunchCtx lc;
        int rc = launch_ctx(p, &launched, &lc);
        if (rc != NA2D_OK) return rc;
        rc = p.dtype == NA2D_BF16 ? na2d_tc::forward_bf16(lc, targ(p.q), targ(p.k), targ(p.v), targ(p.o), p.lse)
                                  : na2d_tc::forward_f16(lc, targ(p.q), targ(p.k), targ(p.v), targ(p.o), p.lse);
        g_launches.fetch_add(launched);
        if (rc == NA2D_ERR_CUDA) return tc_fail("tcgen05 forward launch");
        return rc;
    }
    if (in_tiles(na2d_tile::Work::kForward, g, p.dtype)) {
        const auto run = NA2D_TILE_PICK(p.dtype, forward);
        return at_place(p.device, p.st, p.dtype, g, [&](const na2d_tile::Place& at) {
            return after_tile(run(g, at, tile(p.q), tile(p.k), tile(p.v), tile(p.o), p.lse), 1);
        });
    }
    unsigned grid = 0;
    int rc = grid_for(g.BN, g.Hq, g.W, g.patch, &grid);
    if (rc != NA2D_OK) return rc;
    return simt_dispatch(p.dtype, g.C, [&](auto tt, auto cpl) -> int {
        using T = typename decltype(tt)::type;
        na2d_simt::fwd_kernel<T, decltype(cpl)::value>
            <<<grid, kSimtThreads, na2d_simt::window_smem_bytes(g.kh, g.ks, 1), p.st>>>(
                (const T*)p.q.ptr, (const T*)p.k.ptr, (const T*)p.v.ptr, (T*)p.o.ptr, p.lse, p.q.st, p.k.st, p.v.st,
                p.o.st, g);
        return after_launch();
    });
}

// The dO . o estimate of the row deltas, into p.delta (tensor path: head dim 32, 64 or 128, rows on
// 16-byte boundaries).
template <typename T, int LPP>
int launch_delta_as(const Problem& p, bool overlap) {
    const Na2dGeom& g = p.g;
    const long long hw = (long long)g.Hq * g.W;
    const long long per_image = (hw + na2d_delta::pixels_per_block<LPP>() - 1) / na2d_delta::pixels_per_block<LPP>();
    if (hw > 0x7fffffffLL || per_image * g.BN > 0x7fffffffLL) return NA2D_ERR_TOO_LARGE;
    NA2D_CUDA(na2d_launch::launch(overlap, na2d_delta::delta_kernel<T, LPP>, (unsigned)(per_image * g.BN), na2d_delta::kThreads, 0, p.st,
                                  (const T*)p.d_o.ptr, (const T*)p.o.ptr, p.delta, p.d_o.st, p.o.st, g, (unsigned)per_image));
    g_launches.fetch_add(1);
    return NA2D_OK;
}

int launch_delta(const Problem& p, bool overlap) {
    const bool bf = p.dtype == NA2D_BF16;
    switch (p.g.C) {
        case 32: return bf ? launch_delta_as<__nv_bfloat16, 4>(p, overlap) : launch_delta_as<__half, 4>(p, overlap);
        case 64: return bf ? launch_delta_as<__nv_bfloat16, 8>(p, overlap) : launch_delta_as<__half, 8>(p, overlap);
        case 128: return bf ? launch_delta_as<__nv_bfloat16, 16>(p, overlap) : launch_delta_as<__half, 16>(p, overlap);
        default: return NA2D_ERR_UNSUPPORTED;
    }
}

int run_backward_dq(const Problem& p) {
    const Na2dGeom& g = p.g;
    if (p.tensor) {
        int launched = 0;
        na2d_tc::LaunchCtx lc;
        int rc = launch_ctx(p, &launched, &lc);
        if (rc != NA2D_OK) return rc;
        // With the forward's output at hand, the dQ kernel of the larger windows gets an estimate of
        // the row deltas (dO . o) and walks its key box once; it overwrites the estimate with the
        // exact deltas.
        bool have_estimate = false;
        if (g.ks >= 7 && p.o.ptr && p.d_q.ptr) {
            rc = launch_delta(p, lc.overlap);
            if (rc != NA2D_OK) return rc;
            have_estimate = true;
        }
        rc = p.dtype == NA2D_BF16
                 ? na2d_tc::backward_dq_bf16(lc, targ(p.q), targ(p.k), targ(p.v), p.lse, targ(p.d_o), targ(p.d_q), p.delta, have_estimate)
                 : na2d_tc::backward_dq_f16(lc, targ(p.q), targ(p.k), targ(p.v), p.lse, targ(p.d_o), targ(p.d_q), p.delta, have_estimate);
        g_launches.fetch_add(launched);
        if (rc == NA2D_ERR_CUDA) return tc_fail("tcgen05 dQ launch");
        return rc;
    }
    if (query_half_in_tiles(g, p.dtype)) {
        const auto run = NA2D_TILE_PICK(p.dtype, backward_dq);
        return at_place(p.device, p.st, p.dtype, g, [&](const na2d_tile::Place& at) {
            return after_tile(run(g, at, tile(p.q), tile(p.k), tile(p.v), tile(p.d_o), tile(p.d_q), p.lse, p.delta, p.row_factor), 1);
        });
    }
    unsigned grid = 0;
    int rc = grid_for(g.BN, g.Hq, g.W, g.patch, &grid);
    if (rc != NA2D_OK) return rc;
    return simt_dispatch(p.dtype, g.C, [&](auto tt, auto cpl) -> int {
        using T = typename decltype(tt)::type;
        const auto kernel = na2d_simt::dq_kernel<T, decltype(cpl)::value>;
        const size_t smem = na2d_simt::window_smem_bytes(g.kh, g.ks, 2);
        if (smem > 48 * 1024)                      // kernel sizes 29 and 31
            NA2D_CUDA(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<grid, kSimtThreads, smem, p.st>>>(
                (const T*)p.q.ptr, (const T*)p.k.ptr, (const T*)p.v.ptr, p.lse, (const T*)p.d_o.ptr, (T*)p.d_q.ptr,
                p.delta, p.row_factor, p.q.st, p.k.st, p.v.st, p.d_o.st, p.d_q.st, g);
        return after_launch();
    });
}

int run_backward_dkdv(const Problem& p) {
    const Na2dGeom& g = p.g;
    if (p.tensor) {
        int launched = 0;
        na2d_tc::LaunchCtx lc;
        int rc = launch_ctx(p, &launched, &lc);
        if (rc != NA2D_OK) return rc;
        rc = p.dtype == NA2D_BF16
                 ? na2d_tc::backward_dkdv_bf16(lc, targ(p.q), targ(p.k), targ(p.v), p.lse, targ(p.d_o), p.delta, targ(p.d_k), targ(p.d_v))
                 : na2d_tc::backward_dkdv_f16(lc, targ(p.q), targ(p.k), targ(p.v), p.lse, targ(p.d_o), p.delta, targ(p.d_k), targ(p.d_v));
        g_launches.fetch_add(launched);
        if (rc == NA2D_ERR_CUDA) return tc_fail("tcgen05 dK/dV launch");
        return rc;
    }
    unsigned grid = 0;
    int rc = grid_for(g.BN, g.Hkv, g.W, g.patch, &grid);
    if (rc != NA2D_OK) return rc;
    return simt_dispatch(p.dtype, g.C, [&](auto tt, auto cpl) -> int {
        using T = typename decltype(tt)::type;
        na2d_simt::dkdv_kernel<T, decltype(cpl)::value><<<grid, kSimtThreads, 0, p.st>>>(
            (const T*)p.q.ptr, (const T*)p.k.ptr, (const T*)p.v.ptr, p.lse, (const T*)p.d_o.ptr, p.delta, p.row_factor,
            p.d_k.ptr, p.d_v.ptr, p.dkdv_f32 ? 1 : 0, p.q.st, p.k.st, p.v.st, p.d_o.st, p.d_k.st, p.d_v.st, g);
        return after_launch();
    });
}

// What na2d_backward_workspace asks for at most, unless the rows of weights that a row of key tiles reads need more: a
// launch over that many weights (2 x 64 M) fills the GPU many times over, so taking units, or rows of one unit, in several
// turns costs little (fp32, window 13, head dim 32, both halves: 1024 x 1024 3.3 -> 3.5 ms for 0.5 in place of 1.6 GiB,
// 2048 x 2048 12.9 -> 13.9 ms for 0.5 in place of 6.5 GiB).
constexpr long long kWorkspaceBytes = 512ll << 20;

// Whether the backward hands something on to its key half: the tensor-core kernels form P and dS again, faster than
// they could be read, and row views and fp32 partial sums stay with the halves that can be called by themselves.
bool uses_workspace(const Problem& p, const na2d_args* a) { return !p.tensor && !a->rows && !p.dkdv_f32; }
// P and dS, or else the factors that make P of exp(s - lse): small problems, and windows without tiled kernels.
bool hands_on_weights(const Problem& p) { return in_tiles(na2d_tile::Work::kBackward, p.g, p.dtype); }
size_t row_factor_bytes(const Problem& p) { return (size_t)p.g.BN * p.g.Hq * p.g.W * sizeof(float); }

// Both halves of the backward, sharing a workspace.
int run_backward_shared(const Problem& p, void* workspace, na2d_tile::Turns turns) {
    const auto run = NA2D_TILE_PICK(p.dtype, backward);
    int launches = 0;
    return at_place(p.device, p.st, p.dtype, p.g, [&](const na2d_tile::Place& at) {
        const int rc = run(p.g, at, tile(p.q), tile(p.k), tile(p.v), tile(p.d_o), tile(p.d_q), tile(p.d_k), tile(p.d_v), p.lse,
                           p.delta, (float*)workspace, turns, &launches);
        g_launches.fetch_add(launches);
        return after_tile(rc, 0);
    });
}

// Validate, select the device, check it; then run `step`.
template <typename F>
int enter(const na2d_args* a, F&& step, bool key_side = false) {
    Problem p;
    int rc = make_problem(a, &p, key_side);
    if (rc != NA2D_OK) return rc;
    DeviceScope scope(p.device);
    if (scope.err != cudaSuccess) return cuda_fail(scope.err, "cudaSetDevice");
    rc = check_device(p.device);
    if (rc != NA2D_OK) return rc;
    return step(p);
}

na2d_tensor dense(const void* ptr) { return na2d_tensor{const_cast<void*>(ptr), 0, 0, 0, 0}; }

na2d_args dense_args(int op, int B, int N, int H, int W, int C, int ks, int dtype, const na2d_rows* rows, int path,
                     int device, void* stream) {
    na2d_args a;
    std::memset(&a, 0, sizeof(a));
    a.struct_size = sizeof(a);
    a.op = op;
    a.B = B; a.N = N; a.H = H; a.W = W; a.C = C; a.kernel_size = ks; a.dtype = dtype; a.path = path; a.device = device;
    a.scale = 1.f;
    a.stream = stream;
    a.rows = rows;
    return a;
}

// ---- scratch for na2d_backward_static_scratch ----------------------------------------------------
// The backward pair passes the row delta from the dQ kernel to the dK/dV kernel through global
// memory.  Normally the caller provides that buffer; the entry point below keeps it in this
// file-scope device array instead, so that a caller who may not allocate can still run the
// backward.  Every GPU on which the library's device code has been loaded carries the array
// (4 MiB) until the process exits.
constexpr long long kStaticDeltaFloats = 1LL << 20;
static __device__ __align__(256) float g_static_delta[kStaticDeltaFloats];

// Device address of g_static_delta on `device`, looked up once per device.  In host code the
// name g_static_delta is only a handle for the runtime, not an address a kernel could use; the
// address comes from cudaGetSymbolAddress, asked while `device` is the current device.
int static_delta_address(int device, float** out) {
    static std::mutex mu;
    static float* cache[kMaxDevices];
    if (device < 0 || device >= kMaxDevices) return NA2D_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(mu);
    if (cache[device] == nullptr) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_delta);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_static_delta)");
        cache[device] = static_cast<float*>(p);
    }
    *out = cache[device];
    return NA2D_OK;
}

// ---- the unfused pair -------------------------------------------------------------------------------------
struct PairProblem {
    Na2dGeom g;
    int dtype;
    Na2dStride st;          // dense strides of a (B, N, H, W, C) tensor
    int device;
    cudaStream_t stream;
};

int make_pair_problem(int B, int N, int H, int W, int C, int ks, int dtype, int device, void* stream, PairProblem* out) {
    if (B <= 0 || N <= 0 || H <= 0 || W <= 0 || C <= 0) return NA2D_ERR_BAD_ARG;
    if (ks <= 0 || (ks & 1) == 0) return NA2D_ERR_BAD_ARG;
    if (dtype != NA2D_F32 && dtype != NA2D_BF16 && dtype != NA2D_F16) return NA2D_ERR_UNSUPPORTED;
    if ((long long)B * N > 0x7fffffffLL) return NA2D_ERR_TOO_LARGE;
    if (H < ks || W < ks) return NA2D_ERR_WINDOW;
    if (C > na2d_simt::kMaxC || ks > na2d_simt::kMaxKs) return NA2D_ERR_UNSUPPORTED;
    Na2dGeom g;
    g.BN = B * N; g.N = N; g.n_magic = na2d_heads_magic(g.BN, N); g.Hq = H; g.Hkv = H; g.W = W; g.C = C; g.ks = ks; g.kh = ks;
    g.q_row0 = 0; g.kv_row0 = 0; g.Hg = H; g.scale = 1.f; g.sl2 = 1.4426950408889634f;
    g.patch = simt_patch(g.BN, H, W);
    out->g = g;
    out->dtype = dtype;
    out->st = Na2dStride{(long long)N * H * W * C, (long long)H * W * C, (long long)W * C, C};
    out->device = device;
    out->stream = (cudaStream_t)stream;
    return NA2D_OK;
}

template <typename F>
int enter_pair(int B, int N, int H, int W, int C, int ks, int dtype, int device, void* stream, F&& step) {
    PairProblem p;
    int rc = make_pair_problem(B, N, H, W, C, ks, dtype, device, stream, &p);
    if (rc != NA2D_OK) return rc;
    DeviceScope scope(device);
    if (scope.err != cudaSuccess) return cuda_fail(scope.err, "cudaSetDevice");
    rc = check_device(device);
    if (rc != NA2D_OK) return rc;
    return step(p);
}

na2d_tile::Tensor tile_dense(const PairProblem& p, const void* ptr) { return na2d_tile::Tensor{const_cast<void*>(ptr), p.st}; }

// x . y over the window -> attn
int pair_dot(const PairProblem& p, const void* x, const void* y, void* attn) {
    if (in_tiles(na2d_tile::Work::kDot, p.g, p.dtype))
        return at_place(p.device, p.stream, p.dtype, p.g, [&](const na2d_tile::Place& at) {
            return after_tile(NA2D_TILE_PICK(p.dtype, pair_dot)(p.g, at, tile_dense(p, x), tile_dense(p, y), attn), 1);
        });
    unsigned grid = 0;
    int rc = grid_for(p.g.BN, p.g.Hq, p.g.W, p.g.patch, &grid);
    if (rc != NA2D_OK) return rc;
    return simt_dispatch(p.dtype, p.g.C, [&](auto tt, auto cpl) -> int {
        using T = typename decltype(tt)::type;
        na2d_simt::window_dot_kernel<T, decltype(cpl)::value><<<grid, kSimtThreads, 0, p.stream>>>(
            (const T*)x, (const T*)y, (T*)attn, p.st, p.st, p.g);
        return after_launch();
    });
}
// sum_j attn_j y_j -> out
int pair_apply(const PairProblem& p, const void* attn, const void* y, void* out) {
    if (in_tiles(na2d_tile::Work::kApply, p.g, p.dtype))
        return at_place(p.device, p.stream, p.dtype, p.g, [&](const na2d_tile::Place& at) {
            return after_tile(NA2D_TILE_PICK(p.dtype, pair_apply)(p.g, at, attn, tile_dense(p, y), tile_dense(p, out)), 1);
        });
    unsigned grid = 0;
    int rc = grid_for(p.g.BN, p.g.Hq, p.g.W, p.g.patch, &grid);
    if (rc != NA2D_OK) return rc;
    return simt_dispatch(p.dtype, p.g.C, [&](auto tt, auto cpl) -> int {
        using T = typename decltype(tt)::type;
        na2d_simt::window_apply_kernel<T, decltype(cpl)::value>
            <<<grid, kSimtThreads, na2d_simt::window_smem_bytes(p.g.kh, p.g.ks, 1), p.stream>>>(
                (const T*)attn, (const T*)y, (T*)out, p.st, p.st, p.g);
        return after_launch();
    });
}
// key-side sum over the inverse neighbourhood of attn x -> out
int pair_inverse(const PairProblem& p, const void* attn, const void* x, void* out) {
    if (in_tiles(na2d_tile::Work::kKeySum, p.g, p.dtype))
        return at_place(p.device, p.stream, p.dtype, p.g, [&](const na2d_tile::Place& at) {
            return after_tile(NA2D_TILE_PICK(p.dtype, pair_inverse)(p.g, at, attn, tile_dense(p, x), tile_dense(p, out)), 1);
        });
    unsigned grid = 0;
    int rc = grid_for(p.g.BN, p.g.Hkv, p.g.W, p.g.patch, &grid);
    if (rc != NA2D_OK) return rc;
    return simt_dispatch(p.dtype, p.g.C, [&](auto tt, auto cpl) -> int {
        using T = typename decltype(tt)::type;
        na2d_simt::window_inverse_kernel<T, decltype(cpl)::value><<<grid, kSimtThreads, 0, p.stream>>>(
            (const T*)attn, (const T*)x, (T*)out, p.st, p.st, p.g);
        return after_launch();
    });
}

}  // namespace

extern "C" {

int na2d_version(void) { return 200; }

const char* na2d_strerror(int status) {
    switch (status) {
        case NA2D_OK: return "ok";
        case NA2D_ERR_BAD_ARG: return "bad argument (null pointer, non-positive size, even kernel size, bad scale or bad row view)";
        case NA2D_ERR_UNSUPPORTED: return "unsupported dtype, head dim, kernel size or tensor layout for the requested path";
        case NA2D_ERR_WINDOW: return "grid side smaller than the kernel size, or key band does not cover the query band's windows";
        case NA2D_ERR_CUDA: return "CUDA call failed (see na2d_last_cuda_error)";
        case NA2D_ERR_NO_DEVICE: return "device is not an sm_100 (B200) GPU";
        case NA2D_ERR_TOO_LARGE: return "size beyond a documented maximum";
        case NA2D_ERR_KERNEL_WAIT: return "a bounded wait inside a kernel ran out";
        default: return "unknown status";
    }
}

const char* na2d_last_cuda_error(void) { return t_cuda_err; }

int na2d_window_start(int i, int seq_len, int kernel_size) { return na2d_ws(i, seq_len, kernel_size); }

int na2d_backward_window(int j, int seq_len, int kernel_size, int* lo, int* hi) {
    if (!lo || !hi || kernel_size <= 0 || seq_len <= 0) return NA2D_ERR_BAD_ARG;
    *lo = na2d_bws(j, kernel_size);
    *hi = na2d_bwe(j, seq_len, kernel_size);
    return NA2D_OK;
}

int na2d_dump_index(int32_t* ws, int32_t* bws, int32_t* bwe, int seq_len, int kernel_size,
                    int device, void* stream) {
    if (!ws || !bws || !bwe || seq_len <= 0 || kernel_size <= 0) return NA2D_ERR_BAD_ARG;
    DeviceScope scope(device);
    if (scope.err != cudaSuccess) return cuda_fail(scope.err, "cudaSetDevice");
    na2d_simt::index_dump_kernel<<<(seq_len + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
        ws, bws, bwe, seq_len, kernel_size);
    return after_launch();
}

// ---- strided / scaled / 1D entry points ------------------------------------------------------------------
int na2d_forward_ex(const na2d_args* a) {
    if (!a || !a->q.ptr || !a->k.ptr || !a->v.ptr || !a->o.ptr || !a->lse) return NA2D_ERR_BAD_ARG;
    return enter(a, [](const Problem& p) { return run_forward(p); });
}

int na2d_backward_dq_ex(const na2d_args* a) {
    if (!a || !a->q.ptr || !a->k.ptr || !a->v.ptr || !a->lse || !a->d_o.ptr || !a->delta) return NA2D_ERR_BAD_ARG;
    return enter(a, [](const Problem& p) { return run_backward_dq(p); });
}

int na2d_backward_dkdv_ex(const na2d_args* a) {
    if (!a || !a->q.ptr || !a->k.ptr || !a->v.ptr || !a->lse || !a->d_o.ptr || !a->delta || !a->d_k.ptr || !a->d_v.ptr)
        return NA2D_ERR_BAD_ARG;
    return enter(a, [](const Problem& p) { return run_backward_dkdv(p); }, /*key_side=*/true);
}

size_t na2d_backward_workspace(const na2d_args* a) {
    Problem p;
    if (make_problem(a, &p) != NA2D_OK || !uses_workspace(p, a)) return 0;
    if (!hands_on_weights(p)) return row_factor_bytes(p);
    return sizeof(float) * (size_t)na2d_tile::workspace_floats(p.g, kWorkspaceBytes / (long long)sizeof(float));
}

int na2d_backward_ex(const na2d_args* a) {
    if (!a) return NA2D_ERR_BAD_ARG;
    if ((a->d_k.ptr == nullptr) != (a->d_v.ptr == nullptr)) return NA2D_ERR_BAD_ARG;
    if (!a->d_q.ptr && !a->d_k.ptr) return NA2D_ERR_BAD_ARG;
    if (a->d_k.ptr && a->struct_size >= sizeof(na2d_args) && a->workspace) {
        if (!a->q.ptr || !a->k.ptr || !a->v.ptr || !a->lse || !a->d_o.ptr || !a->delta) return NA2D_ERR_BAD_ARG;
        if (reinterpret_cast<uintptr_t>(a->workspace) % 16) return NA2D_ERR_BAD_ARG;
        return enter(a, [&](const Problem& problem) -> int {
            Problem p = problem;
            if (uses_workspace(p, a)) {
                const long long floats = (long long)(a->workspace_bytes / sizeof(float));
                const na2d_tile::Turns turns = hands_on_weights(p) ? na2d_tile::workspace_turns(p.g, floats) : na2d_tile::Turns{0, 0};
                if (turns.units > 0) return run_backward_shared(p, a->workspace, turns);
                if (a->workspace_bytes >= row_factor_bytes(p)) p.row_factor = (float*)a->workspace;
            }
            const int rc = run_backward_dq(p);
            return rc != NA2D_OK ? rc : run_backward_dkdv(p);
        });
    }
    // the query half always runs: it produces delta, which the key half needs
    int rc = na2d_backward_dq_ex(a);
    if (rc != NA2D_OK || a->d_k.ptr == nullptr) return rc;
    return na2d_backward_dkdv_ex(a);
}

// ---- dense entry points -------------------------------------------------------------------------------------
int na2d_forward(const void* q, const void* k, const void* v, void* o, float* lse,
                 int B, int N, int H, int W, int C, int kernel_size, int dtype,
                 const na2d_rows* rows, int path, int device, void* stream) {
    na2d_args a = dense_args(NA2D_OP_2D, B, N, H, W, C, kernel_size, dtype, rows, path, device, stream);
    a.q = dense(q); a.k = dense(k); a.v = dense(v); a.o = dense(o); a.lse = lse;
    return na2d_forward_ex(&a);
}

int na2d_backward_dq(const void* q, const void* k, const void* v, const void* o, const float* lse,
                     const void* d_o, void* d_q, float* delta,
                     int B, int N, int H, int W, int C, int kernel_size, int dtype,
                     const na2d_rows* rows, int path, int device, void* stream) {
    na2d_args a = dense_args(NA2D_OP_2D, B, N, H, W, C, kernel_size, dtype, rows, path, device, stream);
    a.q = dense(q); a.k = dense(k); a.v = dense(v); a.o = dense(o); a.lse = const_cast<float*>(lse);
    a.d_o = dense(d_o); a.d_q = dense(d_q); a.delta = delta;
    return na2d_backward_dq_ex(&a);
}

int na2d_backward_dkdv(const void* q, const void* k, const void* v, const float* lse,
                       const void* d_o, const float* delta, void* d_k, void* d_v,
                       int B, int N, int H, int W, int C, int kernel_size, int dtype,
                       const na2d_rows* rows, int path, int device, void* stream) {
    na2d_args a = dense_args(NA2D_OP_2D, B, N, H, W, C, kernel_size, dtype, rows, path, device, stream);
    a.q = dense(q); a.k = dense(k); a.v = dense(v); a.lse = const_cast<float*>(lse);
    a.d_o = dense(d_o); a.delta = const_cast<float*>(delta); a.d_k = dense(d_k); a.d_v = dense(d_v);
    return na2d_backward_dkdv_ex(&a);
}

int na2d_backward(const void* q, const void* k, const void* v, const void* o, const float* lse,
                  const void* d_o, void* d_q, void* d_k, void* d_v, float* delta,
                  int B, int N, int H, int W, int C, int kernel_size, int dtype,
                  const na2d_rows* rows, int path, int device, void* stream) {
    na2d_args a = dense_args(NA2D_OP_2D, B, N, H, W, C, kernel_size, dtype, rows, path, device, stream);
    a.q = dense(q); a.k = dense(k); a.v = dense(v); a.o = dense(o); a.lse = const_cast<float*>(lse);
    a.d_o = dense(d_o); a.d_q = dense(d_q); a.d_k = dense(d_k); a.d_v = dense(d_v); a.delta = delta;
    return na2d_backward_ex(&a);
}

int na1d_forward(const void* q, const void* k, const void* v, void* o, float* lse,
                 int B, int N, int T, int C, int kernel_size, int dtype, int device, void* stream) {
    na2d_args a = dense_args(NA2D_OP_1D, B, N, 1, T, C, kernel_size, dtype, nullptr, NA2D_PATH_AUTO, device, stream);
    a.q = dense(q); a.k = dense(k); a.v = dense(v); a.o = dense(o); a.lse = lse;
    return na2d_forward_ex(&a);
}

int na1d_backward(const void* q, const void* k, const void* v, const void* o, const float* lse,
                  const void* d_o, void* d_q, void* d_k, void* d_v, float* delta,
                  int B, int N, int T, int C, int kernel_size, int dtype, int device, void* stream) {
    na2d_args a = dense_args(NA2D_OP_1D, B, N, 1, T, C, kernel_size, dtype, nullptr, NA2D_PATH_AUTO, device, stream);
    a.q = dense(q); a.k = dense(k); a.v = dense(v); a.o = dense(o); a.lse = const_cast<float*>(lse);
    a.d_o = dense(d_o); a.d_q = dense(d_q); a.d_k = dense(d_k); a.d_v = dense(d_v); a.delta = delta;
    return na2d_backward_ex(&a);
}

// ---- the unfused pair -------------------------------------------------------------------------------------------
int na2d_qk_forward(const void* q, const void* k, void* attn,
                    int B, int N, int H, int W, int C, int kernel_size, int dtype, int device, void* stream) {
    if (!q || !k || !attn) return NA2D_ERR_BAD_ARG;
    return enter_pair(B, N, H, W, C, kernel_size, dtype, device, stream,
                      [&](const PairProblem& p) { return pair_dot(p, q, k, attn); });
}

int na2d_qk_backward(const void* q, const void* k, const void* d_attn, void* d_q, void* d_k,
                     int B, int N, int H, int W, int C, int kernel_size, int dtype, int device, void* stream) {
    if (!q || !k || !d_attn || !d_q || !d_k) return NA2D_ERR_BAD_ARG;
    return enter_pair(B, N, H, W, C, kernel_size, dtype, device, stream, [&](const PairProblem& p) {
        int rc = pair_apply(p, d_attn, k, d_q);
        if (rc != NA2D_OK) return rc;
        return pair_inverse(p, d_attn, q, d_k);
    });
}

int na2d_av_forward(const void* attn, const void* v, void* out,
                    int B, int N, int H, int W, int C, int kernel_size, int dtype, int device, void* stream) {
    if (!attn || !v || !out) return NA2D_ERR_BAD_ARG;
    return enter_pair(B, N, H, W, C, kernel_size, dtype, device, stream,
                      [&](const PairProblem& p) { return pair_apply(p, attn, v, out); });
}

int na2d_av_backward(const void* attn, const void* v, const void* d_out, void* d_attn, void* d_v,
                     int B, int N, int H, int W, int C, int kernel_size, int dtype, int device, void* stream) {
    if (!attn || !v || !d_out || !d_attn || !d_v) return NA2D_ERR_BAD_ARG;
    return enter_pair(B, N, H, W, C, kernel_size, dtype, device, stream, [&](const PairProblem& p) {
        int rc = pair_dot(p, d_out, v, d_attn);
        if (rc != NA2D_OK) return rc;
        return pair_inverse(p, attn, d_out, d_v);
    });
}

int na2d_backward_static_scratch(const void* q, const void* k, const void* v, const void* o, const float* lse,
                                 const void* d_o, void* d_q, void* d_k, void* d_v,
                                 int B, int N, int H, int W, int C, int kernel_size, int dtype,
                                 const na2d_rows* rows, int path, int device, void* stream) {
    if (B <= 0 || N <= 0 || H <= 0 || W <= 0) return NA2D_ERR_BAD_ARG;
    const long long hq = rows ? rows->Hq : H;
    if (hq <= 0) return NA2D_ERR_BAD_ARG;
    if ((long long)B * N * hq * W > kStaticDeltaFloats) {
        snprintf(t_cuda_err, sizeof(t_cuda_err),
                 "na2d_backward_static_scratch: B*N*Hq*W = %lld exceeds the built-in scratch of %lld floats",
                 (long long)B * N * hq * W, kStaticDeltaFloats);
        return NA2D_ERR_TOO_LARGE;
    }
    float* delta = nullptr;
    {
        DeviceScope scope(device);                        // the lookup needs `device` current
        if (scope.err != cudaSuccess) return cuda_fail(scope.err, "cudaSetDevice");
        int rc = static_delta_address(device, &delta);
        if (rc != NA2D_OK) return rc;
    }
    // delta is fully rewritten by the query half for every query of this call before the key
    // half reads it, so nothing has to be cleared between calls.
    return na2d_backward(q, k, v, o, lse, d_o, d_q, d_k, d_v, delta, B, N, H, W, C, kernel_size, dtype,
                         rows, path, device, stream);
}

int na2d_check(int device, void* stream) {
    DeviceScope scope(device);
    if (scope.err != cudaSuccess) return cuda_fail(scope.err, "cudaSetDevice");
    Errors err;
    int rc = error_state(device, &err);
    if (rc != NA2D_OK) return rc;
    NA2D_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    const unsigned int kinds = take_errors(err.word);
    if (kinds != 0) {
        snprintf(t_cuda_err, sizeof(t_cuda_err),
                 "error kinds 0x%x (1: load wait, 2: MMA wait, 4: other wait, 8: shared memory base not 1024-byte aligned)", kinds);
        return NA2D_ERR_KERNEL_WAIT;
    }
    return NA2D_OK;
}

int na2d_poll(int device, void* stream) {
    (void)stream;
    if (device < 0 || device >= kMaxDevices) return NA2D_ERR_BAD_ARG;
    volatile unsigned int* word = g_error_words[device].load(std::memory_order_acquire);
    if (word != nullptr) return take_errors(word) == 0 ? NA2D_OK : NA2D_ERR_KERNEL_WAIT;
    // no kernel that waits has run there yet; a device that is none is an error all the same
    static std::atomic<int> devices{0};
    if (device < devices.load(std::memory_order_relaxed)) return NA2D_OK;
    int n = 0;
    NA2D_CUDA(cudaGetDeviceCount(&n));
    devices.store(n, std::memory_order_relaxed);
    return device < n ? NA2D_OK : cuda_fail(cudaErrorInvalidDevice, "na2d_poll");
}

int na2d_selftest_wait_timeout(int device, void* stream, unsigned int limit_us) {
    DeviceScope scope(device);
    if (scope.err != cudaSuccess) return cuda_fail(scope.err, "cudaSetDevice");
    int rc = check_device(device);
    if (rc != NA2D_OK) return rc;
    if (limit_us == 0 || limit_us > 1000000u) return NA2D_ERR_BAD_ARG;       // at most a second
    Errors err;
    rc = error_state(device, &err);
    if (rc != NA2D_OK) return rc;
    wait_timeout_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(err.device, (unsigned long long)limit_us * 1000ull);
    return after_launch();
}

long long na2d_launch_count(void) { return g_launches.load(); }

}  // extern "C"
