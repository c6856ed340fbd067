"""CPU test of the host code that describes operands to TMA, against a stand-in for the driver's encoder."""
import os
import shutil
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "e_natten_b200", "csrc")

PROGRAM = r"""
#include "na2d_tc.cuh"
#include <cstdio>

static int result = 0, calls = 0;
static CUresult encode(CUtensorMap* map, CUtensorMapDataType, cuuint32_t, void* base, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                       const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    ++calls;
    map->opaque[0] = (cuuint64_t)(size_t)base;
    return (CUresult)result;
}
extern "C" cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* found) {
    *fn = (void*)&encode;
    if (found) *found = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
#define EXPECT(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    CUtensorMap map;
    const na2d_tc::TensorArg a{(void*)4096, {1 << 20, 1 << 18, 1 << 13, 64}}, b{(void*)8192, {1 << 20, 1 << 18, 1 << 13, 64}};
    result = 1;
    EXPECT(na2d_tc::make_map(&map, a, NA2D_BF16, 1, 2, 32, 128, 64, 8, 16) == NA2D_ERR_CUDA);
    EXPECT(na2d_tc::last_driver_result() == 1);                  // for the error text
    na2d_tc::last_driver_result() = 0;
    EXPECT(!na2d_tc::try_map(&map, a, NA2D_F32, 1, 2, 32, 128, 64, 17, 8, 16, true));
    EXPECT(na2d_tc::last_driver_result() == 0 && calls == 2);    // the call goes on with other kernels: nothing to report
    result = 0;
    EXPECT(na2d_tc::try_map(&map, a, NA2D_F32, 1, 2, 32, 128, 64, 17, 8, 16, true) && map.opaque[0] == 4096);
    EXPECT(na2d_tc::try_map(&map, b, NA2D_F32, 1, 2, 32, 128, 64, 17, 8, 16, true) && map.opaque[0] == 8192);
    EXPECT(na2d_tc::make_map(&map, a, NA2D_BF16, 1, 2, 32, 128, 64, 8, 16) == NA2D_OK && map.opaque[0] == 4096);
    EXPECT(na2d_tc::make_map(&map, a, NA2D_BF16, 1, 2, 32, 128, 64, 8, 16) == NA2D_OK && map.opaque[0] == 4096 && calls == 5);   // kept
    // a model of ten layers, three steps on the same buffers: nearly all of its maps are still there
    calls = 0;
    for (int step = 0; step < 3; ++step)
        for (int layer = 0; layer < 10; ++layer)
            for (int operand = 0; operand < 12; ++operand) {
                const size_t at = (size_t)(1 + layer * 12 + operand) << 21;
                const na2d_tc::TensorArg x{(void*)at, {1 << 20, 1 << 18, 1 << 13, 64}};
                EXPECT(na2d_tc::make_map(&map, x, NA2D_BF16, 1, 2, 32, 128, 64, 8, 16 + operand % 3) == NA2D_OK && map.opaque[0] == at);
            }
    EXPECT(calls >= 120 && calls < 180);
    // whatever differs in a description makes another map of it
    calls = 0;
    const Na2dStride st{1 << 24, 1 << 20, 1 << 14, 128};
    const na2d_tc::TensorArg y{(void*)(1 << 20), st};
    const int base[9] = {NA2D_BF16, 2, 3, 40, 50, 64, 8, 16, 32};
    for (int i = -1; i < 15; ++i) {
        int n[9];
        for (int j = 0; j < 9; ++j) n[j] = base[j] + (i == j ? (j == 0 ? NA2D_F16 - NA2D_BF16 : 8) : 0);
        na2d_tc::TensorArg x = y;
        if (i == 9) x.ptr = (void*)((1 << 20) + 16);
        if (i == 10) x.st.b += 8;
        if (i == 11) x.st.n += 8;
        if (i == 12) x.st.h += 8;
        if (i == 13) x.st.w += 8;
        EXPECT(na2d_tc::make_map(&map, x, n[0], n[1], n[2], n[3], n[4], n[5], n[6], n[7], n[8], i == 14) == NA2D_OK && calls == i + 2);
    }
    return 0;
}
"""


def test_a_refused_map_leaves_an_error_only_where_the_call_fails(tmp_path):
    """A launcher that hands the call to other kernels leaves nothing behind; one that fails leaves the driver's result for the report."""
    source, program = tmp_path / "maps.cu", tmp_path / "maps"
    source.write_text(PROGRAM)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    build = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "shared", "-I", CSRC, str(source),
                            "-o", str(program)], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(program)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr
    with open(os.path.join(CSRC, "na2d_box.cu")) as f:           # whose launchers leave a call to the tiled kernels
        text = f.read()
    assert "try_map(" in text and "make_map(" not in text
