"""Build libna2d.so in-tree with nvcc for sm_100a.

    python e_natten_b200/build.py [--force] [--verbose]

The library is plain CUDA C++ behind a C ABI (include/na2d.h); it needs no framework headers.
Its kernels are compiled as eleven translation units in parallel (the API with the SIMT kernels, the
tiled CUDA-core kernels once per element type, the fp32 box kernels, and each of the three tcgen05 kernel families once per
16-bit element type) and linked into one shared object.  The Python package's extension module
(_na2d_torch.so, host code over PyTorch's C++ API) is compiled beside it with g++; it belongs to one
PyTorch and one Python version and is compiled again when either changes.
"""
from __future__ import annotations

import concurrent.futures
import importlib.metadata
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
OBJ_DIR = os.path.join(PKG_DIR, "build")
LIB_PATH = os.path.join(PKG_DIR, "libna2d.so")
EXT_PATH = os.path.join(PKG_DIR, "_na2d_torch.so")
# (source, extra defines, object name)
UNITS = [
    ("na2d_api.cu", [], "na2d_api.o"),
    ("na2d_tile.cu", ["-DNA2D_TILE_DT=0"], "na2d_tile_f32.o"),
    ("na2d_tile.cu", ["-DNA2D_TILE_DT=1"], "na2d_tile_bf16.o"),
    ("na2d_tile.cu", ["-DNA2D_TILE_DT=2"], "na2d_tile_f16.o"),
    ("na2d_box.cu", [], "na2d_box.o"),
    ("na2d_tc_fwd.cu", ["-DNA2D_TC_DT=1"], "na2d_tc_fwd_bf16.o"),
    ("na2d_tc_fwd.cu", ["-DNA2D_TC_DT=2"], "na2d_tc_fwd_f16.o"),
    ("na2d_tc_dq.cu", ["-DNA2D_TC_DT=1"], "na2d_tc_dq_bf16.o"),
    ("na2d_tc_dq.cu", ["-DNA2D_TC_DT=2"], "na2d_tc_dq_f16.o"),
    ("na2d_tc_dkdv.cu", ["-DNA2D_TC_DT=1"], "na2d_tc_dkdv_bf16.o"),
    ("na2d_tc_dkdv.cu", ["-DNA2D_TC_DT=2"], "na2d_tc_dkdv_f16.o"),
]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libna2d.so cannot be built")
    return exe


EXT_SOURCE = "na2d_torch.cpp"


def _deps(ext: bool):
    """Sources of the extension module, or of the library."""
    names = [EXT_SOURCE] if ext else [f for f in os.listdir(CSRC) if f != EXT_SOURCE]
    deps = [os.path.join(CSRC, f) for f in names]
    deps.append(os.path.join(os.path.dirname(PKG_DIR), "include", "na2d.h"))
    return [d for d in deps if os.path.isfile(d)]


def _older(path: str, ext: bool) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in _deps(ext))


def _ext_tag() -> str:
    """What the extension module is compiled for; the module carries it as a string."""
    return f"na2d_torch for torch {importlib.metadata.version('torch')}, {sys.implementation.cache_tag}"


def _lib_stale() -> bool:
    return _older(LIB_PATH, ext=False)


def _ext_stale() -> bool:
    if _older(EXT_PATH, ext=True):
        return True
    with open(EXT_PATH, "rb") as f:
        return _ext_tag().encode() not in f.read()


def _compile(unit, verbose: bool, extra, obj_dir):
    src, defines, obj = unit
    cmd = [_nvcc(), *NVCC_FLAGS, *extra, *(["-Xptxas", "-v"] if verbose else []), *defines, "-c",
           os.path.join(CSRC, src), "-o", os.path.join(obj_dir, obj)]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    return obj, proc.returncode, proc.stdout + proc.stderr, " ".join(cmd)


def _compile_torch_ext():
    """The Python extension module over PyTorch's C++ API (host code only)."""
    import torch
    from torch.utils import cpp_extension
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DNA2D_EXT_TAG="{_ext_tag()}"',
           *[f"-isystem{p}" for p in (*cpp_extension.include_paths("cuda"), sysconfig.get_paths()["include"])],
           os.path.join(CSRC, EXT_SOURCE), "-o", EXT_PATH,
           *[f"-L{p}" for p in cpp_extension.library_paths("cuda")],
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    return os.path.basename(EXT_PATH), proc.returncode, proc.stdout + proc.stderr, " ".join(cmd)


def build(force: bool = False, verbose: bool = False, extra_flags=(), lib_path: str = LIB_PATH) -> str:
    """Compile the library and the extension module where they are missing or out of date; return
    the library's path."""
    own = lib_path == LIB_PATH         # a library built elsewhere (a development build) has no extension module
    build_lib = force or not own or _lib_stale()
    build_ext = own and (force or _ext_stale())
    if not (build_lib or build_ext):
        return lib_path
    # one with other flags keeps its objects apart
    obj_dir = OBJ_DIR if own else lib_path + ".objs"
    os.makedirs(obj_dir, exist_ok=True)
    units = UNITS if build_lib else []
    with concurrent.futures.ThreadPoolExecutor(max(1, min(len(UNITS), os.cpu_count() or 1))) as pool:
        ext = pool.submit(_compile_torch_ext) if build_ext else None
        results = list(pool.map(lambda u: _compile(u, verbose, list(extra_flags), obj_dir), units))
        if ext is not None:
            results.append(ext.result())
    for obj, rc, out, cmd in results:
        if verbose or rc != 0:
            sys.stderr.write(f"--- {obj}\n{out}")
        if rc != 0:
            raise RuntimeError("failed compiling %s (command: %s)" % (obj, cmd))
    if not build_lib:
        return lib_path
    link = [_nvcc(), "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a",
            *[os.path.join(obj_dir, u[2]) for u in UNITS], "-o", lib_path]
    proc = subprocess.run(link, capture_output=True, text=True)
    if proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
        raise RuntimeError("nvcc failed linking libna2d.so (command: %s)" % " ".join(link))
    return lib_path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
