"""CPU tests of the C ABI: the library loads, exports what include/na2d.h declares, its host-side
index functions are bit-exact with the reference's, and bad arguments are refused before any CUDA
call.  No compute runs here."""
import ctypes as C
import os
import re

import numpy as np
import pytest
import torch

import e_natten_b200 as na
from e_natten_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_functions():
    text = open(os.path.join(ROOT, "include", "na2d.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(na[12]d_[a-z_0-9]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    names = _declared_functions()
    assert "na2d_forward" in names and "na2d_backward" in names and len(names) >= 10
    raw = C.CDLL(_lib.LIB_PATH)
    for n in names:
        assert hasattr(raw, n), f"{n} declared in include/na2d.h but not exported"
    assert sorted(_lib.SIGNATURES) == names               # the binding covers exactly the header


def test_version_and_strerror():
    assert _lib.lib.na2d_version() >= 200
    for code in range(0, -8, -1):
        assert len(_lib.lib.na2d_strerror(code)) > 0


@pytest.mark.parametrize("ks", list(range(3, 16, 2)))
def test_host_index_functions_bit_exact(golden, ks):
    for L in list(range(ks, 81)) + [192, 256, 1024]:
        ws = np.array([na.get_window_start(i, L, ks) for i in range(L)], dtype=np.int32)
        assert np.array_equal(ws, golden[f"idx/ws/{ks}/{L}"])
        if L <= 40 or L == 1024:
            bs = np.array([na.get_backward_window_start(i, ks) for i in range(L)], dtype=np.int32)
            be = np.array([na.get_backward_window_end(i, L, ks) for i in range(L)], dtype=np.int32)
            assert np.array_equal(bs, golden[f"idx/bws/{ks}/{L}"])
            assert np.array_equal(be, golden[f"idx/bwe/{ks}/{L}"])


def _fwd(ptrs=(1, 1, 1, 1, 1), B=1, N=1, H=8, W=8, Cd=32, ks=5, dtype=0, rows=None, path=0):
    p = [C.c_void_p(x) for x in ptrs]
    return _lib.lib.na2d_forward(*p, B, N, H, W, Cd, ks, dtype, rows, path, 0, None)


def test_forward_refuses_bad_arguments_without_touching_cuda():
    # (non-null dummy pointers are never dereferenced: validation comes first)
    assert _fwd(ptrs=(0, 1, 1, 1, 1)) == _lib.ERR_BAD_ARG
    assert _fwd(ks=4) == _lib.ERR_BAD_ARG
    assert _fwd(ks=-1) == _lib.ERR_BAD_ARG
    assert _fwd(B=0) == _lib.ERR_BAD_ARG
    assert _fwd(dtype=7) == _lib.ERR_UNSUPPORTED
    assert _fwd(H=4, ks=5) == _lib.ERR_WINDOW
    assert _fwd(W=3, ks=5) == _lib.ERR_WINDOW
    assert _fwd(Cd=512, path=_lib.PATH_SIMT) == _lib.ERR_UNSUPPORTED
    assert _fwd(dtype=0, path=_lib.PATH_TENSOR) == _lib.ERR_UNSUPPORTED      # fp32 has no tensor path
    assert _fwd(path=9) == _lib.ERR_BAD_ARG
    # row views: the key band must cover the query band's windows
    ok = _lib.Rows(8, 8, 6, 12, 32)
    assert _fwd(rows=C.byref(_lib.Rows(8, 8, 8, 8, 32))) == _lib.ERR_WINDOW
    assert _fwd(rows=C.byref(_lib.Rows(8, 8, 6, 9, 32))) == _lib.ERR_WINDOW
    assert _fwd(rows=C.byref(_lib.Rows(30, 8, 20, 12, 32))) == _lib.ERR_BAD_ARG
    assert _fwd(rows=C.byref(ok)) in (_lib.ERR_CUDA, _lib.ERR_NO_DEVICE)     # past validation: needs a GPU


def test_checks_refuse_a_device_that_does_not_exist():
    for device in (-1, 64):
        assert _lib.lib.na2d_poll(device, None) == _lib.ERR_BAD_ARG
    assert _lib.lib.na2d_poll(63, None) == _lib.ERR_CUDA and _lib.lib.na2d_check(63, None) == _lib.ERR_CUDA


def _args(**kw):
    a = _lib.Args()
    a.struct_size = C.sizeof(_lib.Args)
    a.op, a.B, a.N, a.H, a.W, a.C, a.kernel_size, a.dtype, a.path, a.device = 0, 1, 1, 8, 8, 32, 5, 1, 0, 0
    a.scale = 1.0
    for name in ("q", "k", "v", "o"):
        setattr(a, name, _lib.TensorDesc(256, 0, 0, 0, 0))       # dummy, never dereferenced
    a.lse = 256
    for k_, v_ in kw.items():
        setattr(a, k_, v_)
    return a


def test_ex_entry_points_refuse_bad_arguments_without_touching_cuda():
    fwd = lambda a: _lib.lib.na2d_forward_ex(C.byref(a))
    assert _lib.lib.na2d_forward_ex(None) == _lib.ERR_BAD_ARG
    assert fwd(_args(struct_size=8)) == _lib.ERR_BAD_ARG            # a caller built against another header
    assert fwd(_args(scale=0.0)) == _lib.ERR_BAD_ARG
    assert fwd(_args(scale=-1.0)) == _lib.ERR_BAD_ARG
    assert fwd(_args(scale=float("nan"))) == _lib.ERR_BAD_ARG
    assert fwd(_args(op=7)) == _lib.ERR_BAD_ARG
    assert fwd(_args(op=_lib.OP_1D)) == _lib.ERR_BAD_ARG            # the 1D operator wants H = 1
    assert fwd(_args(op=_lib.OP_1D, H=1, W=4)) == _lib.ERR_WINDOW   # sequence shorter than the window
    assert fwd(_args(kernel_size=6)) == _lib.ERR_BAD_ARG
    # a layout the tensor-core kernels cannot take (TMA wants 16-byte multiples): refused when that
    # path is demanded, served by the SIMT kernels under AUTO (which then needs a GPU)
    odd = _lib.TensorDesc(256, 8 * 8 * 36, 8 * 8 * 36, 8 * 36, 36)
    assert fwd(_args(q=odd, path=_lib.PATH_TENSOR)) == _lib.ERR_UNSUPPORTED
    assert fwd(_args(q=_lib.TensorDesc(258, 0, 0, 0, 0), path=_lib.PATH_TENSOR)) == _lib.ERR_UNSUPPORTED
    assert fwd(_args(q=odd)) in (_lib.ERR_CUDA, _lib.ERR_NO_DEVICE)
    assert fwd(_args()) in (_lib.ERR_CUDA, _lib.ERR_NO_DEVICE)      # past validation: needs a GPU


def test_header_without_workspace_fields():
    """A struct_size that ends before the workspace fields is accepted, one byte less is not."""
    base = _lib.Args.workspace.offset
    assert _lib.lib.na2d_forward_ex(C.byref(_args(struct_size=base))) in (_lib.ERR_CUDA, _lib.ERR_NO_DEVICE)
    assert _lib.lib.na2d_forward_ex(C.byref(_args(struct_size=base - 1))) == _lib.ERR_BAD_ARG


def test_workspace_is_bounded():
    """What the backward asks for: all weights where they are few, at most 512 MiB else (32 image rows if those are more)."""
    ask = lambda **kw: _lib.lib.na2d_backward_workspace(C.byref(_args(**kw)))
    weights = lambda H, W, ks: 2 * H * W * ks * (ks + 3) * 4           # P and dS, ks + 3 columns for four pixels
    assert ask(dtype=0, H=64, W=64, B=2, N=3) == 6 * weights(64, 64, 5)
    assert ask(dtype=0, H=64, W=64, B=200, N=3) <= 512 << 20
    assert ask(dtype=0, op=_lib.OP_1D, H=1, W=4096, kernel_size=13) == 2 * 4096 * 16 * 4
    for H, W, ks in ((1024, 1024, 13), (4096, 4096, 13), (16384, 2048, 3), (2000, 3000, 9)):
        assert 128 << 20 <= ask(dtype=0, H=H, W=W, kernel_size=ks, B=2) <= 512 << 20
    assert ask(dtype=0, H=1024, W=1 << 17, kernel_size=13) <= weights(32, 1 << 17, 13)
    assert ask(dtype=0, C=128, H=16, W=16, kernel_size=3) == 16 * 16 * 4    # few pixels, no tiles: a factor per row
    assert ask(dtype=0, H=64, W=64, kernel_size=15) == 64 * 64 * 4
    assert ask(C=64, H=64, W=64) == 0                                  # bf16 on tensor cores has no use for one


def test_unfused_pair_and_1d_refuse_bad_arguments_without_touching_cuda():
    p = C.c_void_p(256)
    assert _lib.lib.na2d_qk_forward(None, p, p, 1, 1, 8, 8, 32, 5, 0, 0, None) == _lib.ERR_BAD_ARG
    assert _lib.lib.na2d_qk_forward(p, p, p, 1, 1, 4, 8, 32, 5, 0, 0, None) == _lib.ERR_WINDOW
    assert _lib.lib.na2d_av_forward(p, p, p, 1, 1, 8, 8, 32, 4, 0, 0, None) == _lib.ERR_BAD_ARG
    assert _lib.lib.na2d_av_backward(p, p, p, p, None, 1, 1, 8, 8, 32, 5, 0, 0, None) == _lib.ERR_BAD_ARG
    assert _lib.lib.na1d_forward(p, p, p, p, p, 1, 1, 4, 32, 5, 0, 0, None) == _lib.ERR_WINDOW
    assert _lib.lib.na1d_forward(p, p, p, p, None, 1, 1, 16, 32, 5, 0, 0, None) == _lib.ERR_BAD_ARG


def test_kernel_ready_layouts():
    """Which tensors go to the kernels in place and which are copied first."""
    from e_natten_b200.functional import _kernel_ready
    packed = torch.zeros(2, 10, 9, 3, 4, 64, dtype=torch.bfloat16)          # (B, H, W, 3, heads, C)
    q = packed[:, :, :, 0].permute(0, 3, 1, 2, 4)
    assert not q.is_contiguous() and _kernel_ready(q)
    assert not _kernel_ready(packed[:, :, :, 0].permute(0, 3, 1, 4, 2))     # channels not contiguous
    assert not _kernel_ready(torch.zeros(1, 1, 8, 8, 36, dtype=torch.bfloat16)[..., :32][:, :, :, 1:])  # stride 36
    assert _kernel_ready(torch.zeros(1, 1, 8, 8, 36)[..., :32])             # fp32: any strides
    assert not _kernel_ready(torch.zeros(1, 1, 8, 1, 32).expand(1, 1, 8, 8, 32))


def test_operand_strides():
    """Strides as the library gets them; ranks that are no operand's are refused, not read past their end."""
    strides = _lib.torch_ext.strides
    assert strides(torch.zeros(2, 3, 5, 7, 8)) == (840, 280, 56, 8)
    assert strides(torch.zeros(2, 3, 7, 8)) == (168, 56, 0, 8)              # (B, heads, T, C)
    packed = torch.zeros(2, 5, 7, 3, 4, 8)[:, :, :, 1].permute(0, 3, 1, 2, 4)
    assert strides(packed) == (3360, 8, 672, 96)
    assert strides(torch.zeros(2, 1, 5, 7, 8).as_strided((2, 1, 5, 7, 8), (280, 0, 56, 8, 1))) == (280, 1, 56, 8)
    for shape in ((7, 8), (3, 7, 8), (1, 2, 3, 5, 7, 8)):
        with pytest.raises(ValueError):
            strides(torch.zeros(shape))


def test_python_wrapper_refuses_cpu_tensors_and_bad_shapes():
    q = torch.zeros(1, 1, 8, 8, 32)
    with pytest.raises(ValueError, match="CUDA"):
        na.natten2d(q, q, q, 5)
    with pytest.raises(ValueError):
        na.natten2d(torch.zeros(1, 8, 8, 32), q, q, 5)
    with pytest.raises(TypeError):
        na.natten2d(None, q, q, 5)


def test_check_maps_status_to_exceptions():
    with pytest.raises(ValueError):
        _lib.check(_lib.ERR_WINDOW)
    with pytest.raises(RuntimeError):
        _lib.check(_lib.ERR_KERNEL_WAIT)
    _lib.check(0)


def test_build_is_stale_after_a_pytorch_change(monkeypatch):
    """The extension module belongs to one PyTorch; the library does not."""
    from e_natten_b200 import build
    assert not build._lib_stale() and not build._ext_stale()
    assert _lib.torch_ext.built_for == build._ext_tag()
    monkeypatch.setattr(build.importlib.metadata, "version", lambda name: "9.9.9")
    assert build._ext_stale() and not build._lib_stale()
