"""GPU tests of the tiled CUDA-core kernels (fp32, the 1D operator, head dims without tensor-core kernels)
at the sizes where they can go wrong: image sides around the tile and strip sizes, sides equal to the
window, head dims that leave a channel chunk part empty or rule out 16-byte loads, backwards that take
the units in several turns or have no workspace, and values that must not leave their windows."""
import ctypes as C
import math

import pytest
import torch

import e_natten_b200 as na
from e_natten_b200 import _lib
from e_natten_b200 import functional as F
from oracle import na2d_oracle as orc
from helpers import assert_close, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (kernel size, H, W, C): sides one below, at and above the 8-row, 4-column and 8- / 16-column tile edges,
# whole-window images, and images whose every tile meets two borders
CASES = [(3, 3, 3, 4), (3, 8, 15, 32), (3, 17, 33, 70), (5, 5, 9, 2), (5, 16, 16, 128), (5, 19, 37, 40),
         (7, 7, 16, 33), (7, 21, 22, 96), (9, 9, 9, 48), (9, 25, 24, 36), (11, 11, 43, 64), (11, 26, 26, 20),
         (13, 13, 13, 256), (13, 14, 14, 64), (13, 26, 33, 96)]


def _units(H, W, ks, dtype):
    """Units of so many pixels that the tiled kernels take the call; fewer go to the warp-per-pixel kernels."""
    pixels = {3: 16384, 5: 8192}.get(ks, 4096) if H > 1 else 12288
    return -(-pixels * (1 if dtype == torch.float32 else 2) // (H * W))


def _device(*ts):
    return tuple(t.to(DEV) for t in ts)


@pytest.mark.parametrize("ks,H,W,Cd", CASES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("many", [True, False])
def test_2d_against_oracle(ks, H, W, Cd, dtype, many):
    scale = Cd ** -0.5
    q, k, v, d_o = make_inputs((1, _units(H, W, ks, dtype) if many else 2, H, W, Cd), dtype, 900 + ks + H)
    ro, rlse = orc.natten2d_fwd(q, k, v, ks, scale=scale)
    rdq, rdk, rdv = orc.natten2d_bwd(q, k, v, d_o, ks, scale=scale)
    qd, kd, vd, gd = _device(q, k, v, d_o)
    o, lse = na.natten2d_forward(qd, kd, vd, ks, path="simt", scale=scale)
    a = F._args(qd, ks, None, "simt", scale, q=qd, k=kd, v=vd)
    assert not many or _lib.lib.na2d_backward_workspace(C.byref(a)) > 8 * lse.numel()      # weights, not row factors
    dq, dk, dv = na.natten2d_backward(qd, kd, vd, o, lse, gd, ks, path="simt", scale=scale)
    for got, want, what in ((o, ro, "o"), (lse, rlse, "lse"), (dq, rdq, "dq"), (dk, rdk, "dk"), (dv, rdv, "dv")):
        assert_close(got, want, torch.float32 if what == "lse" else dtype, f"{what} ks={ks} {H}x{W}x{Cd} {dtype}")


@pytest.mark.parametrize("ks,T,Cd", [(3, 3, 8), (5, 127, 40), (7, 128, 32), (9, 129, 48), (11, 11, 6), (13, 300, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("many", [True, False])
def test_1d_against_oracle(ks, T, Cd, dtype, many):
    g = torch.Generator().manual_seed(ks + T)
    q, k, v, d_o = (torch.randn((2, _units(1, T, ks, dtype) if many else 3, T, Cd), generator=g).to(dtype) for _ in range(4))
    ro, rlse = orc.natten1d_fwd(q, k, v, ks, scale=0.3)
    rdq, rdk, rdv = orc.natten1d_bwd(q, k, v, d_o, ks, scale=0.3)
    qd, kd, vd, gd = _device(q, k, v, d_o)
    o, lse = F.natten1d_forward(qd, kd, vd, ks, 0.3)
    dq, dk, dv = F.natten1d_backward(qd, kd, vd, o, lse, gd, ks, scale=0.3)
    for got, want, what in ((o, ro, "o"), (lse, rlse, "lse"), (dq, rdq, "dq"), (dk, rdk, "dk"), (dv, rdv, "dv")):
        assert_close(got, want, torch.float32 if what == "lse" else dtype, f"{what} ks={ks} T={T} C={Cd} {dtype}")


@pytest.mark.parametrize("ks,H,W,Cd", [(5, 19, 37, 40), (13, 14, 30, 64), (3, 9, 9, 30)])
def test_packed_views_equal_dense(ks, H, W, Cd):
    """Strided operands, vector loads or not, give what dense ones give, bit for bit."""
    g = torch.Generator().manual_seed(3)
    N = _units(H, W, ks, torch.float32)
    qkv = torch.randn((2, H, W, 3, N, Cd), generator=g).to(DEV)
    d_o = torch.randn((2, H, W, N, Cd), generator=g).to(DEV).permute(0, 3, 1, 2, 4)
    views = qkv.permute(3, 0, 4, 1, 2, 5).unbind(0)
    dense = tuple(t.contiguous() for t in views)
    o1, l1 = na.natten2d_forward(*views, ks, scale=0.2)
    o2, l2 = na.natten2d_forward(*dense, ks, scale=0.2)
    assert torch.equal(o1, o2) and torch.equal(l1, l2)
    for a, b in zip(na.natten2d_backward(*views, o1, l1, d_o, ks, scale=0.2),
                    na.natten2d_backward(*dense, o2, l2, d_o.contiguous(), ks, scale=0.2)):
        assert torch.equal(a, b)


def _off_boundary(t):
    """The same tensor, its rows starting 4 bytes past a 16-byte boundary: fp32 operands that stay with these kernels in 2D."""
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    return flat[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("ks,H,W", [(5, 20, 21), (9, 12, 33)])
@pytest.mark.parametrize("off", [False, True])
def test_workspace_of_any_size(ks, H, W, off):
    """All units at once, one unit at a time, and no workspace (the key half forms the weights again)."""
    B, N, Cd = 1, _units(H, W, ks, torch.float32), 64
    q, k, v, d_o = _device(*make_inputs((B, N, H, W, Cd), torch.float32, 77))
    if off:
        q, k, v, d_o = (_off_boundary(t) for t in (q, k, v, d_o))
    o, lse = na.natten2d_forward(q, k, v, ks, scale=0.125)
    want = orc.natten2d_bwd(q.cpu(), k.cpu(), v.cpu(), d_o.cpu(), ks, scale=0.125)
    delta = torch.empty_like(lse)

    def run(units):
        grads = [torch.full_like(q, float("nan")) for _ in range(3)]
        a = F._args(q, ks, None, "auto", 0.125, q=q, k=k, v=v, o=o, lse=lse, d_o=d_o, d_q=grads[0], d_k=grads[1],
                    d_v=grads[2], delta=delta)
        per_unit = _lib.lib.na2d_backward_workspace(C.byref(a)) // (B * N)
        assert per_unit >= 2 * H * W * ks * ks * 4 and per_unit % 16 == 0
        scratch = torch.full((units * per_unit // 4 + 4,), -1.0, device=DEV)
        a.workspace, a.workspace_bytes = (scratch.data_ptr(), units * per_unit) if units else (None, 0)
        _lib.check(_lib.lib.na2d_backward_ex(C.byref(a)))
        assert bool((scratch[units * per_unit // 4:] == -1.0).all())            # nothing beyond what was given
        return grads

    whole = run(N)
    for g, w, what in zip(whole, want, ("dq", "dk", "dv")):
        assert_close(g, w, torch.float32, what)
    for units in (1, 2, N - 1):
        assert all(torch.equal(x, y) for x, y in zip(run(units), whole))
    for g, w, what in zip(run(0), want, ("dq", "dk", "dv")):
        assert_close(g, w, torch.float32, what + " without workspace")


def _backward(q, k, v, o, lse, d_o, ks, scale, bytes_of, path="auto"):
    """Gradients with a workspace of bytes_of(what is asked for) bytes; nothing beyond it may be written."""
    delta = torch.empty_like(lse)
    grads = [torch.full_like(q, float("nan")) for _ in range(3)]
    a = F._args(q, ks, None, path, scale, q=q, k=k, v=v, o=o, lse=lse, d_o=d_o, d_q=grads[0], d_k=grads[1], d_v=grads[2],
                delta=delta)
    n = bytes_of(_lib.lib.na2d_backward_workspace(C.byref(a))) // 4
    scratch = torch.full((n + 4,), -1.0, device=DEV)
    a.workspace, a.workspace_bytes = scratch.data_ptr(), 4 * n
    before = na.launch_count()
    _lib.check(_lib.lib.na2d_backward_ex(C.byref(a)))
    assert bool((scratch[n:] == -1.0).all())
    return grads, na.launch_count() - before


@pytest.mark.parametrize("ks,H,W,dtype,off", [(3, 41, 9, torch.float32, False), (5, 67, 18, torch.bfloat16, False),
                                              (9, 50, 19, torch.float32, False), (13, 75, 14, torch.float32, False),
                                              (3, 41, 9, torch.float32, True), (5, 67, 18, torch.float32, True),
                                              (9, 50, 19, torch.float32, True), (13, 75, 14, torch.float32, True)])
def test_workspace_of_some_rows(ks, H, W, dtype, off):
    """A workspace below one image: rows of tiles are used again as the key half is done with them."""
    Cd, scale = 40, 0.2
    N = _units(H, W, ks, dtype)
    q, k, v, d_o = _device(*make_inputs((1, N, H, W, Cd), dtype, 78))
    if off:
        q, k, v, d_o = (_off_boundary(t) for t in (q, k, v, d_o))
    o, lse = na.natten2d_forward(q, k, v, ks, path="simt", scale=scale)
    run = lambda bytes_of: _backward(q, k, v, o, lse, d_o, ks, scale, bytes_of, path="simt")
    whole, launches = run(lambda n: n)
    assert launches == 2
    tile_rows = -(-H // 8)
    least = 3 if ks <= 9 else 4                                  # tile rows that 8 rows of keys meet
    for rows in range(least, tile_rows):
        got, launches = run(lambda n: n // (N * tile_rows) * rows + 60)
        assert launches >= 3 * N - 1 and all(torch.equal(x, y) for x, y in zip(got, whole)), rows
    want = orc.natten2d_bwd(q.cpu(), k.cpu(), v.cpu(), d_o.cpu(), ks, scale=scale)
    short, launches = run(lambda n: n // (N * tile_rows) * (least - 1))
    assert launches == 2                                         # too short: without it
    for g, w, what in zip(short, want, ("dq", "dk", "dv")):
        assert_close(g, w, dtype, what)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_workspace_of_some_sequences(dtype):
    g = torch.Generator().manual_seed(4)
    q, k, v, d_o = _device(*(torch.randn((1, 50, 300, 48), generator=g).to(dtype) for _ in range(4)))
    o, lse = F.natten1d_forward(q, k, v, 7, 0.2)
    run = lambda bytes_of: _backward(q, k, v, None, lse, d_o, 7, 0.2, bytes_of)
    whole, _ = run(lambda n: n)
    for units in (1, 20, 49):
        got, launches = run(lambda n: n // 50 * units + 12)
        assert launches == 2 * -(-50 // units) and all(torch.equal(x, y) for x, y in zip(got, whole))


def test_short_memory():
    """No room for the whole workspace: the extension asks for half as much, and the result stays the same."""
    torch.cuda.empty_cache()                                     # so that no segment below is half empty
    q, k, v, d_o = (torch.randn(1, 4, 256, 256, 32, device=DEV) for _ in range(4))
    o, lse = na.natten2d_forward(q, k, v, 5, scale=0.2)
    before = na.launch_count()
    want = na.natten2d_backward(q, k, v, o, lse, d_o, 5, scale=0.2)
    assert na.launch_count() - before == 2                       # 84 MB of weights, 21 per image
    want = [t.cpu() for t in want]
    torch.cuda.empty_cache()
    outputs = 3 * q.numel() * 4
    limit = torch.cuda.memory_reserved() + outputs + (72 << 20)
    try:
        torch.cuda.set_per_process_memory_fraction(limit / torch.cuda.get_device_properties(0).total_memory)
        before = na.launch_count()
        got = na.natten2d_backward(q, k, v, o, lse, d_o, 5, scale=0.2)
        assert na.launch_count() - before == 4
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert all(torch.equal(x.cpu(), y) for x, y in zip(got, want))


@pytest.mark.parametrize("ks", [3, 5, 9])
@pytest.mark.parametrize("at", [(0, 0), (7, 7), (8, 16), (23, 30)])
@pytest.mark.parametrize("off", [False, True])
def test_infinities_stay_in_their_windows(ks, at, off):
    """An infinite value (and an infinite gradient) reaches the pixels whose windows hold it and no others."""
    H, W = 24, 31
    q, k, v, d_o = _device(*make_inputs((1, _units(H, W, ks, torch.float32), H, W, 32), torch.float32, 5, q_scale=0.2))
    clone = torch.clone
    if off:
        q, k, v, d_o = (_off_boundary(t) for t in (q, k, v, d_o))
        clone = _off_boundary
    v2, g2 = clone(v), clone(d_o)
    v2[0, 0, at[0], at[1]] = float("inf")
    g2[0, 0, at[0], at[1]] = float("inf")
    o, lse = na.natten2d_forward(q, k, v, ks)
    o2, lse2 = na.natten2d_forward(q, k, v2, ks)
    rows = torch.tensor([na.get_window_start(y, H, ks) <= at[0] < na.get_window_start(y, H, ks) + ks for y in range(H)])
    cols = torch.tensor([na.get_window_start(x, W, ks) <= at[1] < na.get_window_start(x, W, ks) + ks for x in range(W)])
    reached = (rows[:, None] & cols[None, :]).to(DEV)
    assert torch.equal(torch.isinf(o2[0, 0]).all(-1), reached) and torch.equal(lse, lse2)
    assert torch.equal(o2[0, 0][~reached], o[0, 0][~reached])
    _, _, dv = na.natten2d_backward(q, k, v, o, lse, d_o, ks)
    dq2, dk2, dv2 = na.natten2d_backward(q, k, v, o, lse, g2, ks)
    ys = slice(na.get_window_start(at[0], H, ks), na.get_window_start(at[0], H, ks) + ks)
    xs = slice(na.get_window_start(at[1], W, ks), na.get_window_start(at[1], W, ks) + ks)
    held = torch.zeros(H, W, dtype=torch.bool, device=DEV)
    held[ys, xs] = True
    assert torch.equal(~torch.isfinite(dv2[0, 0]).all(-1), held)
    assert torch.equal(dv2[0, 0][~held], dv[0, 0][~held])
    assert torch.isfinite(dk2[0, 0][~held]).all()


@pytest.mark.parametrize("excess", [2e-5, 5e-4, 0.3])
@pytest.mark.parametrize("workspace", [True, False])
def test_merged_lse(excess, workspace):
    """An lse over more than the window (a merged one): the weights are exp(s - lse), however little the rest adds."""
    ks, H, W, Cd = 5, 19, 37, 40
    q, k, v, d_o = _device(*make_inputs((1, _units(H, W, ks, torch.float32), H, W, Cd), torch.float32, 31))
    o, lse = na.natten2d_forward(q, k, v, ks, scale=0.2)
    lse = (lse.double() + math.log1p(excess)).float()
    delta, grads = torch.empty_like(lse), [torch.empty_like(q) for _ in range(3)]
    a = F._args(q, ks, None, "auto", 0.2, q=q, k=k, v=v, o=o, lse=lse, d_o=d_o, d_q=grads[0], d_k=grads[1], d_v=grads[2],
                delta=delta)
    scratch = torch.empty(_lib.lib.na2d_backward_workspace(C.byref(a)), dtype=torch.uint8, device=DEV)
    if workspace:
        a.workspace, a.workspace_bytes = scratch.data_ptr(), scratch.numel()
    _lib.check(_lib.lib.na2d_backward_ex(C.byref(a)))
    want = orc.natten2d_bwd(q.cpu(), k.cpu(), v.cpu(), d_o.cpu(), ks, scale=0.2, lse=lse.cpu())
    for g, w, what in zip(grads, want, ("dq", "dk", "dv")):
        # rounding of s and lse: a few 1e-6 of the norm; a sum brought back to 1 would be off by `excess`
        err = (g.cpu().double() - w).norm() / w.norm()
        assert err < 5e-6, f"{what}: {err:.2e}"


@pytest.mark.parametrize("Cd", [32, 40, 64, 96, 128, 256])
@pytest.mark.parametrize("ks", [3, 7])
def test_scores_round_no_more_than_a_sum_over_lanes(Cd, ks):
    """Error of the scores against 64 bits, over normal rows: at most that of the products summed over 32 lanes (lane l
    holds channels l, l + 32, ..., then a tree), the order of the warp-per-pixel kernels.  A running sum
    over all channels has 1.09 times it at 64, 1.25 at 128 and 1.43 at 256."""
    H, W = 40, 44
    B, N = 1, _units(H, W, ks, torch.float32)
    q, k, _, _ = make_inputs((B, N, H, W, Cd), torch.float32, Cd + ks)
    want = orc.natten2d_qk(q, k, ks)
    got = na.natten2dqk(*_device(q, k), ks).cpu().double()
    rows, cols = orc.window_start_table(H, ks), orc.window_start_table(W, ks)
    lane_err = 0.0
    for u, w in ((0, 0), (1, 2), (2, 1)):                         # every member has the same distribution
        kk = k.index_select(2, rows + u).index_select(3, cols + w)
        lanes = torch.zeros(B, N, H, W, 32)
        for c in range(0, Cd, 32):
            n = min(32, Cd - c)
            lanes[..., :n] = (q[..., c:c + n].double() * kk[..., c:c + n].double() + lanes[..., :n].double()).float()
        while lanes.shape[-1] > 1:
            half = lanes.shape[-1] // 2
            lanes = lanes[..., :half] + lanes[..., half:]
        ref = (q.double() * kk.double()).sum(-1)
        lane_err += ((lanes[..., 0].double() - ref).norm() / ref.norm()).item() / 3
    err = ((got - want).norm() / want.norm()).item()
    assert err <= lane_err, f"{err:.3e} against {lane_err:.3e}"


@pytest.mark.parametrize("Cd", [32, 64, 96, 256])
def test_minus_infinite_scores(Cd):
    """A key that scores minus infinity has no weight and takes nothing else with it, whatever is summed around it."""
    ks, H, W, at = 5, 18, 21, (7, 9)
    q, k, v, _ = make_inputs((1, _units(H, W, ks, torch.float32), H, W, Cd), torch.float32, 8, q_scale=0.2)
    q = q.abs()
    k[0, 0, at[0], at[1], Cd // 3] = -float("inf")
    k2 = k.clone()
    k2[0, 0, at[0], at[1]] = -1e4                                    # as good as that
    want, want_lse = orc.natten2d_fwd(q, k2, v, ks)
    o, lse = na.natten2d_forward(*_device(q, k, v), ks)
    assert_close(o, want, torch.float32, "o")
    assert_close(lse, want_lse, torch.float32, "lse")


@pytest.mark.parametrize("Cd,ks", [(32, 3), (64, 5), (128, 3), (64, 15)])
def test_few_pixels_keep_the_rounding_of_lse_out(Cd, ks):
    """The warp-per-pixel halves of small problems, logits of 10 and more: with the factor per row that they ask a
    workspace for, the rounding of lse (half an ulp of 16 here, 1e-6) does not reach dK and dV."""
    H, W = 20, 22
    q, k, v, d_o = make_inputs((1, 2, H, W, Cd), torch.float32, 17 + Cd)
    want = orc.natten2d_bwd(q, k, v, d_o, ks)
    dev = _device(q, k, v)
    o, lse = na.natten2d_forward(*dev, ks)
    err = lambda x, w: ((x.cpu().double() - w).norm() / w.norm()).item()
    given, _ = _backward(*dev, o, lse, d_o.to(DEV), ks, 1.0, lambda n: n)
    without, _ = _backward(*dev, o, lse, d_o.to(DEV), ks, 1.0, lambda n: 0)
    assert all(torch.isfinite(t).all() for t in given + without) and torch.equal(given[0], without[0])
    for i, most, what in ((1, 1.0, "dk"), (2, 0.8, "dv")):       # dK also has the scores' own rounding in dP - delta
        assert err(given[i], want[i]) < most * err(without[i], want[i]), what


@pytest.mark.parametrize("ks", [15, 27, 29, 31])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_windows_beyond_the_tiles(ks, dtype):
    """Kernel sizes up to the largest; from 29 on the query half needs more than 48 KB of shared memory."""
    q, k, v, d_o = make_inputs((1, 2, 31, 34, 40), dtype, ks, q_scale=0.16)
    ro, rlse = orc.natten2d_fwd(q, k, v, ks)
    want = orc.natten2d_bwd(q, k, v, d_o, ks)
    qd, kd, vd, gd = _device(q, k, v, d_o)
    o, lse = na.natten2d_forward(qd, kd, vd, ks)
    assert_close(o, ro, dtype, "o")
    assert_close(lse, rlse, torch.float32, "lse")
    for got, w, what in zip(na.natten2d_backward(qd, kd, vd, o, lse, gd, ks), want, ("dq", "dk", "dv")):
        assert_close(got, w, dtype, what)


@pytest.mark.parametrize("shape,ks,dtype", [((1, 24, 20, 21, 40), 5, torch.float32), ((1, 2, 30, 33, 64), 9, torch.bfloat16),
                                            ((2, 40, 300, 64), 7, torch.bfloat16)])
def test_on_another_stream(shape, ks, dtype):
    """The native path launches on the current stream, behind the work that makes its inputs, and its outputs and
    scratch belong to that stream."""
    g = torch.Generator().manual_seed(9)
    inputs = [torch.randn(shape, generator=g).to(dtype).to(DEV) for _ in range(4)]
    forward, backward = ((na.natten2d_forward, na.natten2d_backward) if len(shape) == 5 else
                         (F.natten1d_forward, F.natten1d_backward))
    o, lse = forward(*inputs[:3], ks)
    want = (o, lse, *backward(*inputs[:3], o, lse, inputs[3], ks))
    torch.cuda.synchronize()
    busy = torch.randn(4096, 4096, device=DEV)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        late = [torch.full_like(t, float("nan")) for t in inputs]
        for _ in range(20):
            busy = (busy @ busy).clamp_(-1, 1)
        for t, x in zip(late, inputs):
            t.copy_(x)                                           # the inputs are there once `busy` is done
        o2, lse2 = forward(*late[:3], ks)
        got = (o2, lse2, *backward(*late[:3], o2, lse2, late[3], ks))
        [torch.full_like(t, float("nan")) for t in got]          # takes freed scratch of this stream again
    stream.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("ks,Cd", [(7, 32), (9, 64), (13, 128)])
def test_infinities_in_the_chunked_query_half(ks, Cd):
    """An infinite value and an infinite gradient in the query half of the larger windows on tensor cores, which walks the
    key box in chunks: dQ of the pixels whose windows hold them, and no others, is not finite.  (o is that of
    finite values: the forward's P V leaves the window's bounds to zeros of P, so there an infinity spreads over a tile.)"""
    H, W, at = 40, 37, (17, 9)
    q, k, v, d_o = _device(*make_inputs((1, 2, H, W, Cd), torch.bfloat16, 6, q_scale=0.2))
    o, lse = na.natten2d_forward(q, k, v, ks, path="tensor")
    clean, _, _ = na.natten2d_backward(q, k, v, o, lse, d_o, ks, path="tensor", need_dkdv=False)
    v2 = v.clone()
    v2[0, 0, at[0], at[1]] = float("inf")
    dirty, _, _ = na.natten2d_backward(q, k, v2, o, lse, d_o, ks, path="tensor", need_dkdv=False)
    holds = lambda n, i: [na.get_window_start(y, n, ks) <= i < na.get_window_start(y, n, ks) + ks for y in range(n)]
    reached = (torch.tensor(holds(H, at[0]))[:, None] & torch.tensor(holds(W, at[1]))[None, :]).to(DEV)
    assert torch.equal(~torch.isfinite(dirty[0, 0]).all(-1), reached)
    assert torch.equal(dirty[0, 0][~reached], clean[0, 0][~reached]) and torch.equal(dirty[0, 1], clean[0, 1])
    g2 = d_o.clone()
    g2[0, 0, at[0], at[1]] = float("inf")
    dirty, _, _ = na.natten2d_backward(q, k, v, o, lse, g2, ks, path="tensor", need_dkdv=False)
    itself = torch.zeros(H, W, dtype=torch.bool, device=DEV)
    itself[at] = True
    assert torch.equal(~torch.isfinite(dirty[0, 0]).all(-1), itself)
    assert torch.equal(dirty[0, 0][~itself], clean[0, 0][~itself])


@pytest.mark.parametrize("ks,Cd,dtype", [(3, 32, torch.float16), (5, 64, torch.bfloat16), (5, 128, torch.bfloat16)])
def test_strip_forward_hand_overs(ks, Cd, dtype):
    """Many tiles per block and many launches beside a kernel that takes instruction slots and memory bandwidth from the
    softmax warps at odd moments: every hand-over between the warps takes place (no bounded wait runs out), and the
    results stay the same."""
    q, k, v, _ = _device(*make_inputs((2, 4, 96, 200, Cd), dtype, 12, q_scale=0.2))
    o, lse = na.natten2d_forward(q, k, v, ks)
    other, noise = torch.cuda.Stream(), torch.randn(1 << 22, device=DEV)
    torch.cuda.synchronize()
    for _ in range(40):
        with torch.cuda.stream(other):
            noise = torch.sin(noise)
        for _ in range(20):
            o2, lse2 = na.natten2d_forward(q, k, v, ks)
        assert torch.equal(o2, o) and torch.equal(lse2, lse)
    na.check_kernels(DEV)
