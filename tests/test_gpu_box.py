"""GPU tests of the fp32 kernels on TMA boxes (na2d_box.cuh) against the CPU oracle and against the tiled kernels, which take the
same call when its operands start off a 16-byte boundary: image sides around the tiles, head dims around the channel chunks, borders
that meet, memory orders of every kind, bands of rows, and infinities at the borders."""
import pytest
import torch

import e_natten_b200 as na
from oracle import na2d_oracle as orc
from helpers import assert_close, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (kernel size, H, W, C): tiles are 8 rows by 16 columns up to window 7, by 8 beyond; chunks are 16 and 32 channels
CASES = [(3, 3, 3, 16), (3, 9, 17, 4), (3, 24, 34, 36), (5, 5, 6, 12), (5, 12, 20, 64), (5, 41, 37, 20), (5, 16, 21, 132), (7, 8, 7, 32),
         (7, 23, 33, 68), (9, 9, 17, 48), (9, 26, 25, 16), (11, 11, 12, 28), (11, 30, 35, 64), (13, 13, 13, 4), (13, 33, 31, 36), (13, 14, 64, 96)]


def _units(H, W):
    """Units of so many pixels that the call is not left to the warp-per-pixel kernels."""
    return -(-20000 // (H * W))


def _off_boundary(t):
    """The same tensor, its rows starting 4 bytes past a 16-byte boundary: no tensor map describes it."""
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    return flat[1:].view(t.shape).copy_(t)


def _step(q, k, v, d_o, ks, scale):
    o, lse = na.natten2d_forward(q, k, v, ks, scale=scale)
    return (o, lse, *na.natten2d_backward(q, k, v, o, lse, d_o, ks, scale=scale))


@pytest.mark.parametrize("ks,H,W,Cd", CASES)
def test_step_against_oracle_and_tiles(ks, H, W, Cd):
    scale = Cd ** -0.5
    ins = make_inputs((1, _units(H, W), H, W, Cd), torch.float32, 40 + ks + W)
    q, k, v, d_o = (t.to(DEV) for t in ins)
    got = _step(q, k, v, d_o, ks, scale)
    tiles = _step(*(_off_boundary(t) for t in (q, k, v, d_o)), ks, scale)
    ro, rlse = orc.natten2d_fwd(*ins[:3], ks, scale=scale)
    want = (ro, rlse, *orc.natten2d_bwd(*ins, ks, scale=scale))
    for a, b, c, what in zip(got, tiles, want, ("o", "lse", "dq", "dk", "dv")):
        assert_close(a, c, torch.float32, f"{what} ks={ks} {H}x{W}x{Cd}")
        # the two sum the same numbers in other orders: each is within 4e-6 of the tensor's largest value of the exact sum (windows up to 13)
        assert (a - b).abs().max().item() <= 2e-5 * c.abs().max().item(), what
    na.check_kernels()


@pytest.mark.parametrize("H,W,Cd,tiles", [(17, 37, 68, 740), (15, 36, 96, 296), (14, 40, 20, 296)])
def test_window_13_of_many_tiles(H, W, Cd, tiles):
    """So many tiles that the query side of the largest window goes to the boxes, too."""
    ks, few = 13, 5
    units = tiles // (-(-H // 8) * 5) + 1
    q, k, v, d_o = (t.to(DEV) for t in make_inputs((1, units, H, W, Cd), torch.float32, Cd))
    got = _step(q, k, v, d_o, ks, Cd ** -0.5)
    tiles = _step(*(_off_boundary(t) for t in (q, k, v, d_o)), ks, Cd ** -0.5)
    ins = [t[:, -few:].cpu() for t in (q, k, v, d_o)]
    want = (*orc.natten2d_fwd(*ins[:3], ks, scale=Cd ** -0.5), *orc.natten2d_bwd(*ins, ks, scale=Cd ** -0.5))
    for a, b, c, what in zip(got, tiles, want, ("o", "lse", "dq", "dk", "dv")):
        assert_close(a[:, -few:], c, torch.float32, what)
        assert (a - b).abs().max().item() <= 2e-5 * b.abs().max().item(), what
    na.check_kernels()


@pytest.mark.parametrize("order", [(0, 1, 2, 3), (0, 2, 1, 3), (2, 0, 1, 3), (1, 2, 0, 3), (0, 3, 2, 1), (3, 2, 1, 0)])
@pytest.mark.parametrize("ks", [5, 9])
def test_any_memory_order(order, ks):
    """Batch, head, row and column may lie in memory in any order (channels last): bit for bit what dense operands give."""
    shape = (3, 4, 26, 37, 36)
    back = [order.index(i) for i in range(4)]
    ts = [t.to(DEV) for t in make_inputs(shape, torch.float32, 7)]
    strided = [t.permute(*order, 4).contiguous().permute(*back, 4) for t in ts]
    for a, b in zip(_step(*strided, ks, 0.2), _step(*ts, ks, 0.2)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("ks,H,W,Cd", [(3, 20, 18, 32), (5, 30, 21, 64), (7, 17, 40, 48), (13, 26, 27, 20)])
def test_pair_against_tiles(ks, H, W, Cd):
    q, k, v, d_o = (t.to(DEV) for t in make_inputs((2, _units(H, W), H, W, Cd), torch.float32, 3, q_scale=Cd ** -0.5))

    def run(q, k, v, d_o):
        q, k, v = (t.requires_grad_() for t in (q, k, v))
        attn = na.natten2dqk(q, k, ks, 1)
        out = na.natten2dav(torch.softmax(attn, -1), v, ks, 1)
        return (attn.detach(), out.detach(), *torch.autograd.grad(out, (q, k, v), d_o))

    r = [t.cpu() for t in (q, k, v, d_o)]
    want = (orc.natten2d_qk(r[0].double(), r[1].double(), ks), orc.natten2d_fwd(*r[:3], ks, scale=1.0)[0], *orc.natten2d_bwd(*r, ks, scale=1.0))
    got = run(q.clone(), k.clone(), v.clone(), d_o)
    tiles = run(*(_off_boundary(t) for t in (q, k, v, d_o)))
    for a, b, c, what in zip(got, tiles, want, ("scores", "o", "dq", "dk", "dv")):
        assert_close(a, c, torch.float32, f"{what} ks={ks} {H}x{W}x{Cd}")
        assert_close(b, c, torch.float32, f"tiles, {what} ks={ks} {H}x{W}x{Cd}")
    na.check_kernels()


@pytest.mark.parametrize("ks,H,W", [(3, 40, 33), (7, 37, 28), (13, 45, 30)])
def test_bands_of_rows_equal_the_image(ks, H, W):
    """Query rows in bands, whose key rows start anywhere: bit for bit the whole image's o and dQ."""
    q, k, v, d_o = (t.to(DEV) for t in make_inputs((1, _units(H, W), H, W, 32), torch.float32, 11))
    o, lse = na.natten2d_forward(q, k, v, ks, scale=0.2)
    dq, _, _ = na.natten2d_backward(q, k, v, o, lse, d_o, ks, scale=0.2)
    for r0, r1 in ((0, 13), (13, 30), (30, H)):
        lo, hi = na.get_window_start(r0, H, ks), na.get_window_start(r1 - 1, H, ks) + ks
        rows = na.make_rows(r0, r1 - r0, lo, hi - lo, H)
        qb, gb, kb, vb = q[:, :, r0:r1], d_o[:, :, r0:r1], k[:, :, lo:hi], v[:, :, lo:hi]
        ob, lseb = na.natten2d_forward(qb, kb, vb, ks, rows=rows, scale=0.2)
        dqb = na.natten2d_backward(qb, kb, vb, ob, lseb, gb, ks, rows=rows, scale=0.2, need_dkdv=False)[0]
        assert torch.equal(ob, o[:, :, r0:r1]) and torch.equal(lseb, lse[:, :, r0:r1]) and torch.equal(dqb, dq[:, :, r0:r1])


@pytest.mark.parametrize("ks", [3, 5, 7, 9, 13])
@pytest.mark.parametrize("column", [0, 1, 5, 14, 15, 16, 27, 32, 33])
@pytest.mark.parametrize("Cd", [32, 100])
def test_infinite_gradients_reach_the_window_only(ks, column, Cd):
    """One channel chunk, and several of them (the last one part empty) with scores parked in between."""
    H, W = 26, 34
    q, k, v, d_o = (t.to(DEV) for t in make_inputs((1, _units(H, W), H, W, Cd), torch.float32, 5, q_scale=0.2))
    o, lse = na.natten2d_forward(q, k, v, ks)
    _, dk, dv = na.natten2d_backward(q, k, v, o, lse, d_o, ks)
    d_o[0, 0, 2, column] = float("inf")
    _, dk2, dv2 = na.natten2d_backward(q, k, v, o, lse, d_o, ks)
    held = torch.zeros(H, W, dtype=torch.bool, device=DEV)
    y, x = na.get_window_start(2, H, ks), na.get_window_start(column, W, ks)
    held[y:y + ks, x:x + ks] = True
    assert torch.equal(~torch.isfinite(dv2[0, 0]).all(-1), held) and torch.equal(dv2[0, 0][~held], dv[0, 0][~held])
    assert torch.equal(dk2[0, 0][~held], dk[0, 0][~held])
