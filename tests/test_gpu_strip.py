"""GPU tests of the tensor-core kernels of the larger windows: column strips, two query tiles in flight."""
import pytest
import torch

import e_natten_b200 as na
from oracle import na2d_oracle as orc
from helpers import assert_close, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def step(q, k, v, d_o, ks):
    qd, kd, vd, gd = (t.to(DEV) for t in (q, k, v, d_o))
    o, lse = na.natten2d_forward(qd, kd, vd, ks)
    grads = na.natten2d_backward(qd, kd, vd, o, lse, gd, ks)
    na.check_kernels(DEV)
    return (o, lse, *grads)


# Units of 2 x 2 and 2 x 3 tiles, enough of them for two tiles on some CTAs and one on others (the forward takes pairs of tiles from
# 149 tiles on); the second tile row and the last column hold one to nine pixels, every border clamps.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("ks,H,W", [(7, 17, 17), (9, 21, 16), (11, 25, 23), (13, 17, 13)])
def test_odd_and_even_tiles_of_a_cta(ks, H, W, D, dtype):
    shape = (2, 20, H, W, D)
    q, k, v, d_o = make_inputs(shape, dtype, ks, q_scale=D ** -0.5)
    got = step(q, k, v, d_o, ks)
    want = orc.natten2d_fwd_bwd(q, k, v, d_o, ks)
    for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), got, want):
        assert_close(g, w, dtype, f"{name} {shape} ks={ks}")


# Three tile rows, the middle one away from both borders, at the sizes on either side of where the forward changes kernels.
@pytest.mark.parametrize("units", [1, 13])
@pytest.mark.parametrize("ks,D", [(7, 32), (9, 64), (13, 128)])
def test_inner_and_border_tiles(ks, D, units):
    shape = (1, units, 48, 30, D)
    q, k, v, d_o = make_inputs(shape, torch.bfloat16, 5, q_scale=D ** -0.5)
    got = step(q, k, v, d_o, ks)
    want = orc.natten2d_fwd_bwd(q, k, v, d_o, ks)
    for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), got, want):
        assert_close(g, w, torch.bfloat16, f"{name} {shape} ks={ks}")


# The key half's two forms of chunks, at images on either side of where they change places (in either direction), and images whose
# last key tile is seen from more rows than a strip is tall.
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("ks,H,W", [(7, 18, 40), (7, 22, 40), (7, 100, 14), (7, 70, 40), (9, 14, 50), (9, 30, 32), (9, 72, 40), (11, 22, 40),
                                    (11, 40, 40), (11, 74, 40), (13, 20, 21), (13, 30, 32), (13, 76, 40)])
def test_both_forms_of_query_chunks(ks, H, W, D):
    shape = (1, 2, H, W, D)
    q, k, v, d_o = make_inputs(shape, torch.bfloat16, ks, q_scale=D ** -0.5)
    got = step(q, k, v, d_o, ks)
    want = orc.natten2d_fwd_bwd(q, k, v, d_o, ks)
    for name, g, w in zip(("o", "lse", "dq", "dk", "dv"), got, want):
        assert_close(g, w, torch.bfloat16, f"{name} {shape} ks={ks}")


@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("ks,D,at", [(7, 32, (8, 9)), (13, 128, (0, 15)), (9, 64, (16, 7))])
def test_a_key_reaches_only_the_windows_that_hold_it(ks, D, at, bad):
    """Two tiles in flight, forward: scores outside a window are left out whatever they hold."""
    q, k, v, _ = (t.to(DEV) for t in make_inputs((1, 80, 17, 17, D), torch.bfloat16, 3, q_scale=D ** -0.5))
    clean, clean_lse = na.natten2d_forward(q, k, v, ks)
    k[:, :, at[0], at[1], D // 2] = bad
    o, lse = na.natten2d_forward(q, k, v, ks)
    na.check_kernels(DEV)
    ws = [orc.window_start(i, 17, ks) for i in range(17)]
    held = torch.tensor([[a <= at[0] < a + ks and b <= at[1] < b + ks for b in ws] for a in ws], device=DEV)
    assert torch.equal(o[:, :, ~held], clean[:, :, ~held]) and torch.equal(lse[:, :, ~held], clean_lse[:, :, ~held])
    if bad != bad:
        assert o[:, :, held].isnan().all()


@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("ks,D,at", [(7, 32, (8, 9)), (9, 64, (16, 20)), (13, 64, (20, 15)), (13, 128, (31, 0))])
def test_a_pixel_reaches_only_the_gradients_of_its_windows(ks, D, at, bad):
    """Backward on strips: a value of one pixel meets the queries whose window holds it, a query or its gradient the keys of its
    window, whatever it is.  (The operand that the other gradients multiply with stays finite here: their weights are zero.)"""
    H = W = 48
    q, k, v, d_o = (t.to(DEV) for t in make_inputs((1, 2, H, W, D), torch.bfloat16, 3, q_scale=D ** -0.5))
    o, lse = na.natten2d_forward(q, k, v, ks)
    ws = [orc.window_start(i, H, ks) for i in range(H)]
    holds = torch.tensor([[a <= at[0] < a + ks and b <= at[1] < b + ks for b in ws] for a in ws], device=DEV)       # queries
    held = torch.zeros(H, W, dtype=torch.bool, device=DEV)                                                          # keys
    held[ws[at[0]]:ws[at[0]] + ks, ws[at[1]]:ws[at[1]] + ks] = True

    def backward(q, v, d_o, delta=None):
        d_q, d_k, d_v, dl = torch.empty_like(q), torch.empty_like(k), torch.empty_like(k), torch.empty_like(lse)
        na.functional.backward_dq_into(q, k, v, o, lse, d_o, d_q, dl, ks)
        na.functional.backward_dkdv_into(q, k, v, lse, d_o, dl if delta is None else delta, d_k, d_v, ks)
        na.check_kernels(DEV)
        return d_q, d_k, d_v, dl

    def changed(t):
        t = t.clone()
        t[:, :, at[0], at[1], D // 2] = bad
        return t
    d_q, d_k, d_v, delta = backward(q, v, d_o)
    got = backward(q, changed(v), d_o, delta)
    assert torch.equal(got[0][:, :, ~holds], d_q[:, :, ~holds]) and torch.equal(got[3][:, :, ~holds], delta[:, :, ~holds])
    got = backward(changed(q), v, d_o, delta)
    assert torch.equal(got[2][:, :, ~held], d_v[:, :, ~held])
    got = backward(q, v, changed(d_o), delta)
    assert torch.equal(got[1][:, :, ~held], d_k[:, :, ~held])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("ks,D", [(7, 32), (9, 64), (13, 64), (13, 128)])
def test_a_gradient_reaches_only_the_key_tiles_whose_box_holds_it(ks, D, bad):
    """Key half on strips, key tiles of 8 columns: a column of d_o beside a tile's box of queries meets none of its keys."""
    q, k, v, d_o = (t.to(DEV) for t in make_inputs((1, 2, 64, 64, D), torch.bfloat16, 3, q_scale=D ** -0.5))
    o, lse = na.natten2d_forward(q, k, v, ks)
    delta, out = torch.empty_like(lse), [torch.empty_like(k) for _ in range(5)]
    na.functional.backward_dq_into(q, k, v, o, lse, d_o, out[0], delta, ks)
    na.functional.backward_dkdv_into(q, k, v, lse, d_o, delta, out[1], out[2], ks)
    for tile in range(8):
        last = 8 * tile + 7
        for beside in (8 * tile - ks // 2 - 1 if 8 * tile >= ks else -1, last + ks // 2 + 1 if last < 64 - ks else -1):
            if beside < 0:
                continue
            g = d_o.clone()
            g[:, :, :, beside] = bad
            na.functional.backward_dkdv_into(q, k, v, lse, g, delta, out[3], out[4], ks)
            for a, b in ((out[1], out[3]), (out[2], out[4])):
                assert torch.equal(a[:, :, :, 8 * tile:last + 1], b[:, :, :, 8 * tile:last + 1]), (tile, beside)
    na.check_kernels(DEV)
