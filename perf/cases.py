"""The work this package is measured by: neighborhood attention calls as a model makes them.

A case is one pass through the public entry points: a training step (forward and backward through
autograd), an inference forward, the 1D operator or the unfused pair.  Sizes are those of the
benchmark and the tests, ragged ones included; ``draw`` spreads further cases over the same ranges.
"""
import math

import torch

import e_natten_b200 as na

_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}

# What a drawn case may hold at most, for the 16-bit tensor-core shapes and for everything else: pixels
# and the multiply-adds of a step, no more than the largest listed cases of either kind.
_MAX_TENSOR = (1 << 23, 1.2e12)
_MAX_OTHER = (1 << 20, 1.2e10)
# Multiply-adds of one contraction above which ``exact`` gives no value (about 20 seconds).
_MAX_EXACT = 1 << 38


def _case(op, B, N, H, W, C, ks, dtype, packed=False, scaled=True):
    """op: "step" (forward and backward), "forward" (inference), "step_1d", "forward_1d" (H is 1) or
    "unfused" (scores, softmax, apply; forward and backward).  packed: q, k and v are views of one
    (B, H, W, 3, heads, C) projection.  scaled: C ** -0.5 goes in as the ``scale`` argument, else q
    carries it already."""
    return {"op": op, "B": B, "N": N, "H": H, "W": W, "C": C, "ks": ks, "dtype": dtype, "packed": packed,
            "scaled": scaled}


def listed():
    cases = {
        # smallest: unit-test sized call in the reference's data type; launches and host time count
        "tiny-fp32-step": _case("step", 1, 2, 16, 16, 32, 5, "fp32", scaled=False),
        # training step on a small feature map: a fraction of a wave of tiles
        "side32-bf16-step": _case("step", 4, 4, 32, 32, 128, 5, "bf16"),
        # the benchmark's headline: image-sized grid, training step
        "side256-bf16-step": _case("step", 4, 4, 256, 256, 128, 5, "bf16"),
        # first stage of a vision backbone, q / k / v sliced out of one projection as models do
        "stage1-bf16-step-packed": _case("step", 32, 2, 56, 56, 32, 7, "bf16", packed=True),
        # deep stages with a window about as large as the grid: clamping at every border
        "deep28-bf16-step": _case("step", 16, 8, 28, 28, 64, 13, "bf16"),
        "deep14-fp16-step": _case("step", 16, 16, 14, 14, 64, 13, "fp16"),
        # one very large image with the largest tensor-core window
        "side1024-bf16-step": _case("step", 1, 8, 1024, 1024, 128, 13, "bf16"),
        # inference on an image whose sides fit no tile
        "ragged-fp16-forward": _case("forward", 2, 6, 97, 131, 64, 9, "fp16", packed=True),
        # the reference's own benchmark, backward plot: fp32, image-sized grid
        "side256-fp32-step": _case("step", 4, 4, 256, 256, 128, 5, "fp32"),
        # fp32 inference, forward plot of the reference's benchmark with a mid-sized odd grid
        "ragged-fp32-forward": _case("forward", 4, 4, 117, 93, 64, 7, "fp32"),
        # sequence model: the 1D operator, training step
        "seq4096-bf16-step-1d": _case("step_1d", 4, 8, 1, 4096, 64, 13, "bf16"),
        # the two-step form (scores, softmax, apply) that the reference's benchmark compares with
        "side64-fp32-unfused": _case("unfused", 4, 4, 64, 64, 128, 5, "fp32", scaled=False),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _taps(case):
    return case["ks"] if case["op"].endswith("1d") else case["ks"] ** 2


def _pixels(case):
    return case["B"] * case["N"] * case["H"] * case["W"]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    while True:
        op = rng.choice(["step"] * 6 + ["forward"] * 3 + ["step_1d"] * 2 + ["forward_1d", "unfused"])
        one_d = op.endswith("1d")
        dtype = rng.choice(["fp32", "fp32", "bf16", "bf16", "fp16"])
        C = rng.choice([32, 32, 64, 64, 64, 128, 128, 128, 48, 96])
        ks = rng.choice([3, 5, 7, 9, 11, 13])
        B, N = _log_int(rng, 1, 32), _log_int(rng, 1, 16)
        if one_d:
            H, W = 1, _log_int(rng, 64, 65536)
        else:
            H = _log_int(rng, 14, 1024)
            W = max(14, min(1024, round(H * rng.uniform(0.6, 1.7))))
        case = _case(op, B, N, H, W, C, ks, dtype, packed=op in ("step", "forward") and rng.random() < 0.4,
                     scaled=op != "unfused" and rng.random() < 0.8)
        tensor = dtype != "fp32" and C in (32, 64, 128) and op in ("step", "forward")
        macs = 7 * _pixels(case) * _taps(case) * C
        max_pixels, max_macs = _MAX_TENSOR if tensor else _MAX_OTHER
        if macs <= max_macs and 1 << 9 <= _pixels(case) <= max_pixels:
            return case


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B, N, H, W, C = (case[n] for n in ("B", "N", "H", "W", "C"))
    train = not case["op"].startswith("forward")
    dtype = _DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)

    state = {"op": case["op"], "ks": case["ks"], "scale": C ** -0.5 if case["scaled"] else None}
    if case["packed"]:
        qkv = normal(B, H, W, 3, N, C)
        if not case["scaled"]:
            qkv[:, :, :, 0] *= C ** -0.5
        state["qkv"] = qkv.requires_grad_(train)
        if train:       # the gradient comes back from the output projection, heads last
            state["d_o"] = normal(B, H, W, N, C).permute(0, 3, 1, 2, 4)
    else:
        shape = (B, N, W, C) if case["op"].endswith("1d") else (B, N, H, W, C)
        q, k, v = normal(*shape), normal(*shape), normal(*shape)
        if not case["scaled"]:
            q *= C ** -0.5
        state["qkv"] = tuple(t.requires_grad_(train) for t in (q, k, v))
        if train:
            state["d_o"] = normal(*shape)
    return state


def _attend(state):
    qkv, ks, scale = state["qkv"], state["ks"], state["scale"]
    q, k, v = qkv.permute(3, 0, 4, 1, 2, 5).unbind(0) if isinstance(qkv, torch.Tensor) else qkv
    if state["op"] == "unfused":
        return na.natten2d_unfused(q, k, v, ks)
    if state["op"].endswith("1d"):
        return na.natten1d(q, k, v, ks, scale)
    return na.natten2d(q, k, v, ks, scale)


def run(state):
    if state["op"].startswith("forward"):
        with torch.no_grad():
            return {"o": _attend(state)}
    o = _attend(state)
    leaves = (state["qkv"],) if isinstance(state["qkv"], torch.Tensor) else state["qkv"]
    grads = torch.autograd.grad(o, leaves, state["d_o"])
    return {"o": o.detach(), **{f"grad{i}": g for i, g in enumerate(grads)}}


def work(case):
    """Each call's inputs read once and its outputs written once.  Forward: q, k, v in, o and one fp32
    statistic per row out.  Backward: q, k, v, o, d_o and the statistic in, three gradients out.  The
    unfused pair also writes and reads the (pixels, window) weights between its calls.  2 operations
    per multiply-add; the backward forms the scores again."""
    pix, taps, C = _pixels(case), _taps(case), case["C"]
    esize = 4 if case["dtype"] == "fp32" else 2
    t, a, stat = pix * C * esize, pix * taps * esize, 4 * pix
    mac = 2.0 * pix * taps * C
    if case["op"] == "unfused":
        return {"bytes": 11 * t + 10 * a, "flops": 6 * mac}
    if case["op"].startswith("forward"):
        return {"bytes": 4 * t + stat, "flops": 2 * mac}
    return {"bytes": 12 * t + 2 * stat, "flops": 7 * mac}


def _window_index(n, ks):
    """(n, ks) indices of each position's window on an axis of n, shifted inwards at the borders."""
    start = (torch.arange(n) - ks // 2).clamp(0, n - ks)
    return (start[:, None] + torch.arange(ks)).cuda()


def _exact_units(q, k, v, d_o, rows, cols, scale):
    """(o, dQ, dK, dV) in 64 bits for (units, H, W, C) operands; the gradients are None without d_o."""
    U, H, W, C = q.shape
    q, k, v = q.double(), k.double(), v.double()
    offsets = [(a, b) for a in range(rows.shape[1]) for b in range(cols.shape[1])]
    flat = [(rows[:, a, None] * W + cols[None, :, b]).flatten() for a, b in offsets]
    k_flat, v_flat = k.reshape(U, H * W, C), v.reshape(U, H * W, C)
    q_flat = q.reshape(U, H * W, C)
    scores = torch.stack([(q_flat * k_flat[:, i]).sum(-1) for i in flat], -1)
    p = torch.softmax(scores.mul_(scale), -1)
    o = torch.zeros_like(q_flat)
    for j, i in enumerate(flat):
        o += p[..., j, None] * v_flat[:, i]
    if d_o is None:
        return o.view(U, H, W, C), None, None, None
    g = d_o.double().reshape(U, H * W, C)
    ds = torch.stack([(g * v_flat[:, i]).sum(-1) for i in flat], -1)
    ds = p * (ds - (p * ds).sum(-1, keepdim=True)) * scale
    d_q, d_k, d_v = torch.zeros_like(o), torch.zeros_like(o), torch.zeros_like(o)
    for j, i in enumerate(flat):
        d_q += ds[..., j, None] * k_flat[:, i]
        d_k.index_add_(1, i, ds[..., j, None] * q_flat)
        d_v.index_add_(1, i, p[..., j, None] * g)
    return tuple(t.view(U, H, W, C) for t in (o, d_q, d_k, d_v))


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits by plain torch; the unfused pair and the fused
    operator have the same value.  None for the few cases that would take too long."""
    B, N, H, W, C, ks = (case[n] for n in ("B", "N", "H", "W", "C", "ks"))
    if _pixels(case) * _taps(case) * C > _MAX_EXACT:
        return None
    state = prepare(case, seed)
    qkv, d_o = state["qkv"], state.get("d_o")
    q, k, v = (qkv.permute(3, 0, 4, 1, 2, 5).unbind(0) if case["packed"] else qkv)
    out_shape = q.shape
    units = [None if t is None else t.detach().reshape(B * N, H, W, C) for t in (q, k, v, d_o)]
    rows = _window_index(H, 1 if case["op"].endswith("1d") else ks)
    cols = _window_index(W, ks)
    scale = C ** -0.5 if case["scaled"] else 1.0
    step = max(1, (1 << 26) // (H * W * C))
    parts = [_exact_units(*(None if t is None else t[u:u + step] for t in units), rows, cols, scale)
             for u in range(0, B * N, step)]
    o, *grads = (None if t[0] is None else torch.cat(t).view(out_shape) for t in zip(*parts))
    if d_o is None:
        return {"o": o}
    if case["packed"]:
        grads = [torch.stack(grads).permute(1, 3, 4, 0, 2, 5)]
    return {"o": o, **{f"grad{i}": g for i, g in enumerate(grads)}}


def tolerance(case):
    """About four times the error against the same arithmetic in 64 bits, over 50 cases of these ranges:
    fp32 2.8e-7 in the norm and 6.9e-6 for the worst element, bf16 2.4e-3 and 2.4e-2 (3.8e-3 and
    4.7e-2 where the weights between the calls are 16 bits wide), fp16 3.0e-4 and 3.7e-3."""
    rel, worst = {"fp32": (1.2e-6, 3e-5), "bf16": (1e-2, 1e-1), "fp16": (1.2e-3, 1.5e-2)}[case["dtype"]]
    if case["op"] == "unfused" and case["dtype"] != "fp32":
        rel, worst = 1.6 * rel, 2 * worst
    return {"rel": rel, "max": worst}
