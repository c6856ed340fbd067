"""CPU tests of the autograd functions, the kernels replaced by the oracle."""
import pytest
import torch

import e_natten_b200 as na
from e_natten_b200 import functional as F
from oracle import na2d_oracle as orc


@pytest.fixture
def on_oracle(monkeypatch):
    def forward(q, k, v, ks, scale=1.0, **_):
        return tuple(t.to(q.dtype) for t in orc.natten2d_fwd(q, k, v, ks, scale=scale))

    def backward(q, k, v, o, lse, d_o, ks, scale=1.0, **_):
        return tuple(t.to(q.dtype) for t in orc.natten2d_bwd(q, k, v, d_o, ks, scale=scale))

    monkeypatch.setattr(F, "natten2d_forward", forward)
    monkeypatch.setattr(F, "natten2d_backward", backward)
    monkeypatch.setattr(F, "poll_kernels", lambda device: None)


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, grad):
        return None


def test_undefined_gradient_counts_as_zeros(on_oracle):
    q, k, v = (torch.randn(1, 1, 6, 7, 4, requires_grad=True) for _ in range(3))
    o = na.natten2d(q, k, v, 3)
    grads = torch.autograd.grad(_NoGradient.apply(o).sum(), (q, k, v), retain_graph=True)
    assert all(g.shape == q.shape and not g.any() for g in grads)
    assert all(g.any() for g in torch.autograd.grad(o, (q, k, v), torch.ones_like(o)))


def test_gradient_with_lse_in_the_graph(on_oracle):
    q, k, v = (torch.randn(1, 1, 6, 7, 4, requires_grad=True) for _ in range(3))
    o, lse = na.natten2d_with_lse(q, k, v, 3)
    assert o.requires_grad and not lse.requires_grad
    got = torch.autograd.grad((o * lse.unsqueeze(-1)).sum(), (q, k, v))
    want = orc.natten2d_bwd(*(t.detach() for t in (q, k, v)), lse.unsqueeze(-1).expand_as(o), 3)
    assert all(torch.allclose(g, w.float(), atol=1e-5) for g, w in zip(got, want))
