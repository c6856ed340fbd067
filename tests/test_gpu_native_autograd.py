"""GPU tests of the native autograd functions against the Python ones: what callers can see of either is the same."""
import pytest
import torch

import e_natten_b200 as na

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FORMS = [((2, 3, 17, 19, 32), 5, lambda *a: na.natten2d(*a), lambda *a: na.Natten2d.apply(*a)[0]),
         ((2, 3, 40, 32), 7, lambda *a: na.natten1d(*a), lambda *a: na.Natten1d.apply(*a))]
form = pytest.mark.parametrize("shape,ks,native,python", FORMS, ids=["2d", "1d"])


def inputs(shape, dtype=torch.float32, grads=(True, True, True)):
    gen = torch.Generator(device=DEV).manual_seed(1)
    q, k, v, d_o = (torch.randn(shape, generator=gen, device=DEV).to(dtype) for _ in range(4))
    return [t.requires_grad_(g) for t, g in zip((q, k, v), grads)], d_o


def run(f, qkv, d_o, ks, scale):
    o = f(*qkv, ks, scale)
    leaves = [t for t in qkv if t.requires_grad]
    return (o, *(torch.autograd.grad(o, leaves, d_o) if leaves else ()))


@form
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("grads", [(1, 1, 1), (1, 0, 0), (0, 0, 1), (0, 0, 0)])
def test_same_bits(shape, ks, native, python, dtype, grads):
    qkv, d_o = inputs(shape, dtype, [bool(g) for g in grads])
    got, want = run(native, qkv, d_o, ks, 0.25), run(python, qkv, d_o, ks, 0.25)
    assert (got[0].grad_fn is None) == (not any(grads)) and len(got) == len(want)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@form
def test_saved_tensor_hooks(shape, ks, native, python):
    qkv, d_o = inputs(shape)
    seen = []
    for f in (native, python):
        packed = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.to(DEV)):
            o = f(*qkv, ks, None)
        seen.append(([tuple(t.shape) for t in packed], torch.autograd.grad(o, qkv, d_o)))
    assert seen[0][0] == seen[1][0] and all(torch.equal(a, b) for a, b in zip(seen[0][1], seen[1][1]))


@form
@pytest.mark.parametrize("change,which", [("half", "all"), ("half", "stat"), ("row", "all"), ("row", "stat"), ("cpu", "all"), ("cpu", "stat")])
def test_saved_tensors_of_another_form_are_refused(shape, ks, native, python, change, which):
    """Hooks that hand back another type, size or device than was saved: an error in either, and no kernel reads them."""
    unpack = {"half": lambda t: t.half(), "row": lambda t: t[:1], "cpu": lambda t: t.cpu()}[change]
    qkv, d_o = inputs(shape)
    raised = []
    for f in (native, python):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: unpack(t) if which == "all" or t.dim() < len(shape) else t):
            o = f(*qkv, ks, None)
            with pytest.raises(ValueError) as e:
                torch.autograd.grad(o, qkv, d_o)
        raised.append(str(e.value).splitlines()[0])
    assert raised[0] == raised[1] or change == "cpu"      # (there the Python function fails at its poll, one step earlier)


@form
def test_a_batch_of_gradients_is_refused(shape, ks, native, python):
    qkv, d_o = inputs(shape)
    raised = []
    for f in (native, python):
        o = f(*qkv, ks, None)
        with pytest.raises(RuntimeError) as e:
            torch.autograd.grad(o, qkv, torch.stack([d_o, d_o]), is_grads_batched=True)
        raised.append(type(e.value))
    assert raised[0] is raised[1]


@form
def test_graph_node(shape, ks, native, python):
    qkv, d_o = inputs(shape)
    outputs = [f(*qkv, ks, 0.5) for f in (native, python)]
    a, b = (o.grad_fn for o in outputs)
    for node in (a, b):
        assert node.name() == type(node).__name__ == f"Natten{len(shape) - 3}dBackward"
        assert node.kernel_size == ks and node.scale == 0.5 and len(node.next_functions) == 3
    assert len(a.saved_tensors) == len(b.saved_tensors) == 5
    assert all(torch.equal(x, y) for x, y in zip(a.saved_tensors, b.saved_tensors))
    o = native(*qkv, ks, None)
    torch.autograd.grad(o, qkv, d_o)
    with pytest.raises(RuntimeError, match="freed"):
        o.grad_fn.saved_tensors


@form
def test_graph_rules(shape, ks, native, python):
    """A freed graph, an input changed in place and a second derivative are refused; no gradient counts as zeros."""
    for f in (native, python):
        qkv, d_o = inputs(shape)
        o = f(*qkv, ks, None)
        torch.autograd.grad(o, qkv, d_o)
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(o, qkv, d_o)
        w = [t * 1 for t in qkv]
        o = f(*w, ks, None)
        w[1].add_(1)
        with pytest.raises(RuntimeError, match="inplace operation"):
            o.sum().backward()
        o = f(*qkv, ks, None)
        (g,) = torch.autograd.grad(o, qkv[:1], d_o, create_graph=True)
        assert not g.requires_grad


@form
def test_calls_that_are_looked_into(shape, ks, native, python):
    """Functional transforms and forward-mode gradients are refused by the Python functions, and so by the operator;
    modes and subclasses see the same call."""
    qkv, d_o = inputs(shape)

    def outcome(f):
        try:
            return f()
        except Exception as e:
            return type(e)

    plain = [t.detach() for t in qkv]
    for f in (lambda g: torch.func.grad(lambda q: g(q, *plain[1:], ks, None).sum())(plain[0]),
              lambda g: torch.vmap(lambda q: g(q, *plain[1:], ks, None))(plain[0][None])):
        assert outcome(lambda: f(native)) == outcome(lambda: f(python))

    def dual(g):
        with torch.autograd.forward_ad.dual_level():
            return g(torch.autograd.forward_ad.make_dual(plain[0], d_o), *plain[1:], ks, None)
    assert outcome(lambda: dual(native)) == outcome(lambda: dual(python))

    class Mode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with Mode():
        assert torch.equal(native(*plain, ks, None), python(*plain, ks, None))

    class Sub(torch.Tensor):
        pass
    sub = [t.as_subclass(Sub) for t in plain]
    assert type(native(*sub, ks, None)) is type(python(*sub, ks, None))


@form
def test_arguments_keep_their_errors(shape, ks, native, python):
    qkv, _ = inputs(shape)
    for args in ((qkv[0], qkv[1], qkv[2], 4, None), (qkv[0], qkv[1][:1], qkv[2], ks, None), (qkv[0], qkv[1].half(), qkv[2], ks, None),
                 (qkv[0], qkv[1], qkv[2], 43, None), (qkv[0].cpu(), qkv[1], qkv[2], ks, None), (qkv[0], qkv[1], None, ks, None),
                 (*qkv, ks, -1.0), (*qkv, ks, "x")):
        raised = []
        for f in (native, python):
            with pytest.raises(Exception) as e:
                f(*args)
            raised.append((type(e.value), str(e.value)))
        assert raised[0] == raised[1]
