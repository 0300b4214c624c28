"""What a call through torch's dispatcher keeps, whichever host path the op takes: tracing, second derivatives, batched
gradients, tangents that are differentiated, saved-tensor hooks, tensor subclasses and function modes."""

import pytest
import torch
import torch.utils.checkpoint
from torch.overrides import TorchFunctionMode

from dmf_b200 import _native, adaln, flash_attn_func, flash_attn_qkvpacked_func
from dmf_b200.rms_norm import rms_norm

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _randn(*shape, dtype=torch.bfloat16, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + sum(shape))
    return torch.randn(*shape, device=DEV, dtype=dtype, generator=g)


def _case(op, seed=0):
    """(function, its tensor inputs)"""
    r = lambda *s, **k: _randn(*s, seed=seed + 1000 * len(made), **k)
    made = []

    def new(*s, **k):
        made.append(r(*s, **k))
        return made[-1]

    if op == "attn":
        return flash_attn_func, [new(2, 256, 3, 72), new(2, 256, 3, 72), new(2, 256, 3, 72)]
    if op == "packed":
        return flash_attn_qkvpacked_func, [new(2, 128, 3, 2, 64)]
    if op == "rms":
        return rms_norm, [new(2, 20, 3, 72), new(72, dtype=torch.float32)]
    if op == "ln":
        return adaln.ln_modulate, [new(2, 24, 384), new(2, 1, 384), new(2, 1, 384)]
    if op == "gate":
        return adaln.gate_residual, [new(2, 24, 384), new(2, 1, 384), new(2, 24, 384)]
    return adaln.gelu, [new(3, 50, 40)]


ALL = ("attn", "packed", "rms", "ln", "gate", "gelu")


@pytest.mark.parametrize("op", ALL)
def test_a_traced_call_replays_on_new_inputs(op):
    fn, args = _case(op)
    traced = torch.jit.trace(fn, tuple(args))
    new = _case(op, seed=7)[1]
    assert torch.equal(traced(*new), fn(*new))


@pytest.mark.parametrize("op", ("attn", "packed", "rms", "ln", "gate"))
def test_second_derivatives_are_refused(op):
    """Neither the kernels nor their host code compute them: a loss that asks for one must not get a number without it."""
    fn, args = _case(op)
    args = [a.requires_grad_(True) for a in args]
    out = fn(*args)
    first = torch.autograd.grad(out, args, torch.ones_like(out), create_graph=True)
    plain = torch.autograd.grad(fn(*args), args, torch.ones_like(out))
    assert all(torch.equal(a, b) for a, b in zip(first, plain, strict=True))
    which = {"gate": 2}.get(op, 0)                  # (the gradient of the gate's x is the incoming one: linear)
    loss = (first[which].float() * args[which].float()).sum()
    with pytest.raises(RuntimeError):
        torch.autograd.grad(loss, args, allow_unused=True)


def test_gelu_has_its_second_derivative():
    lib = lambda x: torch.nn.functional.gelu(x, approximate="tanh")
    x, dy, v = (_randn(3, 50, 40, seed=s) for s in (1, 2, 3))
    res = []
    for fn in (adaln.gelu, lib):
        a, g = x.clone().requires_grad_(True), dy.clone().requires_grad_(True)
        first, = torch.autograd.grad(fn(a), a, g, create_graph=True)
        res.append((first, *torch.autograd.grad(first, (a, g), v)))
    for a, b in zip(*res, strict=True):
        assert torch.equal(a, b)


def test_gelu_tangent_carries_its_gradient():
    """The library's GELU differentiates its tangent in reverse; so does this one."""
    lib = lambda x: torch.nn.functional.gelu(x, approximate="tanh")
    x, t, dy, dty = (_randn(3, 50, 40, seed=s) for s in (1, 2, 3, 4))
    res = []
    for fn in (adaln.gelu, lib):
        a, ta = x.clone().requires_grad_(True), t.clone().requires_grad_(True)
        y, ty = torch.func.jvp(fn, (a,), (ta,))
        res.append(torch.autograd.grad((y, ty), (a, ta), (dy, dty), retain_graph=True)
                   + torch.autograd.grad(ty, (a, ta), dty))
    for a, b in zip(*res, strict=True):
        # the primal's and the tangent's share of the gradient are added in 16 bits, in either order: half an ulp of each
        assert torch.allclose(a.float(), b.float(), rtol=2.0 ** -7, atol=2.0 ** -7)


@pytest.mark.parametrize("op", ("attn", "packed", "rms", "gelu"))
def test_batched_gradients(op):
    fn, args = _case(op)
    args = [a.requires_grad_(True) for a in args]
    out = fn(*args)
    douts = torch.stack([_randn(*out.shape, seed=s) for s in (1, 2, 3)])
    batched = torch.autograd.grad(out, args, douts, is_grads_batched=True, retain_graph=True)
    for i, dout in enumerate(douts):
        for a, b in zip(batched, torch.autograd.grad(out, args, dout, retain_graph=True), strict=True):
            assert torch.equal(a[i], b)


@pytest.mark.parametrize("op", ALL)
def test_gradients_of_the_tangent_alone(op):
    """Backward differentiates the primal output; the gradient that the tangent output brings is zero, for every input."""
    if op == "gelu":
        pytest.skip("differentiates its tangent")
    fn, args = _case(op)
    args = [a.requires_grad_(True) for a in args]
    if op == "rms":
        fn_, w = fn, args[1]
        _, tangent = torch.func.jvp(lambda x: fn_(x, w), (args[0],), (torch.ones_like(args[0]),))
    else:
        _, tangent = torch.func.jvp(fn, tuple(args), tuple(torch.ones_like(a) for a in args))
    for a, g in zip(args, torch.autograd.grad(tangent.float().sum(), args), strict=True):
        assert g.shape == a.shape and g.dtype == a.dtype and not g.any()


@pytest.mark.parametrize("op", ("attn", "packed", "rms", "ln", "gate"))
def test_a_tangent_that_requires_grad_keeps_the_graph(op):
    """Outputs of inputs without gradients belong to a graph when a tangent does, and its gradient is None."""
    fn, args = _case(op)
    tangents = [torch.ones_like(a).requires_grad_(True) for a in args]
    if op == "rms":
        fn_, w = fn, args[1]
        fn, args, tangents = (lambda x: fn_(x, w)), args[:1], tangents[:1]
    out, _ = torch.func.jvp(fn, tuple(args), tuple(tangents))
    assert out.requires_grad
    assert torch.autograd.grad(out.float().sum(), tangents, allow_unused=True) == (None,) * len(tangents)


@pytest.mark.parametrize("op", ALL)
def test_saved_tensors_in_another_layout(op):
    """A saved-tensor hook may hand back equal values with other strides."""
    fn, args = _case(op)
    args = [a.requires_grad_(True) for a in args]
    other = lambda t: t.transpose(0, -1).clone(memory_format=torch.contiguous_format).transpose(0, -1) if t.dim() > 1 else t.clone()
    dout = torch.ones_like(fn(*args))
    plain = torch.autograd.grad(fn(*args), args, dout)
    with torch.autograd.graph.saved_tensors_hooks(other, lambda t: t):
        out = fn(*args)
    for a, b in zip(torch.autograd.grad(out, args, dout), plain, strict=True):
        assert torch.equal(a, b)
    # ... but a tensor on another device is refused
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t):
        out = fn(*args)
    with pytest.raises((RuntimeError, ValueError)):
        torch.autograd.grad(out, args, dout)


class Named(torch.Tensor):
    """A subclass without a Python dispatch key: only __torch_function__ sees its calls."""


@pytest.mark.parametrize("op", ("attn", "packed", "rms", "gelu"))
def test_subclasses_and_function_modes_see_the_op(op):
    fn, args = _case(op)
    want = fn(*args)
    got = fn(args[0].as_subclass(Named), *args[1:])
    assert type(got) is Named and torch.equal(got.as_subclass(torch.Tensor), want)
    seen = []

    class Spy(TorchFunctionMode):
        def __torch_function__(self, func, types, a=(), kw=None):
            seen.append(str(func))
            return func(*a, **(kw or {}))

    with Spy():
        got = fn(*args)
    assert torch.equal(got, want)
    assert any(("gelu" if op == "gelu" else "dmf_b200") in s for s in seen), seen
    with torch.device(DEV):                         # a function mode as well, but not one that looks at ops
        assert _native.takes(*args) and not _native.takes(args[0].as_subclass(Named), *args[1:])
        assert _native.takes(torch.nn.Parameter(args[0]))


@pytest.mark.parametrize("op", ALL)
@pytest.mark.parametrize("reentrant", [True, False])
def test_checkpointed_calls(op, reentrant):
    """Recomputation in backward: without reentry it runs inside a saved-tensor hook, and needs autograd as usual there."""
    fn, args = _case(op)
    args = [a.requires_grad_(True) for a in args]
    body = lambda *a: fn(a[0] * 2, *a[1:]).sin()

    def gradients(out):
        for a in args:
            a.grad = None
        out.backward(torch.ones_like(out))
        return [a.grad for a in args]

    plain = gradients(body(*args))
    again = gradients(torch.utils.checkpoint.checkpoint(body, *args, use_reentrant=reentrant))
    for a, b in zip(plain, again, strict=True):
        assert torch.equal(a, b)
