"""The native host path against the general Python route it stands in front of: the same kernels on the same tensors, so
outputs, tangents and gradients agree bit for bit; and what it does not handle reaches the general route."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD

from dmf_b200 import _native, adaln, flash_attn_func, flash_attn_qkvpacked_func, ops
from dmf_b200.rms_norm import rms_norm

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAMES = ("attn_func", "attn_qkvpacked", "rms_norm", "ln_modulate", "gate_residual")


def _randn(*shape, dtype=torch.bfloat16):
    return torch.randn(*shape, device=DEV, dtype=dtype)


def _case(op):
    """(function of dual inputs, inputs, tangents, captured leaves)"""
    torch.manual_seed(3)
    if op == "attn":
        return flash_attn_func, [_randn(2, 256, 3, 72) for _ in range(3)], [_randn(2, 256, 3, 72) for _ in range(3)], []
    if op == "packed":
        return flash_attn_qkvpacked_func, [_randn(2, 256, 3, 3, 64)], [_randn(2, 256, 3, 3, 64)], []
    if op == "rms":
        w = (1 + 0.1 * torch.randn(72, device=DEV)).requires_grad_(True)
        return (lambda x: rms_norm(x, w)), [_randn(2, 100, 3, 3, 72)[:, :, 1]], [_randn(2, 100, 3, 72)], [w]
    x, mod = _randn(2, 70, 384, dtype=torch.float32), _randn(2, 1, 6 * 384)
    if op == "ln":
        fn = lambda x, m: adaln.ln_modulate(x, *m.chunk(6, dim=-1)[:2], out_dtype=torch.bfloat16)
        return fn, [x, mod], [torch.randn_like(x), torch.randn_like(mod)], []
    fn = lambda x, m, h: adaln.gate_residual(x, m.chunk(6, dim=-1)[2], h)
    return fn, [x, mod, _randn(2, 70, 384)], [torch.randn_like(x), torch.randn_like(mod), _randn(2, 70, 384)], []


def _passes(op):
    fn, args, tangents, leaves = _case(op)
    args = [a.detach().requires_grad_(True) for a in args]
    out, tangent = torch.func.jvp(fn, tuple(args), tuple(tangents))
    dout = torch.ones_like(out)
    res = [out, tangent, *torch.autograd.grad(out, args + leaves, dout)]
    out = fn(*args)
    res += [out, *torch.autograd.grad(out, args + leaves, dout)]
    with torch.no_grad():
        res.append(fn(*args))
    with fwAD.dual_level():                       # a tangent on the first input only, no functorch level
        dual = fwAD.unpack_dual(fn(fwAD.make_dual(args[0].detach(), tangents[0]), *[a.detach() for a in args[1:]]))
    return res + [dual.primal, dual.tangent]


@pytest.mark.parametrize("op", ["attn", "packed", "rms", "ln", "gate"])
def test_native_path_is_the_general_route(op, monkeypatch):
    ops.check_device_status(DEV)      # the status word exists (a process's first attention call creates it on the general route)
    handled = []
    for name in NAMES:
        native = getattr(_native, name)
        monkeypatch.setattr(_native, name, lambda *a, native=native: handled.append(native(*a)) or handled[-1])
    fast = _passes(op)
    assert handled and all(h is not None for h in handled)
    for name in NAMES:
        monkeypatch.setattr(_native, name, lambda *a: None)
    for a, b in zip(fast, _passes(op), strict=True):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


def test_what_the_native_path_leaves_to_the_general_route():
    q = _randn(1, 128, 1, 64)
    assert _native.attn_func(q.float(), q.float(), q.float(), None) is None
    with pytest.raises(TypeError):
        flash_attn_func(q.float(), q.float(), q.float())
    with pytest.raises(RuntimeError):
        flash_attn_func(q[:, :100], q[:, :100], q[:, :100])       # not a multiple of 128 tokens
    seen = []
    nested = lambda a: torch.func.jvp(lambda b: seen.append(_native.attn_func(b, b, b, None)) or b, (a,), (a,))[0]
    torch.func.jvp(nested, (q,), (q,))
    assert seen == [None]                                          # two levels
    out = flash_attn_func(q, q, q, 0.3)
    assert torch.equal(out, torch.ops.dmf_b200.attn_fwd(q, q, q, 0.3)[0])
