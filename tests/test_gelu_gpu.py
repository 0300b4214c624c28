"""GELU (tanh form) with tangent and backward as one kernel against its formula in fp64."""

import math

import pytest
import torch

from dmf_b200 import _native, adaln, ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _oracle(x, t):
    """gelu(x) and gelu'(x) t in fp64."""
    x, t = x.double().cpu(), t.double().cpu()
    c = math.sqrt(2 / math.pi)
    s = torch.sigmoid(2 * c * (x + 0.044715 * x ** 3))
    return x * s, (s + x * s * (1 - s) * 2 * c * (1 + 3 * 0.044715 * x * x)) * t


def _close(a, ref, scale):
    # half a unit in the last place of the 16-bit result, and the fp32 arithmetic behind it: exponential and reciprocal
    # to about 1e-6 relative, times |x| or |t|; half the smallest step of a subnormal fp16
    half = 2.0 ** -8 if a.dtype == torch.bfloat16 else 2.0 ** -11
    bound = half * 1.01 * ref.abs() + 4e-6 * scale.double().cpu().abs() + 2.0 ** -25
    assert bool(((a.double().cpu() - ref).abs() <= bound).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1,), (7,), (8,), (8 * 1024 + 3,), (3, 257, 40), (2, 64, 1536)])
def test_value_tangent_and_gradient(dtype, shape):
    g = torch.Generator(device=DEV).manual_seed(sum(shape))
    x, t, dy = (torch.randn(shape, device=DEV, generator=g).mul(k).to(dtype) for k in (3.0, 1.0, 1.0))
    assert ops._CHECK_EVERY_CALL or _native.gelu(x) is not None     # the kernel takes it, not the general route
    y = adaln.gelu(x)
    xr = x.clone().requires_grad_(True)
    y2, ty = torch.func.jvp(adaln.gelu, (xr,), (t,))
    y2.backward(dy)
    ref, ref_t = _oracle(x, t)
    _close(y, ref, x)
    _close(ty, ref_t, t * (1 + x.abs()))
    _close(xr.grad, _oracle(x, dy)[1], dy * (1 + x.abs()))
    assert torch.equal(y, y2)


def test_limits_strides_and_other_types():
    x = torch.tensor([float("inf"), -float("inf"), float("nan"), 0.0, -0.0, 3e38, -3e38, -9.0, 1e-30], device=DEV).bfloat16()
    lib = torch.nn.functional.gelu(x, approximate="tanh")
    y = adaln.gelu(x)
    assert torch.equal(y.isnan(), lib.isnan()) and torch.equal(y.isinf(), lib.isinf())
    a = torch.randn(64, 48, device=DEV).bfloat16()
    assert torch.equal(adaln.gelu(a.t()), adaln.gelu(a).t())                       # not contiguous
    assert torch.equal(adaln.gelu(a.view(-1)[1:]), adaln.gelu(a).view(-1)[1:])     # base not on a 16-byte boundary
    f = torch.randn(33, device=DEV)
    assert torch.equal(adaln.gelu(f), torch.nn.functional.gelu(f, approximate="tanh"))
    assert adaln.gelu(a[:0]).shape == (0, 48)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_value_is_the_library_s_bit_for_bit(dtype):
    """All 65536 inputs: the value; and the tangent and the gradient for several factors each (NaN where the library's are)."""
    lib = lambda x: torch.nn.functional.gelu(x, approximate="tanh")
    same = lambda a, b: bool(((a == b) | (a.isnan() & b.isnan())).all())
    x = torch.arange(-32768, 32768, dtype=torch.int32, device=DEV).to(torch.int16).view(dtype)
    assert ops._CHECK_EVERY_CALL or _native.gelu(x) is not None
    assert same(adaln.gelu(x), lib(x))
    for seed in range(8):
        t = torch.randn(65536, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)).to(dtype)
        res = []
        for fn in (adaln.gelu, lib):
            xr = x.clone().requires_grad_(True)
            y, ty = torch.func.jvp(fn, (xr,), (t,))
            res.append((y, ty, *torch.autograd.grad(y, xr, t)))
        assert all(same(a, b) for a, b in zip(*res, strict=True))
    # finite where the function is: x^3 overflows above 7e12, and gelu' is 0 or 1 there
    big = torch.tensor([2e13, -2e13, 1e18, -1e18], device=DEV).bfloat16().requires_grad_(True)
    y, ty = torch.func.jvp(adaln.gelu, (big,), (torch.ones_like(big),))
    assert ty.tolist() == [1, 0, 1, 0] and torch.autograd.grad(y.sum(), big)[0].tolist() == [1, 0, 1, 0]
