"""The plain forward with two query tiles per CTA where it can go wrong: an odd tile count (the last unit of a head has one
tile), one key block, single-tile units (a GPU that is not filled), several units per CTA, maxima that move late, every
head-dim class; against the fp64 oracle, with the bf16 / fp16 rounding of P and of the result as the tolerance."""

import pytest
import torch

from dmf_b200 import _lib
from oracle import attn_jvp_oracle as orc
from tests import _cabi

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("shape", [(1, 256, 128, 1, 64), (16, 384, 256, 4, 72), (25, 384, 128, 8, 72), (16, 640, 640, 8, 64),
                                   (3, 256, 1152, 5, 80), (32, 640, 384, 4, 96), (20, 1024, 128, 5, 128), (8, 2048, 512, 6, 104)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_plain_forward_two_tiles_per_cta(shape, dtype):
    B, Lq, Lk, H, D = shape
    assert "duo" in _lib.kernel_name("fwd", Lq, Lk, D) and "duo" in _lib.kernel_name("fwd", Lq, Lk, D, batch=B, heads=H)
    q = orc.make_inputs(B, Lq, H, D, seed=Lq + D)[0].to(dtype)
    k, v = (x.to(dtype) for x in orc.make_inputs(B, Lk, H, D, seed=Lk + H)[1:3])
    k = k * torch.linspace(0.5, 3.0, Lk).view(1, Lk, 1, 1).to(dtype)      # later blocks hold the larger logits
    o, _, lse, _ = _cabi.fwd(*(x.to(DEV) for x in (q, k, v)))
    assert not torch.isnan(o).any() and not torch.isnan(lse).any()
    for b in {0, B // 2, B - 1}:
        o_ref, lse_ref = orc.attn_fwd_closed_form(*[x[b:b + 1].float() for x in (q, k, v)])
        # P and o are rounded to 8 (11) bits: 2^-9 (2^-12) relative each, independent over the keys
        assert orc.rel_l2(o[b:b + 1].float().cpu(), o_ref) < (6e-3 if dtype == torch.bfloat16 else 1e-3)
        # a quarter of the exponentials are cubics with 7.5e-5 relative error
        assert float((lse[b:b + 1].cpu().double() - lse_ref).abs().max()) < 1e-4


@pytest.mark.parametrize("shape", [(2, 384, 256, 3, 72), (30, 384, 384, 4, 96), (12, 640, 640, 7, 64), (40, 384, 128, 8, 72), (24, 384, 256, 5, 128),
                                   (1, 2048, 2048, 2, 104)])
def test_plain_forward_one_tile_per_cta_where_that_takes_fewer_rounds(shape):
    """Odd tile counts and head_dim above 96 with few heads: the other kernel, to the same tolerances."""
    B, Lq, Lk, H, D = shape
    assert "duo" not in _lib.kernel_name("fwd", Lq, Lk, D, batch=B, heads=H)
    q = orc.make_inputs(B, Lq, H, D, seed=Lq + D)[0].bfloat16()
    k, v = (x.bfloat16() for x in orc.make_inputs(B, Lk, H, D, seed=Lk + H)[1:3])
    o, _, lse, _ = _cabi.fwd(*(x.to(DEV) for x in (q, k, v)))
    for b in {0, B - 1}:
        o_ref, lse_ref = orc.attn_fwd_closed_form(*[x[b:b + 1].float() for x in (q, k, v)])
        assert orc.rel_l2(o[b:b + 1].float().cpu(), o_ref) < 6e-3
        assert float((lse[b:b + 1].cpu().double() - lse_ref).abs().max()) < 1e-4


@pytest.mark.parametrize("shape", [(16, 384, 256, 4, 72), (16, 640, 384, 8, 64), (32, 640, 384, 4, 96), (20, 1024, 256, 5, 128),
                                   (12, 1152, 1152, 12, 128), (64, 512, 512, 4, 72)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_plain_forward_bits_do_not_depend_on_the_batch(shape, dtype):
    """One element alone takes one tile per CTA, the batch two: the same o and lse bit for bit, late maxima included."""
    B, Lq, Lk, H, D = shape
    q = orc.make_inputs(B, Lq, H, D, seed=Lq + D)[0].to(dtype)
    k, v = (x.to(dtype) for x in orc.make_inputs(B, Lk, H, D, seed=Lk + H)[1:3])
    k = k * torch.linspace(0.5, 6.0, Lk).view(1, Lk, 1, 1).to(dtype)
    q, k, v = (x.to(DEV) for x in (q, k, v))
    o, _, lse, _ = _cabi.fwd(q, k, v)
    for b in {0, B // 2, B - 1}:
        o1, _, lse1, _ = _cabi.fwd(*(x[b:b + 1].contiguous() for x in (q, k, v)))
        assert torch.equal(o[b:b + 1], o1) and torch.equal(lse[b:b + 1], lse1)
