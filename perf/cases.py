"""The work that users of this framework have it do, as cases that can be timed.

Five families, each through the entry points that a program calls:

* ``attn``    - ``flash_attn_func`` / ``flash_attn_qkvpacked_func``: a forward without gradients (a sampler's step), the
  forward + tangent under ``torch.func.jvp``, and either of them followed by the backward of its primal output (the
  flow-matching and the MeanFlow term of the training loss);
* ``qk_norm`` - ``rms_norm`` of the q and k slices of a packed projection, the op in front of the attention;
* ``adaln``   - ``ln_modulate`` and ``gate_residual``, the elementwise half of a transformer block;
* ``tail``    - ``FlatAdamW.step_tail``, the end of an optimisation step over flat buffers;
* ``sample`` / ``train`` - the whole model: the few-step Euler sampler and the optimisation step.

Sizes are those of the four model configurations (hidden 384 / 768 / 1024 / 1152, 6 / 12 / 16 heads, 12 to 28 blocks), of
the 256- and 512-pixel settings (256 and 1024 tokens) and of the head dimensions and token counts the tests cover.
"""

from __future__ import annotations

import torch

from dmf_b200 import adaln, flash_attn_func, flash_attn_qkvpacked_func
from dmf_b200.harness import train as training
from dmf_b200.harness.model import DMFT_CONFIGS, build_dmft
from dmf_b200.harness.sampler import GraphedSampler, euler_sampler
from dmf_b200.rms_norm import rms_norm
from dmf_b200.step import FlatAdamW

DEV = "cuda:0"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
PARAMS = {"DMFT-S/2": 33_000_000, "DMFT-B/2": 130_000_000, "DMFT-L/2": 458_000_000, "DMFT-XL/2": 675_000_000}
STEPS = 4          # Euler steps of the sampler, as the 512-pixel setting uses


def listed():
    return [
        # one small image (12-block model, 256 pixels) goes through one attention layer of the sampler
        _attn("sample_attn_1_image", "fwd", 1, 256, 6, 64, packed=True),
        # the small standalone op: forward + tangent at 8 x 256 tokens, 12 heads
        _attn("jvp_attn_small", "jvp", 8, 256, 12, 64, packed=False),
        # forward + tangent at the 256-pixel shapes, read from the packed projection (no qk-norm there)
        _attn("jvp_attn_256px", "jvp", 256, 256, 16, 72, packed=True),
        # forward + tangent at the 512-pixel shapes, q and k normalised per head, v a slice of the projection
        _attn("jvp_attn_512px", "jvp", 64, 1024, 16, 72, packed=False),
        # MeanFlow term of a training micro-batch at 256 pixels: forward + tangent, then the backward
        _attn("train_jvp_attn_256px", "jvp_train", 128, 256, 16, 72, packed=True),
        # flow-matching term of a training micro-batch at 512 pixels: forward, then the backward
        _attn("train_attn_512px", "train", 32, 1024, 16, 72, packed=False),
        # an odd number of row tiles, fp16, the widest head: fine-tuning at another resolution
        _attn("train_attn_odd_fp16_d128", "train", 6, 1152, 12, 128, packed=True, dtype="fp16"),
        # per-head norm of q and k with tangents and its backward, a training micro-batch at 512 pixels
        {"name": "qk_norm_512px", "kind": "qk_norm", "mode": "jvp_train", "B": 32, "L": 1024, "H": 16, "D": 72},
        # a block's adaLN ops with tangents and their backward, fp32 residual stream under bf16 autocast
        {"name": "adaln_train_256px", "kind": "adaln", "mode": "jvp_train", "B": 32, "L": 256, "C": 1152},
        # clip + AdamW + EMA of the 130M-parameter model
        {"name": "step_tail_130m", "kind": "tail", "count": 130_000_000},
        # 512-pixel sampling of 8 images with the largest model, the loop kept as a CUDA graph as a server would
        {"name": "sample_xl_512px", "kind": "sample", "model": "DMFT-XL/2", "B": 8, "px": 512, "graphs": True},
        # one optimisation step of the largest model on the share one of 8 GPUs gets of a global batch of 256
        {"name": "train_xl_256px", "kind": "train", "model": "DMFT-XL/2", "B": 32, "px": 256},
    ]


def _attn(name, mode, B, L, H, D, *, packed, dtype="bf16"):
    return {"name": name, "kind": "attn", "mode": mode, "B": B, "L": L, "H": H, "D": D, "packed": packed, "dtype": dtype}


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choices(("attn", "qk_norm", "adaln", "tail", "sample", "train"), (8, 2, 2, 1, 2, 1))[0]
    if kind == "attn":
        mode = rng.choice(("fwd", "jvp", "train", "jvp_train"))
        L = 128 * _spread(rng, 1, 32)                       # 128 to 4096 tokens, odd tile counts among them
        H, D = rng.choice(((6, 64), (12, 64), (16, 64), (16, 72), (16, 72), (16, 72), (12, 80), (8, 96), (12, 128)))
        most = max(1, int(64 * 1024 ** 2 * 16 * 72 / (L * L * H * D)))
        most = min(most, int(256 * 256 * 16 * 72 / (L * H * D)) or 1, 256)
        c = _attn("", mode, _spread(rng, 1, most), L, H, D, packed=rng.random() < 0.5,
                  dtype="fp16" if rng.random() < 0.15 else "bf16")
        del c["name"]
        return c
    if kind == "qk_norm":
        L = 128 * _spread(rng, 1, 32)
        H, D = rng.choice(((6, 64), (12, 64), (16, 64), (16, 72), (16, 72), (12, 128)))
        return {"kind": kind, "mode": rng.choice(("fwd", "jvp_train")), "B": _spread(rng, 1, 65536 // L), "L": L, "H": H, "D": D}
    if kind == "adaln":
        L = 128 * _spread(rng, 1, 32)
        return {"kind": kind, "mode": rng.choice(("fwd", "jvp_train")), "B": _spread(rng, 1, 65536 // L), "L": L,
                "C": rng.choice((384, 768, 1024, 1152))}
    if kind == "tail":
        return {"kind": kind, "count": _spread(rng, 1_000_000, 300_000_000)}
    model, px = rng.choice(sorted(DMFT_CONFIGS)), rng.choice((256, 512))
    if kind == "sample":
        return {"kind": kind, "model": model, "B": _spread(rng, 1, 32 if px == 256 else 8), "px": px, "graphs": rng.random() < 0.6}
    return {"kind": kind, "model": model, "B": _spread(rng, 2, 32 if px == 256 else 8), "px": px}


# ---- what a program has in hand before the call ---------------------------------------------------------------------

def _randn(gen, *shape, dtype=torch.bfloat16, std=1.0):
    x = torch.randn(*shape, device=DEV, dtype=dtype, generator=gen)
    return x if std == 1.0 else x.mul_(std)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return {"attn": _prepare_attn, "qk_norm": _prepare_qk_norm, "adaln": _prepare_adaln, "tail": _prepare_tail,
            "sample": _prepare_sample, "train": _prepare_train}[case["kind"]](case, gen, seed)


def _prepare_attn(case, gen, seed):
    B, L, H, D, dt = case["B"], case["L"], case["H"], case["D"], DTYPES[case["dtype"]]
    dual, grad = case["mode"].startswith("jvp"), case["mode"].endswith("train")

    def inputs(std):
        qkv = _randn(gen, B, L, 3, H, D, dtype=dt, std=std)
        if case["packed"]:
            return (qkv,)
        # behind a qk-norm q and k are tensors of their own and v is still a slice of the projection
        unit = (lambda x: (x.float() * torch.rsqrt(x.float().square().mean(-1, keepdim=True) + 1e-6)).to(dt)) if std == 1.0 \
            else (lambda x: x.contiguous())
        return unit(qkv[:, :, 0]), unit(qkv[:, :, 1]), qkv[:, :, 2]

    args = inputs(1.0)
    if grad:
        args = tuple(x.requires_grad_(True) if x.is_leaf else x.detach().requires_grad_(True) for x in args)
    return {"kind": "attn", "args": args, "tangents": inputs(0.1) if dual else None, "grad": grad,
            "fn": flash_attn_qkvpacked_func if case["packed"] else flash_attn_func,
            "dout": _randn(gen, B, L, H, D, dtype=dt) if grad else None}


def _prepare_qk_norm(case, gen, seed):
    B, L, H, D = case["B"], case["L"], case["H"], case["D"]
    train = case["mode"] == "jvp_train"
    qkv, tqkv = _randn(gen, B, L, 3, H, D), _randn(gen, B, L, 3, H, D, std=0.1)
    w = [1.0 + _randn(gen, D, dtype=torch.float32, std=0.1) for _ in range(2)]
    if not train:
        return {"kind": "qk_norm", "args": (qkv[:, :, 0], qkv[:, :, 1], *(x.bfloat16() for x in w)), "tangents": None}
    args = tuple(x.detach().requires_grad_(True) for x in (qkv[:, :, 0], qkv[:, :, 1], *w))
    return {"kind": "qk_norm", "args": args, "tangents": (tqkv[:, :, 0], tqkv[:, :, 1]),
            "dout": (_randn(gen, B, L, H, D), _randn(gen, B, L, H, D))}


def _prepare_adaln(case, gen, seed):
    B, L, C = case["B"], case["L"], case["C"]
    train = case["mode"] == "jvp_train"
    stream = torch.float32 if train else torch.bfloat16
    x, h, mod = _randn(gen, B, L, C, dtype=stream), _randn(gen, B, L, C), _randn(gen, B, 1, 6 * C, std=0.5)
    if not train:
        return {"kind": "adaln", "args": (x, h, mod), "tangents": None}
    args = tuple(t.requires_grad_(True) for t in (x, h, mod))
    return {"kind": "adaln", "args": args,
            "tangents": (_randn(gen, B, L, C, dtype=stream, std=0.1), _randn(gen, B, L, C, std=0.1), _randn(gen, B, 1, 6 * C, std=0.05)),
            "dout": (_randn(gen, B, L, C), _randn(gen, B, L, C, dtype=stream))}


def _prepare_tail(case, gen, seed):
    f = lambda std: _randn(gen, case["count"], dtype=torch.float32, std=std)
    param = f(0.02)
    opt = FlatAdamW(param, lr=1e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.0)
    opt.exp_avg.copy_(f(1e-4))
    opt.exp_avg_sq.copy_(f(1e-4).square_())
    opt.step_count = 1000
    return {"kind": "tail", "opt": opt, "param": param, "ema": f(0.02), "grad": f(1e-3)}


def _prepare_sample(case, gen, seed):
    side = case["px"] // 8
    torch.manual_seed(seed)
    with torch.device(DEV):
        model = build_dmft(case["model"], input_size=side, dmf_depth=_dmf_depth(case), use_logvar=False, num_classes=1000,
                           attn_func="fa3", qk_norm=case["px"] == 512)
        model.initialize_weights(zero_init=False)           # trained gates are not zero
    model = model.to(torch.bfloat16).eval().requires_grad_(False)
    z = _randn(gen, case["B"], 4, side, side)
    y = torch.randint(0, 1000, (case["B"],), device=DEV, generator=gen)
    kw = dict(num_steps=STEPS, shift=1.5 if case["px"] == 512 else 1.0, cfg_scale=1.0)
    if case["graphs"]:
        call = GraphedSampler(model, case["B"], (4, side, side), torch.bfloat16, DEV, **kw)
    else:
        call = lambda z, y: euler_sampler(model, z, y, **kw)
    return {"kind": "sample", "call": call, "model": model, "z": z, "y": y}   # a captured graph reads the model's weights


def _prepare_train(case, gen, seed):
    torch.manual_seed(seed)
    with torch.device(DEV):
        state = training.build_train_state(torch.device(DEV), name=case["model"], input_size=case["px"] // 8,
                                           dmf_depth=_dmf_depth(case), attn_func="fa3", qk_norm=case["px"] == 512,
                                           seed=seed, zero_init=False, graphs=True)
    batch = training.synthetic_batch(state, case["B"], generator=gen)
    # the program's first step captures its graph; it is undone below so that run() starts from known weights
    keep = [t.clone() for t in (state.flat_param, state.flat_ema)]
    training.train_step(state, [batch])
    for t, k in zip((state.flat_param, state.flat_ema), keep):
        t.copy_(k)
    opt = state.flat_opt
    opt.exp_avg.zero_(), opt.exp_avg_sq.zero_()
    opt.step_count = 0
    torch.manual_seed(seed)                                 # the loss draws its times and noise inside the step
    return {"kind": "train", "state": state, "batch": batch}


def _dmf_depth(case):
    """Encoder blocks, in the proportion the 28-block model uses (20)."""
    return DMFT_CONFIGS[case["model"]]["depth"] * 20 // 28


# ---- one pass -------------------------------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "attn":
        return _run_grad(s, s["fn"]) if s.get("grad") else (
            s["fn"](*s["args"]) if s["tangents"] is None else torch.func.jvp(s["fn"], s["args"], s["tangents"]))
    if kind == "qk_norm":
        if s["tangents"] is None:
            return _norms(*s["args"])
        q, k, wq, wk = s["args"]
        out, tangent = torch.func.jvp(lambda q, k: _norms(q, k, wq, wk), (q, k), s["tangents"])
        return (*out, *tangent, *torch.autograd.grad(out, s["args"], s["dout"]))
    if kind == "adaln":
        if s["tangents"] is None:
            return _block_ops(*s["args"])
        out, tangent = torch.func.jvp(_block_ops, s["args"], s["tangents"])
        return (*out, *tangent, *torch.autograd.grad(out, s["args"], s["dout"]))
    if kind == "tail":
        opt = s["opt"]
        opt.step_tail(s["grad"], s["param"], s["ema"], s["grad"].norm(2), max_grad_norm=1.0, ema_decay=0.9999)
        return s["param"], s["ema"], opt.exp_avg, opt.exp_avg_sq, s["grad"]
    if kind == "sample":
        return s["call"](s["z"], s["y"])
    state = s["state"]
    loss = training.train_step(state, [s["batch"]])
    return loss, state.flat_param, state.flat_ema, state.flat_opt.exp_avg


def _run_grad(s, fn):
    if s["tangents"] is None:
        out = fn(*s["args"])
        return (out, *torch.autograd.grad(out, s["args"], s["dout"]))
    out, tangent = torch.func.jvp(fn, s["args"], s["tangents"])
    return (out, tangent, *torch.autograd.grad(out, s["args"], s["dout"]))


def _norms(q, k, wq, wk):
    return rms_norm(q, wq), rms_norm(k, wk)


def _block_ops(x, h, mod):
    """What one half of a block does around its attention or MLP: `h` stands for that branch's output."""
    shift, scale, gate = mod.chunk(6, dim=-1)[:3]
    return adaln.ln_modulate(x, shift, scale, out_dtype=torch.bfloat16), adaln.gate_residual(x, gate, h)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "attn":
        B, L, H, D, mode = case["B"], case["L"], case["H"], case["D"], case["mode"]
        n, rows = 2 * B * L * H * D, 4 * B * H * L
        flops, size = (12, 8 * n + rows) if mode.startswith("jvp") else (4, 4 * n + rows)
        if mode.endswith("train"):
            flops, size = flops + 10, size + 8 * n + rows
        return {"bytes": size, "flops": flops * B * H * L * L * D}
    if kind == "qk_norm":
        n = 2 * case["B"] * case["L"] * case["H"] * case["D"]
        # forward: x, y (and tangents); backward: dy, x, dx; twice (q and k)
        return {"bytes": 2 * n * (7 if case["mode"] == "jvp_train" else 2), "flops": 2 * n * (10 if case["mode"] == "jvp_train" else 2)}
    if kind == "adaln":
        n = case["B"] * case["L"] * case["C"]
        if case["mode"] == "fwd":                           # read x, h; write y, out: all bf16
            return {"bytes": 8 * n, "flops": 12 * n}
        # forward: x, tx (fp32), h, th (bf16) in, y, ty (bf16), out, tout (fp32) out;
        # backward: dy (bf16), dout (fp32), x (fp32), h (bf16) in, dx (fp32), dh (bf16) out
        return {"bytes": 24 * n + 18 * n, "flops": 60 * n}
    if kind == "tail":                                      # norm: grad; step: grad, param, two moments, EMA both ways
        return {"bytes": (4 + 40) * case["count"], "flops": 20 * case["count"]}
    cfg, L = DMFT_CONFIGS[case["model"]], (case["px"] // 16) ** 2
    C, depth, B, P = cfg["hidden_size"], cfg["depth"], case["B"], PARAMS[case["model"]]
    linear = depth * (24 * C * C * B * L + 12 * C * C * B)  # one forward through the block's Linear layers
    attn = depth * B * L * L * C
    if kind == "sample":
        return {"bytes": STEPS * 2 * P, "flops": STEPS * (linear + 4 * attn)}
    # flow-matching forward, forward + tangent, two backwards (each twice a forward's products)
    return {"bytes": 44 * P, "flops": (1 + 2 + 2 + 2) * linear + (4 + 12 + 10 + 10) * attn}


def tolerance(case):
    kind = case["kind"]
    if kind == "tail":
        return {"rel": 1e-5}                                # fp32 throughout
    if kind in ("sample", "train"):
        return {"rel": 2e-2}                                # bf16 products through every block
    return {"rel": 2e-3 if case.get("dtype") == "fp16" else 1e-2}
