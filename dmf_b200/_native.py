"""The native host path (csrc/torch_host.cpp): one C++ call per op for plain CUDA tensors, with or without autograd and under
one ``torch.func.jvp``.  Its functions return None for everything else, and the caller takes the general route.

``takes`` comes before them: what torch.compile traces, and tensors or modes with a __torch_function__ of their own, have to see
the ops of the general route.

With DMF_ATTN_CHECK=1 (which reads the device status word back after every call) every function returns None.
"""

from __future__ import annotations

import importlib.util
import os

import torch
from torch.overrides import _get_current_function_mode_stack, has_torch_function
from torch.utils._device import DeviceContext

from . import _lib
from . import build as _build


def takes(*tensors) -> bool:
    """Whether a call on these tensors may go past torch's Python-level dispatch."""
    if torch.compiler.is_compiling():
        return False
    if not has_torch_function(tensors):
        return True
    # `with torch.device(...)` and set_default_device are function modes too, but concern factory functions only
    return (all(type(m) is DeviceContext for m in _get_current_function_mode_stack())
            and all(type(t) is torch.Tensor or type(t).__torch_function__ is torch._C._disabled_torch_function_impl
                    for t in tensors))


def _load():
    _lib.load()                    # libdmf_attn.so first: built if stale, ABI version checked
    spec = importlib.util.spec_from_file_location("_dmf_torch", _build.build_host())
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


_module = _load()
launch_count, set_launch_count, set_status_word = _module.launch_count, _module.set_launch_count, _module.set_status_word

# DMF_ATTN_CHECK=1 reads the status word back after every call (synchronises; for tests and debugging).
CHECK_EVERY_CALL = os.environ.get("DMF_ATTN_CHECK", "0") == "1"

if CHECK_EVERY_CALL:
    attn_func = attn_qkvpacked = rms_norm = ln_modulate = gate_residual = gelu = lambda *args: None
else:
    attn_func, attn_qkvpacked = _module.attn_func, _module.attn_qkvpacked
    rms_norm, ln_modulate, gate_residual, gelu = _module.rms_norm, _module.ln_modulate, _module.gate_residual, _module.gelu
