"""The native host path (csrc/torch_host.cpp): one C++ call per op for plain CUDA tensors, with or without autograd and under
one ``torch.func.jvp``.  Its functions return None for everything else, and the caller takes the general route.

``takes`` comes before them: what torch.compile traces, and tensors or modes with a __torch_function__ of their own, have to see
the ops of the general route.

The module is built (if stale) and loaded by the first call with a CUDA tensor, like libdmf_attn.so: a program that runs none
of the kernels needs neither the libraries nor a CUDA toolkit.

With DMF_ATTN_CHECK=1 (which reads the device status word back after every call) every function returns None.
"""

from __future__ import annotations

import importlib.util
import os
import threading

import torch
from torch.overrides import _get_current_function_mode_stack, has_torch_function
from torch.utils._device import DeviceContext

from . import _lib
from . import build as _build

# DMF_ATTN_CHECK=1 reads the status word back after every call (synchronises; for tests and debugging).
CHECK_EVERY_CALL = os.environ.get("DMF_ATTN_CHECK", "0") == "1"


def takes(*tensors) -> bool:
    """Whether a call on these tensors may go past torch's Python-level dispatch."""
    if torch.compiler.is_compiling():
        return False
    if not has_torch_function(tensors):
        return True
    # `with torch.device(...)` and set_default_device are function modes too, but concern factory functions only
    return (all(type(m) is DeviceContext for m in _get_current_function_mode_stack())
            and all(type(t) is torch.Tensor
                    or getattr(type(t), "__torch_function__", None) is torch._C._disabled_torch_function_impl
                    for t in tensors))


_module = None
_lock = threading.Lock()


def _loaded():
    """The native module, built and loaded on first use."""
    global _module
    if _module is None:
        with _lock:
            if _module is None:
                _lib.load()            # libdmf_attn.so first: built if stale, ABI version checked
                spec = importlib.util.spec_from_file_location("_dmf_torch", _build.build_host())
                module = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(module)
                for name, stub in _stubs.items():      # later calls go straight to the native function
                    if globals()[name] is stub and not CHECK_EVERY_CALL:
                        globals()[name] = getattr(module, name)
                _module = module
    return _module


def _stub(name):
    def first_call(*args):
        if CHECK_EVERY_CALL or not any(isinstance(a, torch.Tensor) and a.is_cuda for a in args):
            return None
        return getattr(_loaded(), name)(*args)
    return first_call


_stubs = {name: _stub(name) for name in ("attn_func", "attn_qkvpacked", "rms_norm", "ln_modulate", "gate_residual", "gelu")}
globals().update(_stubs)


def set_status_word(index: int, pointer: int) -> None:
    _loaded().set_status_word(index, pointer)


def launch_count() -> int:
    return 0 if _module is None else _module.launch_count()


def add_launches(n: int) -> None:
    """One step, unlike reading, adding and setting: the native functions count without the GIL, backward on other threads."""
    _loaded().add_launches(n)


def set_launch_count(n: int) -> None:
    if n or _module is not None:
        _loaded().set_launch_count(n)
