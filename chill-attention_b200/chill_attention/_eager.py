"""Eager-mode call path of ``chill_attention``: same kernels, less host time per call.

Under ``torch.compile`` the operator is reached through its dispatcher ops
(``chill_attention::forward<Name>`` / ``backward<Name>``, chill.py).  In plain eager mode that route costs
more host time than a short sequence needs on the GPU: a Python custom op is entered through the dispatcher
twice and its autograd rule is another Python layer.  Here an eager call goes to one native function
(csrc/torch_ext.cpp, built next to the kernel library) that checks the arguments, allocates the outputs, calls the
C ABI and records a C++ autograd node, so the backward runs without the interpreter.  Measured back to back against a
Python autograd.Function over ctypes: forward of (8, 4, 128, 128) 17 -> 8 us, forward + backward of (1, 2, 128, 64)
138 -> 78 us, most of the latter in torch's autograd engine and in five kernel launches.

The path is taken only for plain CUDA tensors outside of tracing / dispatch modes / functorch transforms
(``usable``); everything else, and every ``torch.compile`` graph, uses the dispatcher ops.  So does every call if the
native module is missing or does not load (the kernel library built alone, another torch than it was built for).  Set
``CHILL_ATTENTION_EAGER_FAST=0`` to switch it off.
"""
from __future__ import annotations

import ctypes as C
import importlib.util
import os
import threading
import warnings

import torch

from . import _cabi

ENABLED = os.environ.get("CHILL_ATTENTION_EAGER_FAST", "1") not in ("", "0")
EXTENSION = os.path.join(_cabi.LIB_DIR, "_chill_torch.so")

_dispatch_depth = getattr(torch._C, "_len_torch_dispatch_stack", None)
_function_depth = getattr(torch._C, "_len_torch_function_stack", None)
_functorch_top = getattr(getattr(torch._C, "_functorch", None), "peek_interpreter_stack", None)
_PROBES_OK = None not in (_dispatch_depth, _function_depth, _functorch_top)
_Tensor = torch.Tensor

_extension = None
_lock = threading.Lock()
#: entry points a native Library object is made of, in its order
_ENTRY_POINTS = ("chill_fwd", "chill_bwd_delta", "chill_bwd", "chill_bwd_uses_tensor_cores", "chill_bwd_dq_accum_bytes",
                 "chill_status_string", "chill_last_cuda_error")


def usable(q, k, v, lens) -> bool:
    """True when nothing is watching the dispatcher: plain tensors, no tracing, no modes, no transforms.
    (A torch without the probes used here stays on the dispatcher path.)"""
    if not (ENABLED and _PROBES_OK) or type(q) is not _Tensor or type(k) is not _Tensor or type(v) is not _Tensor:
        return False
    if not q.is_cuda or (lens is not None and type(lens) is not _Tensor):
        return False
    return _dispatch_depth() == 0 and _function_depth() == 0 and _functorch_top() is None


def extension():
    """The native module; built by ``python chill-attention_b200/build.py`` together with the kernel library."""
    global _extension
    if _extension is None:
        with _lock:
            if _extension is None:
                if not os.path.exists(EXTENSION):
                    raise _cabi.ChillLibraryError(f"{EXTENSION} not found: build it first (python chill-attention_b200/build.py)")
                spec = importlib.util.spec_from_file_location("_chill_torch", EXTENSION)
                mod = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(mod)
                if mod.abi_version != _cabi.ABI_VERSION:
                    raise _cabi.ChillLibraryError(f"{EXTENSION}: ABI version {mod.abi_version} != {_cabi.ABI_VERSION}")
                mod.set_deterministic(_cabi._deterministic)
                _extension = mod
    return _extension


def native_library(lib, functor_id):
    """The native call object of one mask functor: the kernel library's entry points and the functor id.  None, after one
    warning, if there is no native module to make it; ``usable`` says no from then on."""
    global ENABLED
    try:
        module = extension()
    except (ImportError, OSError, _cabi.ChillLibraryError) as e:
        ENABLED = False
        warnings.warn(f"chill_attention: eager calls go through the dispatcher ops, which take longer on the host: {e}", stacklevel=3)
        return None
    addresses = [C.cast(getattr(lib, name), C.c_void_p).value for name in _ENTRY_POINTS]
    return module.Library(addresses, functor_id)


def attention(native, q, k, v, lens, mask_args, sm_scale, return_lse, flags):
    """O, or (O, LSE): the eager counterpart of chill._chill_attention.  None if an argument check failed."""
    return _extension.attention(native, q, k, v, lens, mask_args, sm_scale, return_lse, flags)
