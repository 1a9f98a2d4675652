"""Loader of the compiled torch binding (``cott_torch_binding.so``, built from ``csrc_torch/torch_binding.cpp`` by
``python -m cottention_transformer_b200.build``).

The binding is a thin C++ layer over the same C ABI that ``_lib`` reaches through ctypes: the reference's four
``FastAttention2.kernel`` functions with their pybind signature, and the fused operators as ``torch.ops.cottention_b200.*``.
When the file is there the package uses it (fewer Python-level calls per step); when it is not, the ctypes route does
the same work -- both end in the same CUDA kernels, neither is a fallback off the GPU.
"""
from __future__ import annotations

import importlib.util
import os

import torch
from torch.autograd import forward_ad as _fw

_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cott_torch_binding.so")
_mod = None
_tried = False
# (bound here: transformed() runs before every call)
_compiling, _tracing, _functorch, _modes = (torch.compiler.is_compiling, torch._C._is_tracing, torch._C._functorch.peek_interpreter_stack,
                                            torch._C._len_torch_dispatch_stack)


def module():
    """The compiled module, or None when it has not been built."""
    global _mod, _tried
    if not _tried:
        _tried = True
        if os.path.exists(_PATH) and os.environ.get("COTT_NO_TORCH_BINDING", "") != "1":
            spec = importlib.util.spec_from_file_location("cott_torch_binding", _PATH)
            mod = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(mod)  # also registers torch.ops.cottention_b200.*
            _mod = mod
    return _mod


def transformed() -> bool:
    """Whether something looks at a Python function and its operators, or refuses them by name, and would not see the nodes
    of the compiled module: tracing, compilation, functorch transforms, forward-mode differentiation, dispatch modes (which
    count, record or choose operators, as selective checkpointing does)."""
    return _compiling() or _tracing() or _functorch() is not None or _modes() > 0 or _fw._current_level >= 0


def autograd():
    """The module whose functions carry their own autograd nodes, or None where the Python autograd functions are needed:
    without the binding, and where the call is ``transformed()``."""
    return None if transformed() else module()


def ops():
    """``torch.ops.cottention_b200`` when the binding is loaded, else None."""
    if module() is None:
        return None
    return torch.ops.cottention_b200
