"""Access to ``_host``, the C++ host side of the package's frequent calls (``csrc/host_binding.cpp``).

``host()`` is the module, or None where it was not built; ``plain_mode()`` says whether nothing is active that the Python
autograd functions take part in and C++ ones do not: tracing, compilation, functorch transforms, dispatch and function
modes.
"""
from __future__ import annotations

import torch
from torch.overrides import _get_current_function_mode_stack as _function_modes
from torch.utils._device import DeviceContext as _DeviceContext

_module = None
_looked = False
_TENSORS = (torch.Tensor, torch.nn.Parameter)
_NUMBERS = (int, float)


def host():
    global _module, _looked
    if not _looked:
        from . import _cabi

        _cabi.lib()                     # the CUDA library first, with its own error where it is missing
        try:
            from . import _host as module
        except ImportError:
            module = None
        _module, _looked = module, True
    return _module


def plain_mode() -> bool:
    c = torch._C
    if (c._functorch.peek_interpreter_stack() is not None or c._get_tracing_state() is not None
            or c._len_torch_dispatch_stack() or torch.compiler.is_compiling()):
        return False
    # a default device is a function mode too, but every allocation here names its device
    return not c._len_torch_function_stack() or all(type(m) is _DeviceContext for m in _function_modes())


def plain_tensors(*tensors) -> bool:
    """Tensors on a CUDA device that are no subclass with a behaviour of its own."""
    for t in tensors:
        if type(t) not in _TENSORS or not t.is_cuda:
            return False
    return True


def plain_numbers(*values) -> bool:
    for x in values:
        if type(x) not in _NUMBERS:
            return False
    return True
