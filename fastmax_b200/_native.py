"""Access to ``_host``, the C++ host side of the package's frequent calls (``csrc/host_binding.cpp``).

``host()`` is the module, or None where it was not built; ``plain_mode()`` says whether nothing is active that the Python
autograd functions take part in and C++ ones do not: tracing, compilation, functorch transforms, dispatch and function
modes.  A torch that does not offer these queries counts as one in which something is active.
"""
from __future__ import annotations

import torch

_module = None
_looked = False
_TENSORS = (torch.Tensor, torch.nn.Parameter)
_NUMBERS = (int, float)

try:
    from torch.overrides import _get_current_function_mode_stack as _function_modes
    from torch.utils._device import DeviceContext as _DeviceContext

    _queries = (torch._C._functorch.peek_interpreter_stack, torch._C._get_tracing_state, torch._C._len_torch_dispatch_stack,
                torch._C._len_torch_function_stack)
except (ImportError, AttributeError):
    _queries = None


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
    if torch.compiler.is_compiling() or _queries is None:
        return False
    transforms, tracing, dispatch_modes, function_modes = _queries
    if transforms() is not None or tracing() is not None or dispatch_modes():
        return False
    # a default device is a function mode too, but every allocation here names its device
    return not function_modes() or all(type(m) is _DeviceContext for m in _function_modes())


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
