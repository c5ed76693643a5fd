"""The layers' projections with bias gradients from the package's own column-sum kernel.

``project(module, x)`` is ``module(x)`` and ``project_pair(a, b, x)`` is ``(a(x), b(x))``: same
values, same gradients.  A plain ``nn.Linear`` on a large CUDA input that takes part in training
runs through ``csrc/torch_host.cpp`` instead of ``F.linear``: the products are the same library
calls, but the bias gradient comes from ``csrc/msda_linear.cu`` (torch's reduction took 230 of the
840 us of an encoder layer's forward + backward), and the two projections of one input add their
input gradients inside the second product instead of in a pass of its own.  Anything else - other
modules in the layer's place, hooks, autocast, tracing, small inputs - calls the modules.
"""

from __future__ import annotations

import torch
from torch import Tensor, nn
from torch.nn.modules import module as _module

from .._loader import host_module

__all__ = ["project", "project_pair"]

_HOOKS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")


def _plain(m: nn.Module) -> bool:
    return (type(m) is nn.Linear and m.bias is not None and not any(getattr(m, h) for h in _HOOKS)
            and "forward" not in m.__dict__)


def _native(x: Tensor, *modules: nn.Module):
    if (torch.compiler.is_compiling() or not x.is_cuda or not torch.is_grad_enabled()
            or _module._has_any_global_hook() or not all(map(_plain, modules))):
        return None
    return host_module()


def project(module: nn.Module, x: Tensor) -> Tensor:
    native = _native(x, module)
    if native is not None:
        out = native.linear(x, module.weight, module.bias)
        if out is not None:
            return out
    return module(x)


def project_pair(a: nn.Module, b: nn.Module, x: Tensor) -> tuple[Tensor, Tensor]:
    native = _native(x, a, b)
    if native is not None:
        out = native.linear_pair(x, a.weight, a.bias, b.weight, b.bias)
        if out is not None:
            return out
    return a(x), b(x)
