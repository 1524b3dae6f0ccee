"""Linear layer routed through :func:`torchtune_b200.ops.linear`."""
from __future__ import annotations

import torch
from torch import nn

from .. import ops


class Linear(nn.Linear):
    """Drop-in ``nn.Linear`` (same parameters / state-dict keys) whose forward, dgrad
    and wgrad run the tcgen05 GEMM for bf16 CUDA tensors."""

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return ops.linear(x, self.weight, self.bias)


def has_hooks(module: nn.Module) -> bool:
    """Whether calling ``module`` runs anything beside its class's ``forward``: hooks of its own, hooks on all modules, a replaced ``forward`` or a
    compiled one (``module.compile()``)."""
    everywhere = nn.modules.module
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks or "forward" in module.__dict__
                or module._compiled_call_impl is not None
                or everywhere._global_forward_hooks or everywhere._global_forward_pre_hooks or everywhere._global_backward_hooks or everywhere._global_backward_pre_hooks)


def is_plain_linear(module: nn.Module) -> bool:
    """Whether calling ``module`` is nothing but ``x @ weight.T (+ bias)`` on ordinary tensors: no derived class, no hooks, no parameter in another
    form (a quantised or sharded tensor subclass).  Callers may then take the weight and join the product with what surrounds it."""
    if type(module) not in (nn.Linear, Linear) or has_hooks(module):
        return False
    own = module._parameters
    return type(own.get("weight")) is nn.Parameter and type(own.get("bias", module)) in (nn.Parameter, type(None))
