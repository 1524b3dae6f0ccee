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


_PLAIN_TENSORS = (torch.Tensor, nn.Parameter, type(None))


def is_plain_linear(module: nn.Module) -> bool:
    """Whether calling ``module`` is nothing but ``x @ weight.T (+ bias)`` on ordinary tensors: no derived class, no hooks, no parameter in another
    form (a quantised or sharded tensor subclass).  Callers may then take the weight and join the product with what surrounds it."""
    return type(module) in (nn.Linear, Linear) and not has_hooks(module) and type(module.weight) in _PLAIN_TENSORS and type(module.bias) in _PLAIN_TENSORS
