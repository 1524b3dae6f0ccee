"""When a projection may be joined with its surroundings instead of being called."""
import pytest
import torch
from torch import nn

from torchtune_b200.models.llama3_1 import llama3_1
from torchtune_b200.modules.linear import Linear, has_hooks, is_plain_linear


def _layer():
    return llama3_1(vocab_size=64, num_layers=1, num_heads=4, num_kv_heads=2, embed_dim=32, max_seq_len=32, intermediate_dim=64).layers[0]


def _watched(how, module):
    if how == "forward hook":
        module.register_forward_hook(lambda *a: None)
    elif how == "forward pre-hook":
        module.register_forward_pre_hook(lambda *a: None)
    elif how == "backward hook":
        module.register_full_backward_hook(lambda *a: None)
    elif how == "replaced forward":
        module.forward = module.forward
    else:
        module.compile(backend="eager")


WAYS = ["forward hook", "forward pre-hook", "backward hook", "replaced forward", "compiled"]


@pytest.mark.parametrize("how", WAYS)
@pytest.mark.parametrize("kind", [Linear, nn.Linear])
def test_watched_and_compiled_projections_are_called(kind, how):
    lin = kind(8, 8)
    assert is_plain_linear(lin) and not has_hooks(lin)
    _watched(how, lin)
    assert has_hooks(lin) and not is_plain_linear(lin)


@pytest.mark.parametrize("how", WAYS)
@pytest.mark.parametrize("name", ["w1", "w3", "activation"])
def test_watched_gates_are_called(name, how):
    mlp = _layer().mlp
    assert mlp._fusable()
    _watched(how, getattr(mlp, name))
    assert not mlp._fusable()
    if how == "forward hook":  # and what it returns counts
        getattr(mlp, name).register_forward_hook(lambda m, args, out: torch.zeros_like(out))
        assert not mlp(torch.randn(3, 32)).any()


class _Wrapped(torch.Tensor):
    """Stands for a weight that is held in another form and has no bytes of its own to point to."""


@pytest.mark.parametrize("kind", [Linear, nn.Linear])
@pytest.mark.parametrize("part", ["weight", "bias"])
def test_projections_with_wrapped_parameters_are_called(kind, part):
    lin = kind(8, 8)
    setattr(lin, part, nn.Parameter(getattr(lin, part).detach().as_subclass(_Wrapped), requires_grad=False))
    assert isinstance(getattr(lin, part), _Wrapped) and not is_plain_linear(lin)


@pytest.mark.parametrize("kind", [Linear, nn.Linear])
@pytest.mark.parametrize("grad", [False, True])
def test_only_this_package_s_projections_are_joined_and_only_outside_autograd(kind, grad, monkeypatch):
    """torch's own linear layers keep torch's own product: autocast, weights in other forms and modes that look at operations see it."""
    from torchtune_b200 import ops
    from torchtune_b200.modules import MultiHeadAttention

    joined = []
    plain = ops.linear_group
    monkeypatch.setattr(ops, "linear_group", lambda *a: joined.append(a) or plain(*a))
    attn = MultiHeadAttention(embed_dim=32, num_heads=4, num_kv_heads=2, head_dim=8, q_proj=kind(32, 32), k_proj=kind(32, 16), v_proj=kind(32, 16), output_proj=kind(32, 32))
    x = torch.randn(1, 3, 32)
    with torch.set_grad_enabled(grad):
        attn(x, x)
    assert len(joined) == (kind is Linear and not grad)
