"""What the native call for all layers of a decoder needs on the host."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from torchtune_b200.generation._native_layers import NativeLayers


@pytest.mark.parametrize("device", ["cpu", "meta"])
def test_addresses_stay_on_the_host(device):
    """The call reads the layers' addresses from host memory, whatever device the program makes its tensors on."""
    layers = [SimpleNamespace(attn=SimpleNamespace(kv_cache=SimpleNamespace(cache_pos=torch.arange(4)))) for _ in range(2)]
    words = [2**63 - 1, 0, 7, 140_000_000_000_016]
    with torch.device(device):
        native = NativeLayers(SimpleNamespace(layers=layers), 1, (8, 1, 1, 8, 8, 4), 1e-5, 1.0, 0, words)
    assert isinstance(native.words, ctypes.Array) and list(native.words) == words
