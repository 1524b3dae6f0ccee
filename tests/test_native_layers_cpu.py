"""What the native call for all layers of a decoder needs on the host."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from torchtune_b200.generation._native_layers import NativeLayers
from torchtune_b200.ops import _cuda, _lib


@pytest.mark.parametrize("device", ["cpu", "meta"])
def test_addresses_stay_on_the_host(device):
    """The call reads the layers' addresses from host memory, whatever device the program makes its tensors on."""
    layers = [SimpleNamespace(attn=SimpleNamespace(kv_cache=SimpleNamespace(cache_pos=torch.arange(4)))) for _ in range(2)]
    words = [2**63 - 1, 0, 7, 140_000_000_000_016]
    with torch.device(device):
        native = NativeLayers(SimpleNamespace(layers=layers), 1, (8, 1, 1, 8, 8, 4), 1e-5, 1.0, 0, words)
    assert isinstance(native.words, ctypes.Array) and list(native.words) == words


@pytest.mark.skipif(not _lib.LIB_PATH.exists(), reason="the kernel library is not built")
def test_products_are_dealt_out_as_by_the_modules(monkeypatch):
    """The native call's rules for which kernel takes a product are those of the wrappers, on both sides of every line that they draw."""
    monkeypatch.setattr(_cuda, "_PAIR_KERNEL", True)
    near = lambda *lines: sorted({v + d for v in lines for d in (-1, 0, 1) if v + d > 0})
    sizes_m = near(1, 8, 16, 32, 64, 128, 256, 384, 512, 640, 768, 1024, 1152, 2048, 9472, 16384)
    sizes_n = near(8, 64, 128, 256, 1024, 2048, 4096, 8192, 9472, 14336, 18944, 32768, 128256)
    sizes_k = near(8, 64, 120, 128, 512, 1024, 2048, 4096, 4608, 8192, 14336, 128256)
    rules = _lib.lib().ttb_product_rules
    got = (ctypes.c_int * 4)()
    for pairs in (1, 66, 74):
        monkeypatch.setattr(_cuda, "_SM_PAIRS", pairs)
        for M in sizes_m:
            for N in sizes_n:
                for K in sizes_k:
                    rules(M, N, K, pairs, got)
                    want = [_cuda._runs_rows(M, N, K), _cuda._splits(M, N, K), _cuda._fills_pairs(M, N, K, None), _cuda._gates_in_pairs(M, N, K, None)]
                    assert list(got) == want, (M, N, K, pairs)
