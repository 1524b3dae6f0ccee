"""What a KV cache believes about its own level: the device decides, and is asked once per append or once per forward pass."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from torchtune_b200.models.llama3_1 import llama3_1
from torchtune_b200.modules import KVCache
from torchtune_b200.modules.kv_cache import counted_appends


class _Reads(TorchDispatchMode):
    """Counts the values that operations hand to the host."""

    def __init__(self):
        super().__init__()
        self.count = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.count += func in (torch.ops.aten._local_scalar_dense.default, torch.ops.aten.item.default)
        return func(*args, **(kwargs or {}))


def _kv(n, b=2):
    return torch.randn(b, n, 1, 4), torch.randn(b, n, 1, 4)


@pytest.mark.parametrize("inference", [False, True])
def test_one_read_per_append(inference):
    with torch.inference_mode(inference):
        cache = KVCache(2, 8, 1, 4, torch.float32)
        cache.update(*_kv(3))
        with _Reads() as reads:
            cache.update(*_kv(2))
        assert reads.count <= 1 and cache.size == 5


@pytest.mark.parametrize("inference", [False, True])
def test_writes_past_the_module_are_seen(inference):
    """Through ``.data`` or a replayed graph no version counter moves; the cache is as full as its positions say."""
    with torch.inference_mode(inference):
        cache = KVCache(2, 8, 1, 4, torch.float32)
        cache.update(*_kv(3))
        assert cache.size == 3
        cache.cache_pos.data.add_(4)
        assert cache.size == 7
        with pytest.raises(AssertionError, match="full"):
            cache.update(*_kv(2))
        cache.update(*_kv(1))
        cache.cache_pos.data.sub_(8)
        k, _ = _kv(8)
        assert torch.equal(cache.update(k, k)[0], k)


def test_counted_appends():
    caches = [KVCache(2, 8, 1, 4, torch.float32) for _ in range(3)]
    caches[1].update(*_kv(2))
    with _Reads() as reads, counted_appends(caches):
        before = reads.count
        for c in caches:
            c.update(*_kv(5))
        with counted_appends(caches[:1]):  # within another block: that one goes on counting
            caches[0].update(*_kv(1))
        assert [c.size for c in caches] == [6, 7, 5] and reads.count == before
        with pytest.raises(AssertionError, match="full"):
            caches[1].update(*_kv(2))
        caches[2].reset()
        assert caches[2].size == 0
    assert [c._level for c in caches] == [None] * 3 and [c.size for c in caches] == [6, 7, 0]
    with pytest.raises(ValueError, match="stop"), counted_appends(caches):
        raise ValueError("stop")
    assert [c._level for c in caches] == [None] * 3


@pytest.mark.parametrize("inference", [False, True])
def test_one_read_per_forward_pass(inference):
    torch.manual_seed(0)
    model = llama3_1(vocab_size=64, num_layers=4, num_heads=4, num_kv_heads=2, embed_dim=32, max_seq_len=32, intermediate_dim=64).eval()
    with torch.inference_mode(inference), torch.no_grad():
        model.setup_caches(batch_size=1, dtype=torch.float32, decoder_max_seq_len=12)
        mask = torch.tril(torch.ones(12, 12, dtype=torch.bool))[None]
        x = torch.randint(0, 64, (1, 12))
        first = model(x[:, :7], input_pos=torch.arange(7)[None], mask=mask[:, :7])
        for layer in model.layers:  # back by two tokens, past the version counter
            layer.attn.kv_cache.cache_pos.data.sub_(2)
        with _Reads() as reads:
            second = model(x[:, 5:9], input_pos=torch.arange(5, 9)[None], mask=mask[:, 5:9])
        assert reads.count <= 1 and [layer.attn.kv_cache.size for layer in model.layers] == [9] * 4
        torch.testing.assert_close(second[:, :2], first[:, 5:])
