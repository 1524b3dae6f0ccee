"""Forward passes of a plain decoder on its KV caches with all layers issued by one native call (``ops/csrc/decoder_layers.cu``)."""
from __future__ import annotations

import ctypes
import os
from typing import List, Optional

import torch
from torch import nn

from .. import ops
from ..modules import FeedForward, KVCache, RMSNorm, TransformerDecoder
from ..modules.linear import Linear, has_hooks, is_plain_linear
from ..modules.position_embeddings import RotaryPositionalEmbeddings


def _plain(t: Optional[torch.Tensor], shape: tuple) -> bool:
    return type(t) in (torch.Tensor, nn.Parameter) and t.dtype == torch.bfloat16 and t.shape == shape and t.is_contiguous() and t.data_ptr() % 16 == 0


def _projection(module: nn.Module, rows: int, cols: int, bias: bool = False) -> bool:
    if type(module) is not Linear or not is_plain_linear(module) or not _plain(module.weight, (rows, cols)):
        return False
    return module.bias is None or (bias and _plain(module.bias, (rows,)))


class NativeLayers:
    """``model.norm`` of the layers' output for one ``generate`` call, on caches that nobody else writes to: addresses are taken when it is made.  The launches and results are
    those of the modules."""

    @classmethod
    def of(cls, model: TransformerDecoder, batch: int) -> Optional["NativeLayers"]:
        """For a model that :class:`StepGraph` suits; ``None`` if some module computes what the call does not."""
        from ..ops._cuda import _PAIR_KERNEL

        emb = model.tok_embeddings.weight
        if not emb.is_cuda or not ops.cuda_ops_enabled(emb) or not len(model.layers):
            return None
        if not _PAIR_KERNEL or any(os.environ.get(name, "1") == "0" for name in ("TTB_FUSE_RESIDUAL", "TTB_FUSE_SWIGLU")):  # switches that the modules follow
            return None
        if type(model.norm) is not RMSNorm or not _plain(model.norm.scale, emb.shape[1:]):
            return None
        first, dim, eps = model.layers[0], emb.shape[1], model.norm.eps
        hq, hkv, D, scale, cache = first.attn.num_heads, first.attn.num_kv_heads, first.attn.head_dim, first.attn.scale, first.attn.kv_cache
        hidden = getattr(getattr(first.mlp, "w1", None), "out_features", 0)
        interleaved = getattr(first.attn.pos_embeddings, "interleaved", True)
        words: List[int] = []
        for layer in model.layers:
            attn, mlp, kv, pe = layer.attn, layer.mlp, layer.attn.kv_cache, layer.attn.pos_embeddings
            if type(layer.sa_norm) is not RMSNorm or type(layer.mlp_norm) is not RMSNorm or layer.sa_norm.eps != eps or layer.mlp_norm.eps != eps:
                return None
            if type(layer.sa_scale) is not nn.Identity or type(layer.mlp_scale) is not nn.Identity or type(mlp) is not FeedForward or mlp.w3 is None:
                return None
            if type(mlp.activation) is not nn.SiLU or not mlp._silu or mlp._glu is not None or has_hooks(mlp.activation):
                return None
            if (attn.num_heads, attn.num_kv_heads, attn.head_dim, attn.scale) != (hq, hkv, D, scale) or attn.q_norm is not None or (attn.softcap or 0.0) > 0.0:
                return None
            if not isinstance(pe, RotaryPositionalEmbeddings) or type(pe).forward is not RotaryPositionalEmbeddings.forward or pe.interleaved != interleaved:
                return None
            table = pe.cache
            if table.dtype != torch.float32 or tuple(table.shape[1:]) != (D // 2, 2) or not table.is_contiguous() or table.data_ptr() % 16 or table.device != emb.device:
                return None
            shape = (cache.k_cache.shape[0], cache.max_seq_len, hkv, D)
            if type(kv) is not KVCache or shape[0] < batch or kv.cache_pos.dtype != torch.int64 or not kv.cache_pos.is_contiguous() or not (_plain(kv.k_cache, shape) and _plain(kv.v_cache, shape)):
                return None
            if not (_projection(attn.q_proj, hq * D, dim, True) and _projection(attn.k_proj, hkv * D, dim, True) and _projection(attn.v_proj, hkv * D, dim, True)):
                return None
            if not (_projection(attn.output_proj, dim, hq * D) and _projection(mlp.w1, hidden, dim) and _projection(mlp.w3, hidden, dim) and _projection(mlp.w2, dim, hidden)):
                return None
            if not (_plain(layer.sa_norm.scale, (dim,)) and _plain(layer.mlp_norm.scale, (dim,))):
                return None
            projections = (attn.q_proj, attn.k_proj, attn.v_proj)
            words += [layer.sa_norm.scale.data_ptr(), *(m.weight.data_ptr() for m in projections), attn.output_proj.weight.data_ptr(), layer.mlp_norm.scale.data_ptr(),
                      mlp.w1.weight.data_ptr(), mlp.w3.weight.data_ptr(), mlp.w2.weight.data_ptr(), *(0 if m.bias is None else m.bias.data_ptr() for m in projections),
                      kv.k_cache.data_ptr(), kv.v_cache.data_ptr(), kv.cache_pos.data_ptr(), table.data_ptr(), table.shape[0]]
        scale = D**-0.5 if scale is None else scale
        return None if scale <= 0.0 else cls(model, batch, (dim, hq, hkv, D, hidden, cache.max_seq_len), float(eps), float(scale), int(interleaved), words)

    def __init__(self, model: TransformerDecoder, batch: int, sizes: tuple, eps: float, scale: float, interleaved: int, words: List[int]) -> None:
        self.model, self.batch, self.sizes, self.eps, self.scale, self.interleaved = model, batch, sizes, eps, scale, interleaved
        self.caches = [layer.attn.kv_cache for layer in model.layers]
        self.positions = [cache.cache_pos for cache in self.caches]
        self.words = (ctypes.c_longlong * len(words))(*words)  # read by the host, so not a tensor, which would lie wherever the program makes tensors

    def __call__(self, x: torch.Tensor, input_pos: torch.Tensor, mask: torch.Tensor) -> Optional[torch.Tensor]:
        """Normalised hidden states ``[b, s, dim]`` of new tokens ``x`` ``[b, s]``, whose keys and values are appended; ``None``, with nothing done, for a mask or sizes that the call
        does not take."""
        from ..ops._cuda import _positions
        from ..ops._lib import check, err_word, lib, stream_ptr

        b, s = x.shape
        if b != self.batch or mask.dtype != torch.bool or mask.dim() != 3 or mask.shape[0] not in (1, b) or tuple(mask.shape[1:]) != (s, self.sizes[5]) or mask.stride(2) != 1:
            return None
        if not mask.is_cuda or not x.is_cuda or x.dtype not in (torch.int32, torch.int64):
            return None
        self.model._validate_inputs(s, mask=mask, input_pos=input_pos)
        count = len(self.caches)
        need = lib().ttb_decoder_layers_workspace(count, b, s, *self.sizes)
        if not need:
            return None
        for cache in self.caches:
            cache.reserve(b, s)  # raises when the cache is full
        h = ops.embed_tokens(self.model.tok_embeddings, x)
        y, work = torch.empty_like(h), torch.empty(need, dtype=torch.uint8, device=h.device)
        pos = _positions(input_pos, b, s, h.device)
        check(lib().ttb_decoder_layers(self.words, count, b, s, *self.sizes, self.eps, self.scale, self.interleaved, h.data_ptr(), y.data_ptr(), self.model.norm.scale.data_ptr(),
                                       pos.data_ptr(), mask.data_ptr(), mask.stride(0) if mask.shape[0] > 1 else 0, mask.stride(1), work.data_ptr(), err_word(h.device).data_ptr(),
                                       stream_ptr()), f"decoder layers for {b} x {s} tokens")
        if not self.caches[0].recording:  # a recorded step moves the positions on itself
            torch._foreach_add_(self.positions, s)
            for cache in self.caches:
                cache.advanced(s)
        return y

    def last_logits(self, x: torch.Tensor, input_pos: torch.Tensor, mask: torch.Tensor) -> Optional[torch.Tensor]:
        """Logits ``[b, vocab]`` of the last position."""
        h = self(x, input_pos, mask)
        return None if h is None else self.model.unembed_normed(h[:, -1:])[:, 0]
