"""The one-token step of a plain decoder on its KV caches as a CUDA graph.

A step of a small model is a few hundred launches of a few microseconds each, and the host needs longer to issue one than the GPU to run it."""
from __future__ import annotations

import threading
from typing import Optional, Set, Tuple

import torch
from torch import nn
from torch.utils._device import DeviceContext

from .. import ops
from ..modules import FeedForward, KVCache, MultiHeadAttention, RMSNorm, TransformerDecoder, TransformerSelfAttentionLayer
from ..modules.linear import Linear, has_hooks
from ..modules.position_embeddings import RotaryPositionalEmbeddings
from ..modules.tied_linear import TiedLinear
from ._native_layers import NativeLayers

# Modules whose forward pass of one token is the same sequence of launches in every step and needs no look at the device.
_PLAIN = (TransformerDecoder, TransformerSelfAttentionLayer, MultiHeadAttention, FeedForward, KVCache, RMSNorm, Linear, nn.Linear, nn.Embedding, nn.ModuleList, nn.Identity,
          nn.SiLU, nn.GELU, nn.ReLU)


def _alone() -> bool:
    """Whether no other thread of this program could get in the way of a recording or be hurt by it: until it ends, a thread that waits for the device or draws random
    numbers on it fails, and the former breaks the recording.  Any other thread counts, except the one that keeps progress bars up to date."""
    here = threading.current_thread()
    return all(t is here or type(t).__module__ == "tqdm._monitor" for t in threading.enumerate())


class _LastGraph:
    """The graph that last ran on a cache and the stream it was recorded on.  The next one shares both and with them the memory pool (its blocks belong to a
    stream), so that any number of generations on one set of caches hold one pool, which goes with the caches.  Copies and pickles of the cache
    come without it."""

    def __init__(self) -> None:
        self.graph: Optional[torch.cuda.CUDAGraph] = None
        self.stream: Optional[torch.cuda.Stream] = None
        self.stepped: Set[Tuple[int, ...]] = set()  # the way (native or not), batch and mask shape of the steps that have run as they are

    def __deepcopy__(self, memo) -> "_LastGraph":
        return _LastGraph()

    def __reduce__(self):
        return _LastGraph, ()


class StepGraph:
    """``model(x, input_pos, mask)[:, -1]`` for one token per row: a call is recorded, and it and all later ones replay the recording on the inputs
    that they are given.  The first step of a batch and mask shape on a set of caches, by the modules and by the native call, runs as it is, so that the one-time set-up of the kernels that
    these sizes choose stays out of the recording.  While the program has other threads, all calls run as they are."""

    @staticmethod
    def suits(model: nn.Module, like: torch.Tensor) -> bool:
        if type(model) is not TransformerDecoder or not like.is_cuda or model.tok_embeddings.weight.dtype != torch.bfloat16 or model.loop is not None:
            return False
        if model.num_output_chunks or model.output_hidden_states or model.skip_output_layer or model.pos_embeddings is not None:
            return False
        if type(model.output) not in (Linear, nn.Linear, TiedLinear):
            return False
        modes = torch.overrides._get_current_function_mode_stack()
        if not ops.cuda_ops_enabled(like) or torch._C._len_torch_dispatch_stack() or any(type(m) is not DeviceContext for m in modes):  # somebody wants to see every operation
            return False
        if torch.is_inference_mode_enabled() or torch.cuda.is_current_stream_capturing() or torch.autograd.forward_ad._current_level >= 0:
            return False
        for m in model.modules():
            rotary = isinstance(m, RotaryPositionalEmbeddings) and type(m).forward is RotaryPositionalEmbeddings.forward
            if not (rotary or type(m) in _PLAIN) or has_hooks(m):
                return False
        for layer in model.layers:
            if type(layer) is not TransformerSelfAttentionLayer or layer.mask_mod is not None or type(layer.attn) is not MultiHeadAttention:
                return False
            attn = layer.attn
            if type(attn.kv_cache) is not KVCache or not attn.cache_enabled or attn.kv_cache.cache_pos.is_inference() or getattr(attn, "context_parallel", None) is not None:
                return False
            if attn.training and attn.attn_dropout:
                return False
        return all(p.device == like.device and p.dtype == torch.bfloat16 for p in model.parameters())

    def __init__(self, model: TransformerDecoder, batch: int, native: Optional[NativeLayers] = None) -> None:
        self.model, self.batch, self.native = model, batch, native
        self.caches = [layer.attn.kv_cache for layer in model.layers]
        self.graph: Optional[torch.cuda.CUDAGraph] = None
        self.home: _LastGraph = self.caches[0].__dict__.setdefault("last_graph", _LastGraph())

    def __call__(self, x: torch.Tensor, input_pos: torch.Tensor, mask: torch.Tensor) -> torch.Tensor:
        if self.graph is None:
            sizes = (self.native is not None, self.batch, *mask.shape)  # the native call runs kernels of its own
            if sizes not in self.home.stepped or not _alone():
                logits = self._step(x, input_pos, mask)
                self.home.stepped.add(sizes)
                return logits
            self._record(x, input_pos, mask)
        for cache in self.caches:
            cache.reserve(self.batch, 1)  # raises when the cache is full
        self.x.copy_(x)
        self.pos.copy_(input_pos.view(-1, 1))
        self.mask.copy_(mask)
        self.graph.replay()
        for cache in self.caches:
            cache.advanced(1)
        return self.logits.clone()

    def _step(self, x: torch.Tensor, input_pos: torch.Tensor, mask: torch.Tensor) -> torch.Tensor:
        logits = None if self.native is None else self.native.last_logits(x, input_pos, mask)
        return self.model(x, input_pos=input_pos, mask=mask)[:, -1] if logits is None else logits

    def _record(self, x: torch.Tensor, input_pos: torch.Tensor, mask: torch.Tensor) -> None:
        device = x.device
        for cache in self.caches:
            cache.reserve(self.batch, 1)
        self.x, self.mask = torch.empty_like(x), torch.empty_like(mask)
        self.pos = torch.empty(self.batch, 1, dtype=torch.int32, device=device)
        if self.home.stream is None or self.home.stream.device != device:
            self.home.stream = torch.cuda.Stream(device=device)
        graph, stream = torch.cuda.CUDAGraph(), self.home.stream
        stream.wait_stream(torch.cuda.current_stream(device))
        for cache in self.caches:
            cache.recording = True
        try:
            with torch.cuda.stream(stream):
                graph.capture_begin(**({} if self.home.graph is None else {"pool": self.home.graph.pool()}), capture_error_mode="thread_local")
                try:
                    self.logits = self._step(self.x, self.pos, self.mask)
                    torch._foreach_add_([cache.cache_pos for cache in self.caches], 1)
                finally:
                    graph.capture_end()
        finally:
            for cache in self.caches:
                cache.recording = False
        torch.cuda.current_stream(device).wait_stream(stream)
        self.graph = self.home.graph = graph
