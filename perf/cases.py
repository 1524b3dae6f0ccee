"""The workloads that this framework's speed is judged by, each as one call through its public entry points.

A case is a dict of plain values.  ``prepare`` makes what a training or serving program holds before the call (model, batch, caches),
``run`` is one pass, ``work`` the bytes and operations that the pass cannot do without, ``exact`` the same outputs in 64 bits from
plain torch, and ``draw`` gives further cases of the same ranges.

Models are the two Llama-3 decoders that the recipes and the benchmark train and serve, at their real widths, heads and vocabulary (8B:
128 channels per head, 1B: 64) and with fewer layers, since layers repeat; the expert layer has the sizes of Llama-4 Scout's."""
from __future__ import annotations

import math
from typing import Any, Dict, List, Optional, Tuple

import torch
from torch.utils.checkpoint import checkpoint

VOCAB = 128_256
WIDTHS = {  # dim, query heads, key heads, feed-forward width
    "8b": (4096, 32, 8, 14336),
    "1b": (2048, 32, 8, 8192),
}
EXPERTS, EXPERT_DIM, EXPERT_HIDDEN = 16, 5120, 8192
EPS, ROPE_BASE, ROPE_SCALE, ROPE_OLD = 1e-5, 500_000, 8, 8192
IGNORE, PAD = -100, 0
ADAPTED = ("q_proj", "v_proj", "output_proj")  # and the feed-forward block: the recipes' LoRA configurations, rank 8, alpha 16
RANK, ALPHA = 8, 16
DEV = "cuda"


def listed() -> List[Dict[str, Any]]:
    return [
        # Full fine-tuning, forward + loss + backward.  The benchmark's batch: 4 x 2048 packed tokens, activations recomputed in backward.
        dict(name="sft_8b_packed", kind="sft", model="8b", layers=2, batch=4, seq=2048, doc=512, recompute=True),
        # Long-context fine-tuning: one document of 16384 tokens; the largest case.
        dict(name="sft_8b_long", kind="sft", model="8b", layers=2, batch=1, seq=16384, doc=0, recompute=False),
        # The small model of the family, longer packed rows, 64 channels per head.
        dict(name="sft_1b_packed", kind="sft", model="1b", layers=2, batch=8, seq=2048, doc=700, recompute=False),
        # A small padded batch of an instruction data set (batch size 2, odd lengths): launches and small products count.
        dict(name="sft_1b_small", kind="sft", model="1b", layers=2, batch=2, seq=333, doc=0, recompute=False),
        # LoRA fine-tuning of a padded batch with an odd length, and QLoRA (4-bit base) of a short one.
        dict(name="lora_8b", kind="lora", model="8b", layers=2, batch=2, seq=1413, doc=0, nf4=False),
        dict(name="qlora_8b", kind="lora", model="8b", layers=2, batch=2, seq=512, doc=0, nf4=True),
        # Generation: one short chat turn of a whole 16-layer model, the smallest calls there are (batch 1, one token each).
        dict(name="chat_1b", kind="generate", model="1b", layers=16, batch=1, prompt=37, tokens=24),
        # Rollouts for preference and policy optimisation: 16 rows of one prompt length, sampled with the recipes' temperature and top-k.
        dict(name="rollout_8b", kind="generate", model="8b", layers=4, batch=16, prompt=700, tokens=32),
        # Long prompts (summaries, retrieval): the prefill dominates, decoding reads long caches.
        dict(name="long_prompt_8b", kind="generate", model="8b", layers=4, batch=2, prompt=8000, tokens=12),
        # Scoring of sampled responses under the reference model (the forward-only half of a GRPO / PPO step).
        dict(name="score_8b", kind="score", model="8b", layers=2, batch=8, seq=768, context=256),
        # One mixture-of-experts feed-forward block, forward + backward.
        dict(name="moe_scout", kind="moe", batch=2, seq=2048, top=1),
    ]


def _log(rng, low: int, high: int) -> int:
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng) -> Dict[str, Any]:
    kind = rng.choice(["sft", "sft", "lora", "generate", "generate", "score", "moe"])
    if kind == "sft":
        tokens = _log(rng, 300, 16384)
        seq = min(tokens, _log(rng, 128, 16384))
        doc = rng.choice([0, _log(rng, 48, max(64, seq))])
        return dict(kind=kind, model=rng.choice(["8b", "1b"]), layers=2, batch=max(1, tokens // seq), seq=seq, doc=doc, recompute=rng.random() < 0.5)
    if kind == "lora":
        tokens = _log(rng, 300, 6000)
        seq = min(tokens, _log(rng, 128, 4096))
        return dict(kind=kind, model=rng.choice(["8b", "1b"]), layers=2, batch=max(1, tokens // seq), seq=seq, doc=rng.choice([0, _log(rng, 48, max(64, seq))]), nf4=rng.random() < 0.4)
    if kind == "generate":
        model = rng.choice(["8b", "1b"])
        batch = _log(rng, 1, 48)
        prompt = _log(rng, 8, min(12000, 18000 // batch))
        return dict(kind=kind, model=model, layers=4 if model == "8b" else 16, batch=batch, prompt=prompt, tokens=rng.randint(8, 32))
    if kind == "score":
        seq = _log(rng, 64, 2048)
        batch = _log(rng, 1, max(1, min(16, 7000 // seq)))
        return dict(kind=kind, model=rng.choice(["8b", "1b"]), layers=2, batch=batch, seq=seq, context=rng.randint(8, seq // 2))
    tokens = _log(rng, 64, 6000)
    seq = min(tokens, _log(rng, 64, 4096))
    return dict(kind=kind, batch=max(1, tokens // seq), seq=seq, top=rng.choice([1, 1, 2]))


# ------------------------------------------------------------------------------------------------- weights and inputs
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(1000 + seed)


def _decoder_weights(case, seed: int) -> Dict[str, torch.Tensor]:
    """bf16 weights by name, from the seed alone.  Embeddings of unit scale, projections of the usual 0.02, those into the
    residual stream scaled by the depth.  For generation the output rows
    are embeddings in another order, so that one next token stands out as it does in a trained model."""
    g = _gen(seed)
    dim, heads, kv, hidden = WIDTHS[case["model"]]
    hd = dim // heads

    def normal(*shape, std=0.02):
        return torch.empty(*shape, dtype=torch.bfloat16, device=DEV).normal_(0, std, generator=g)

    w = {"tok_embeddings.weight": normal(VOCAB, dim, std=1.0)}
    for i in range(case["layers"]):
        shapes = {"attn.q_proj": (heads * hd, dim), "attn.k_proj": (kv * hd, dim), "attn.v_proj": (kv * hd, dim), "attn.output_proj": (dim, heads * hd),
                  "mlp.w1": (hidden, dim), "mlp.w2": (dim, hidden), "mlp.w3": (hidden, dim)}
        for name, shape in shapes.items():
            into = name in ("attn.output_proj", "mlp.w2")
            w[f"layers.{i}.{name}.weight"] = normal(*shape, std=0.02 / math.sqrt(case["layers"]) if into else 0.02)
            if case["kind"] == "lora" and (name.startswith("mlp.") or name.split(".")[1] in ADAPTED):
                w[f"layers.{i}.{name}.lora_a.weight"] = normal(RANK, shape[1], std=1.0 / math.sqrt(shape[1]))
                w[f"layers.{i}.{name}.lora_b.weight"] = normal(shape[0], RANK, std=0.01)
        for name in ("sa_norm", "mlp_norm"):
            w[f"layers.{i}.{name}.scale"] = 1 + normal(dim, std=0.1)
    w["norm.scale"] = 1 + normal(dim, std=0.1)
    if case["kind"] == "generate":
        order = torch.randperm(VOCAB, generator=g, device=DEV)
        w["output.weight"] = w["tok_embeddings.weight"][order] * 0.03
    else:
        w["output.weight"] = normal(VOCAB, dim)
    return w


def _lengths(case, seed: int) -> List[int]:
    """Real tokens of each row of a padded batch; the longest fills the row."""
    g = torch.Generator().manual_seed(5000 + seed)
    n = case["seq"]
    low = max(1, n // 3)
    rows = torch.randint(low, n + 1, (case["batch"],), generator=g).tolist()
    rows[0] = n
    return rows


def _documents(case, seed: int) -> List[List[int]]:
    """Document lengths of every packed row: around the mean, the last one cut by the end of the row."""
    g = torch.Generator().manual_seed(6000 + seed)
    rows = []
    for _ in range(case["batch"]):
        left, row = case["seq"], []
        while left > 0:
            n = min(left, max(1, int(case["doc"] * (0.5 + torch.rand(1, generator=g).item()))))
            row.append(n)
            left -= n
        rows.append(row)
    return rows


def _batch(case, seed: int) -> Tuple[torch.Tensor, torch.Tensor]:
    """Tokens and labels of a training batch: labels are the next tokens; padding, prompts' heads and document ends don't count."""
    g = _gen(seed + 77)
    b, s = case["batch"], case["seq"]
    tokens = torch.randint(1, VOCAB, (b, s), generator=g, device=DEV)
    labels = torch.roll(tokens, -1, 1)
    labels[:, -1] = IGNORE
    if case["doc"]:
        for r, row in enumerate(_documents(case, seed)):
            ends = torch.tensor(row).cumsum(0) - 1
            labels[r, ends.to(DEV)] = IGNORE
    else:
        for r, n in enumerate(_lengths(case, seed)):
            tokens[r, n:] = PAD
            labels[r, max(n - 1, 0) :] = IGNORE
            if n > 8:
                labels[r, : n // 8] = IGNORE
    return tokens, labels


def _prompts(case, seed: int) -> torch.Tensor:
    return torch.randint(1, VOCAB, (case["batch"], case["prompt"]), generator=_gen(seed + 77), device=DEV)


def _responses(case, seed: int) -> torch.Tensor:
    """Prompts padded on the left and responses padded on the right, as rollouts leave them."""
    b, s, ctx = case["batch"], case["seq"], case["context"]
    tokens = torch.randint(1, VOCAB, (b, s), generator=_gen(seed + 77), device=DEV)
    g = torch.Generator().manual_seed(7000 + seed)
    for r in range(1, b):
        tokens[r, : int(torch.randint(0, ctx, (1,), generator=g))] = PAD
        tokens[r, s - int(torch.randint(0, max(1, (s - ctx) // 2), (1,), generator=g)) :] = PAD
    return tokens


# ------------------------------------------------------------------------------------------------- the framework
def _build(case, seed: int, max_seq_len: int):
    from torchtune_b200 import training
    from torchtune_b200.models.llama3_1 import llama3_1, lora_llama3_1

    dim, heads, kv, hidden = WIDTHS[case["model"]]
    sizes = dict(vocab_size=VOCAB, num_layers=case["layers"], num_heads=heads, num_kv_heads=kv, embed_dim=dim, max_seq_len=max_seq_len, intermediate_dim=hidden,
                 norm_eps=EPS, rope_base=ROPE_BASE)
    with training.set_default_dtype(torch.bfloat16), torch.device(DEV):
        if case["kind"] == "lora":
            model = lora_llama3_1(list(ADAPTED), apply_lora_to_mlp=True, lora_rank=RANK, lora_alpha=ALPHA, quantize_base=case["nf4"], **sizes)
        else:
            model = llama3_1(**sizes)
    model.load_state_dict(_decoder_weights(case, seed))
    return model


def prepare(case, seed: int) -> Dict[str, Any]:
    from torchtune_b200 import training
    from torchtune_b200.modules import TransformerSelfAttentionLayer
    from torchtune_b200.modules.loss import LinearCrossEntropyLoss
    from torchtune_b200.ops import AttentionMask

    kind = case["kind"]
    if kind == "moe":
        return _prepare_experts(case, seed)
    if kind in ("sft", "lora"):
        model = _build(case, seed, max(8192, case["seq"]))
        if kind == "lora":
            from torchtune_b200.modules.peft import get_adapter_params, set_trainable_params

            set_trainable_params(model, get_adapter_params(model))
        elif case["recompute"]:
            training.set_activation_checkpointing(model, auto_wrap_policy={TransformerSelfAttentionLayer})
        loss = LinearCrossEntropyLoss()
        loss.set_model_output(model)
        tokens, labels = _batch(case, seed)
        mask = AttentionMask.from_seq_lens(_documents(case, seed)).to(DEV) if case["doc"] else None
        return {"kind": kind, "model": model.train(), "loss": loss, "tokens": tokens, "labels": labels, "mask": mask}
    if kind == "generate":
        model = _build(case, seed, max(8192, case["prompt"] + case["tokens"])).eval()
        with torch.device(DEV):
            model.setup_caches(batch_size=case["batch"], dtype=torch.bfloat16, decoder_max_seq_len=case["prompt"] + case["tokens"])
        return {"kind": kind, "model": model, "prompt": _prompts(case, seed), "tokens": case["tokens"], "seed": seed}
    tokens = _responses(case, seed)
    return {"kind": kind, "model": _build(case, seed, max(8192, case["seq"])).eval(), "tokens": tokens, "context": case["context"]}


def _expert_weights(case, seed: int) -> Tuple[Dict[str, torch.Tensor], torch.Tensor, torch.Tensor]:
    """Weights, input and upstream gradient of the expert block.  Tokens lean towards the gate rows of their experts, unevenly, as a
    trained router's do, so that which expert takes a token doesn't hang on rounding."""
    g = _gen(seed)

    def normal(*shape, std=0.02):
        return torch.empty(*shape, dtype=torch.bfloat16, device=DEV).normal_(0, std, generator=g)

    E, D, H = EXPERTS, EXPERT_DIM, EXPERT_HIDDEN
    w = {"experts.gate_proj": normal(E, D, H), "experts.up_proj": normal(E, D, H), "experts.down_proj": normal(E, H, D), "router.gate.weight": normal(E, D),
         "shared_expert.w1.weight": normal(H, D), "shared_expert.w2.weight": normal(D, H), "shared_expert.w3.weight": normal(H, D)}
    n = case["batch"] * case["seq"]
    load = 1.0 + torch.arange(E, device=DEV) % 4
    first = torch.multinomial(load, n, replacement=True, generator=g)
    second = (first + 1 + torch.randint(0, E - 1, (n,), generator=g, device=DEV)) % E
    gate = w["router.gate.weight"].float()
    x = torch.randn(n, D, generator=g, device=DEV)
    basis = torch.linalg.qr(gate.t()).Q
    lean = torch.randn(n, 2, generator=g, device=DEV)
    x = x - (x @ basis) @ basis.t() + (2.0 + 0.3 * lean[:, :1]) * gate[first] + (1.0 + 0.2 * lean[:, 1:]) * gate[second]
    x = x.to(torch.bfloat16)
    return w, x.view(case["batch"], case["seq"], D), normal(case["batch"], case["seq"], D, std=1.0)


def _prepare_experts(case, seed: int) -> Dict[str, Any]:
    from torchtune_b200 import training
    from torchtune_b200.models.llama4._component_builders import llama4_moe

    with training.set_default_dtype(torch.bfloat16), torch.device(DEV):
        block = llama4_moe(EXPERT_DIM, EXPERT_HIDDEN, num_experts=EXPERTS, experts_per_token=case["top"], use_shared_expert=True)
    w, x, dy = _expert_weights(case, seed)
    block.load_state_dict(w)
    return {"kind": "moe", "model": block.train(), "x": x.requires_grad_(), "dy": dy}


def run(state):
    from torchtune_b200 import generation, rlhf

    kind, model = state["kind"], state["model"]
    if kind in ("sft", "lora"):
        model.zero_grad(set_to_none=True)
        loss = state["loss"](model(state["tokens"], mask=state["mask"]), state["labels"])
        loss.backward()
        return {"loss": loss.detach(), "grads": {n: p.grad for n, p in model.named_parameters() if p.requires_grad}}
    if kind == "moe":
        model.zero_grad(set_to_none=True)
        state["x"].grad = None
        y = model(state["x"])
        y.backward(state["dy"])
        return {"y": y.detach(), "dx": state["x"].grad, "grads": {n: p.grad for n, p in model.named_parameters()}}
    if kind == "generate":
        model.reset_caches()
        rng = torch.Generator(device=DEV).manual_seed(state["seed"])
        tokens, logits = generation.generate(model, state["prompt"], max_generated_tokens=state["tokens"], pad_id=PAD, temperature=0.6, top_k=300, rng=rng)
        return {"tokens": tokens, "logits": logits}
    tokens, ctx = state["tokens"], state["context"]
    with torch.no_grad():
        real = tokens != PAD
        masks = generation.get_causal_mask_from_padding_mask(real)
        positions = generation.get_position_ids_from_padding_mask(real)
        logits = rlhf.truncate_sequence_for_logprobs(model(tokens, input_pos=positions, mask=masks), ctx)
        return {"logprobs": rlhf.logits_to_logprobs(logits, tokens[:, ctx:], 1.0)}


# ------------------------------------------------------------------------------------------------- what a pass cannot do without
def _layer_params(model: str) -> int:
    dim, heads, kv, hidden = WIDTHS[model]
    return dim * dim * 2 + 2 * dim * kv * (dim // heads) + 3 * dim * hidden


def _pairs(rows: List[List[int]]) -> int:
    return sum(n * (n + 1) // 2 for row in rows for n in row)


def work(case) -> Dict[str, float]:
    kind = case["kind"]
    if kind == "moe":
        n, per = case["batch"] * case["seq"], 3 * EXPERT_DIM * EXPERT_HIDDEN
        used = min(EXPERTS, n * case["top"])
        return {"flops": 6.0 * n * (case["top"] + 1) * per, "bytes": 2.0 * (2 * (used + 1) * per + 4 * n * EXPERT_DIM)}
    dim, heads, kv, _ = WIDTHS[case["model"]]
    layers, per, head = case["layers"], _layer_params(case["model"]), VOCAB * dim
    if kind == "generate":
        b, s, n = case["batch"], case["prompt"], case["tokens"]
        rows = [s] * b
        prompt = 2.0 * sum(rows) * layers * per + 4.0 * dim * layers * _pairs([rows])
        later = sum(2.0 * b * (layers * per + head) + 4.0 * dim * layers * (sum(rows) + b * t) for t in range(1, n)) + 2.0 * b * head
        cache = 2 * 2 * layers * kv * (dim // heads)  # bytes of one cached token
        read = 2.0 * n * (layers * per + head) + cache * sum(rows) + sum(cache * (sum(rows) + b * t) for t in range(1, n))
        return {"flops": prompt + later, "bytes": read + 4.0 * b * n * VOCAB}
    rows = _documents(case, 0) if case.get("doc") else [[n] for n in (_lengths(case, 0) if kind != "score" else [case["seq"]] * case["batch"])]
    n, pairs = sum(map(sum, rows)), _pairs(rows)
    if kind == "score":
        answers = case["batch"] * (case["seq"] - case["context"])
        return {"flops": 2.0 * n * layers * per + 2.0 * answers * head + 4.0 * dim * layers * pairs, "bytes": 2.0 * (layers * per + head) + 2.0 * n * dim}
    if kind == "lora":
        base = (0.5 + 2.0 / 64) if case["nf4"] else 2.0
        return {"flops": 4.0 * n * (layers * per + head) + 12.0 * dim * layers * pairs, "bytes": base * layers * per + 2.0 * head + 4.0 * n * dim}
    return {"flops": 6.0 * n * (layers * per + head) + 12.0 * dim * layers * pairs, "bytes": 4.0 * (layers * per + 2 * head) + 4.0 * n * dim}


def tolerance(case):
    # bf16 activations and gradients between fp32 sums: against exact() logits were 0.006 ... 0.012 off, log-probabilities 0.001 and gradients
    # 0.009 ... 0.016 (0.02 behind the experts)
    if case["kind"] == "generate":
        return {"rel": 0.03, "max": 0.5, "differ": 0.002}
    if case["kind"] == "score":
        return {"rel": 0.004, "max": 0.05}
    return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _norm(x: torch.Tensor, scale: torch.Tensor) -> torch.Tensor:
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * scale


def _angles(head_dim: int, count: int) -> torch.Tensor:
    """Rotation angles ``[count, head_dim / 2]`` with the published wavelength scaling of this family."""
    freq = ROPE_BASE ** -(torch.arange(0, head_dim, 2, dtype=torch.float64, device=DEV) / head_dim)
    wave = 2 * math.pi / freq
    blend = ((ROPE_OLD / wave - 1) / (4 - 1)).clamp(0, 1)
    return torch.arange(count, dtype=torch.float64, device=DEV)[:, None] * ((1 - blend) * freq / ROPE_SCALE + blend * freq)


def _rotate(x: torch.Tensor, ang: torch.Tensor) -> torch.Tensor:
    """``x`` ``[b, s, h, d]`` rotated by ``ang`` ``[b, s, d / 2]``, neighbouring channels as pairs."""
    c, s = ang.cos().unsqueeze(2), ang.sin().unsqueeze(2)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)


def _attend_piece(q, k, v, lo, hi, first: int):
    at = torch.arange(first, first + k.shape[0], device=q.device)
    seen = (at >= lo[:, None]) & (at <= hi[:, None])
    p = torch.softmax((torch.einsum("qhd,kd->hqk", q, k) / math.sqrt(q.shape[-1])).masked_fill(~seen, float("-inf")), -1)
    return torch.einsum("hqk,kd->qhd", p, v)


def _attend(q, k, v, lo, hi) -> torch.Tensor:
    """Grouped-query attention in which query i of row b sees keys lo[b, i] ... hi[b, i]; pieces small enough to hold their scores."""
    b, s, h, d = q.shape
    group = h // k.shape[2]
    step = max(1, (1 << 27) // max(1, group * k.shape[1]))
    rows = []
    for r in range(b):
        parts = []
        for i in range(0, s, step):
            j = min(s, i + step)
            first, last = int(lo[r, i:j].min()), int(hi[r, i:j].max()) + 1
            heads = []
            for n in range(k.shape[2]):
                args = (q[r, i:j, n * group : (n + 1) * group], k[r, first:last, n], v[r, first:last, n], lo[r, i:j], hi[r, i:j], first)
                heads.append(checkpoint(_attend_piece, *args, use_reentrant=False) if torch.is_grad_enabled() else _attend_piece(*args))
            parts.append(torch.cat(heads, 1))
        rows.append(torch.cat(parts))
    return torch.stack(rows)


def _linear(w, name: str, x):
    y = x @ w[f"{name}.weight"].double().t()
    if f"{name}.lora_a.weight" in w:
        y = y + (ALPHA / RANK) * (x @ w[f"{name}.lora_a.weight"].double().t()) @ w[f"{name}.lora_b.weight"].double().t()
    return y


def _layer(w, i: int, heads: int, kv: int, h, ang, lo, hi, cache):
    b, s, dim = h.shape
    hd = dim // heads
    x = _norm(h, w[f"layers.{i}.sa_norm.scale"].double())
    q = _rotate(_linear(w, f"layers.{i}.attn.q_proj", x).view(b, s, heads, hd), ang)
    k = _rotate(_linear(w, f"layers.{i}.attn.k_proj", x).view(b, s, kv, hd), ang)
    v = _linear(w, f"layers.{i}.attn.v_proj", x).view(b, s, kv, hd)
    if cache is not None:
        if i in cache:
            k, v = torch.cat([cache[i][0], k], 1), torch.cat([cache[i][1], v], 1)
        cache[i] = (k, v)
    h = h + _linear(w, f"layers.{i}.attn.output_proj", _attend(q, k, v, lo, hi).reshape(b, s, dim))
    x = _norm(h, w[f"layers.{i}.mlp_norm.scale"].double())
    gate = torch.nn.functional.silu(_linear(w, f"layers.{i}.mlp.w1", x)) * _linear(w, f"layers.{i}.mlp.w3", x)
    return h + _linear(w, f"layers.{i}.mlp.w2", gate)


def _hidden(case, w, tokens, pos, lo, hi, cache: Optional[dict] = None):
    dim, heads, kv, _ = WIDTHS[case["model"]]
    h = torch.nn.functional.embedding(tokens, w["tok_embeddings.weight"]).double()
    ang = _angles(dim // heads, int(pos.max()) + 1)[pos]
    for i in range(case["layers"]):
        if torch.is_grad_enabled():
            h = checkpoint(_layer, w, i, heads, kv, h, ang, lo, hi, None, use_reentrant=False)
        else:
            h = _layer(w, i, heads, kv, h, ang, lo, hi, cache)
    return _norm(h, w["norm.scale"].double())


def _loss_piece(h, out, labels):
    return torch.nn.functional.cross_entropy(h @ out.double().t(), labels, ignore_index=IGNORE, reduction="sum")


def _nf4(w: torch.Tensor) -> torch.Tensor:
    """The values a 4-bit NormalFloat copy of ``w`` stands for (blocks of 64, scales in 8 bits around their mean by groups of 256)."""
    half = torch.special.ndtri(torch.linspace(0.9677083, 0.5, 9, dtype=torch.float64, device=DEV)[:-1])
    other = -torch.special.ndtri(torch.linspace(0.9677083, 0.5, 8, dtype=torch.float64, device=DEV)[:-1])
    code = torch.cat([half, other, torch.zeros(1, dtype=torch.float64, device=DEV)]).sort().values
    code = code / code.max()
    blocks = w.double().reshape(-1, 64)
    top = blocks.abs().amax(1)
    centred = (top - top.mean()).view(-1, 256)
    factor = 127.0 / centred.abs().amax(1, keepdim=True).clamp_min(1e-30)
    scale = ((centred * factor).round().clamp(-128, 127) / factor).view(-1, 1) + top.mean()
    edges = (code[1:] + code[:-1]) / 2
    return (code[torch.bucketize((blocks / scale.clamp_min(1e-30)).clamp(-1, 1), edges)] * scale).view(w.shape)


def _exact_train(case, seed: int):
    w = _decoder_weights(case, seed)
    lora = case["kind"] == "lora"
    for name in w:
        if lora and case["nf4"] and name.startswith("layers.") and w[name].dim() == 2 and "lora" not in name:
            w[name] = _nf4(w[name])
        elif not lora or "lora" in name:
            w[name] = w[name].double().requires_grad_()
    tokens, labels = _batch(case, seed)
    b, s = tokens.shape
    pos = torch.arange(s, device=DEV).expand(b, s)
    lo = torch.zeros_like(pos)
    if case["doc"]:
        lo = torch.stack([torch.repeat_interleave(torch.tensor(row).cumsum(0) - torch.tensor(row), torch.tensor(row)) for row in _documents(case, seed)]).to(DEV)
    h = _hidden(case, w, tokens, pos, lo, pos).view(b * s, -1)
    y = labels.reshape(-1)
    total = sum(checkpoint(_loss_piece, h[i : i + 2048], w["output.weight"], y[i : i + 2048], use_reentrant=False) for i in range(0, b * s, 2048))
    loss = total / (y != IGNORE).sum().clamp_min(1)
    loss.backward()
    return {"loss": loss.detach(), "grads": {n: t.grad for n, t in w.items() if t.requires_grad}}


@torch.no_grad()
def _exact_generate(case, seed: int):
    w, prompt = _decoder_weights(case, seed), _prompts(case, seed)
    b, s = prompt.shape
    pos, cache, out, steps, x = torch.arange(s, device=DEV).expand(b, s), {}, prompt, [], prompt
    rng = torch.Generator(device=DEV).manual_seed(seed)
    for t in range(case["tokens"]):
        logits = _hidden(case, w, x, pos, torch.zeros_like(pos), pos, cache)[:, -1] @ w["output.weight"].double().t()
        steps.append(logits)
        u = torch.rand((b, VOCAB), generator=rng, device=DEV)
        q = -torch.log((1.0 - u).clamp(min=torch.finfo(u.dtype).eps / 2))
        warm = logits / 0.6
        warm = warm.masked_fill(warm < warm.topk(300).values[:, -1:], float("-inf"))
        p = torch.softmax(warm, -1)
        x = torch.where(p > 0, p / q, 0.0).argmax(-1, keepdim=True).int()
        out = torch.cat([out, x], 1)
        pos = torch.full((b, 1), s + t, device=DEV)
    return {"tokens": out, "logits": torch.stack(steps, 1)}


@torch.no_grad()
def _exact_score(case, seed: int):
    w, tokens = _decoder_weights(case, seed), _responses(case, seed)
    b, s = tokens.shape
    real, slot = tokens != PAD, torch.arange(s, device=DEV).expand(b, s)
    start = real.int().argmax(1, keepdim=True)
    # a padded query sees the real keys before it and itself; on the left that is itself alone, on the right they end with the response
    length = s - real.flip(1).int().argmax(1, keepdim=True)
    pos = (real.cumsum(1) - 1) * real
    h = _hidden_right_padded(case, w, tokens, pos, torch.where(slot < start, slot, start.expand(b, s)), slot, length)
    ctx, rows = case["context"], []
    for r in range(b):
        logits = h[r, ctx - 1 : -1] @ w["output.weight"].double().t()
        rows.append(torch.log_softmax(logits, -1).gather(-1, tokens[r, ctx:, None]).squeeze(-1))
    return {"logprobs": torch.stack(rows)}


def _hidden_right_padded(case, w, tokens, pos, lo, hi, length):
    """Hidden states where padding follows the response: the padded queries are run row by row behind the others, on the real keys and
    their own."""
    dim, heads, kv, _ = WIDTHS[case["model"]]
    rows = []
    for r in range(tokens.shape[0]):
        n, cache = int(length[r]), {}
        h = _hidden(case, w, tokens[r : r + 1, :n], pos[r : r + 1, :n], lo[r : r + 1, :n], hi[r : r + 1, :n], cache)
        if n < tokens.shape[1]:  # all padded queries hold the same token at position 0 and see the same keys: one stands for all
            first = lo[r : r + 1, n - 1 : n]
            pad = _hidden(case, w, tokens[r : r + 1, n : n + 1], pos[r : r + 1, n : n + 1], first, hi[r : r + 1, n : n + 1], cache)
            h = torch.cat([h, pad.expand(1, tokens.shape[1] - n, dim)], 1)
        rows.append(h)
    return torch.cat(rows)


def _exact_experts(case, seed: int):
    w, x, dy = _expert_weights(case, seed)
    silu = torch.nn.functional.silu
    flat, dflat = x.double().view(-1, EXPERT_DIM).requires_grad_(), dy.double().view(-1, EXPERT_DIM)
    n, E = flat.shape[0], EXPERTS
    gate = w["router.gate.weight"].double().requires_grad_()
    scores = torch.sigmoid(flat @ gate.t())
    top, chosen = scores.topk(case["top"], 1)
    used = {k: [None] * E for k in ("experts.gate_proj", "experts.up_proj", "experts.down_proj")}
    shared = {k: w[k].double().requires_grad_() for k in ("shared_expert.w1.weight", "shared_expert.w2.weight", "shared_expert.w3.weight")}
    y = (silu(flat @ shared["shared_expert.w1.weight"].t()) * (flat @ shared["shared_expert.w3.weight"].t())) @ shared["shared_expert.w2.weight"].t()
    for e in range(E):
        token, place = (chosen == e).nonzero(as_tuple=True)
        leaf = {k: w[k][e].double().requires_grad_() for k in used}
        xe = flat[token] * top[token, place][:, None]
        ye = (silu(xe @ leaf["experts.gate_proj"]) * (xe @ leaf["experts.up_proj"])) @ leaf["experts.down_proj"]
        y = y.index_add(0, token, ye)
        for k in used:
            used[k][e] = leaf[k]
    y.backward(dflat)
    grads = {"router.gate.weight": gate.grad, **{k: t.grad for k, t in shared.items()}}
    for k, ts in used.items():
        grads[k] = torch.stack([t.grad if t.grad is not None else torch.zeros_like(t) for t in ts])
    shape = x.shape
    return {"y": y.detach().view(shape), "dx": flat.grad.view(shape), "grads": grads}


def exact(case, seed: int):
    return {"sft": _exact_train, "lora": _exact_train, "generate": _exact_generate, "score": _exact_score, "moe": _exact_experts}[case["kind"]](case, seed)
