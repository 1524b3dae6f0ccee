"""All layers of a decoder issued by one native call: bit for bit what the modules give."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu


def _model(layers, dim, heads, kv, hidden, vocab, rows, slots, bias=False):
    from torchtune_b200 import training
    from torchtune_b200.models.llama3_1 import llama3_1
    from torchtune_b200.modules.linear import Linear

    torch.manual_seed(dim + hidden)
    with training.set_default_dtype(torch.bfloat16), torch.device("cuda"):
        model = llama3_1(vocab_size=vocab, num_layers=layers, num_heads=heads, num_kv_heads=kv, embed_dim=dim, max_seq_len=8192, intermediate_dim=hidden).eval()
        if bias:
            for layer in model.layers:
                for name in ("q_proj", "k_proj", "v_proj"):
                    old = getattr(layer.attn, name)
                    setattr(layer.attn, name, Linear(old.in_features, old.out_features, bias=True))
        model.setup_caches(batch_size=rows, dtype=torch.bfloat16, decoder_max_seq_len=slots)
    return model


SHAPES = [  # layers, dim, heads, key heads, hidden, rows, slots, tokens
    (2, 512, 8, 2, 1024, 3, 60, 1),  # kernels for few tokens
    (2, 1024, 16, 1, 1024, 5, 1030, 1),  # one token: 16 query heads to a key head, ranges of keys
    (1, 1024, 8, 4, 512, 9, 65, 1),  # head dimension 128
    (2, 2048, 32, 8, 8192, 1, 61, 37),  # gate and up projection apart, the rest for few tokens
    (1, 1024, 8, 8, 4096, 2, 300, 4),  # several queries on the kernel for few queries
    (1, 1024, 8, 8, 4096, 2, 300, 200),  # contraction in ranges, residual by itself
    (1, 4096, 32, 8, 14336, 1, 700, 640),  # CTA pairs, alone and with ranges
    (1, 2048, 32, 8, 8192, 3, 1100, 1030),  # CTA pairs throughout, ragged
    (1, 192, 3, 3, 264, 5, 40, 33),
]


@pytest.mark.parametrize("padded,bias,start", [(False, False, 0), (True, True, 0), (True, False, 5)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@torch.no_grad()
def test_results_and_caches_are_those_of_the_modules(shape, padded, bias, start):
    from torchtune_b200 import generation
    from torchtune_b200.generation._native_layers import NativeLayers
    from torchtune_b200.generation._rows import hidden_states

    layers, dim, heads, kv, hidden, rows, slots, n = shape
    model = _model(layers, dim, heads, kv, hidden, 1024, rows, slots, bias)
    native = NativeLayers.of(model, rows)
    assert native is not None
    x = torch.randint(1, 1024, (rows, n), device="cuda")

    def restart():  # caches that hold `start` tokens
        model.reset_caches()
        for i, layer in enumerate(model.layers):
            cache = layer.attn.kv_cache
            g = torch.Generator(device="cuda").manual_seed(i)
            cache.k_cache[:, :start].normal_(generator=g), cache.v_cache[:, :start].normal_(generator=g)
            cache.cache_pos.add_(start)
            layer.attn.pos_embeddings.interleaved = start == 0

    restart()
    native = NativeLayers.of(model, rows)
    if padded:
        real = torch.ones(rows, n, dtype=torch.bool, device="cuda")
        for r in range(1, rows):
            real[r, : min(n - 1, 3 * r)] = False
        real = torch.nn.functional.pad(real, (start, 0), value=True)
        mask, pos = generation.get_causal_mask_from_padding_mask(real, target_seq_len=slots)[:, start:], generation.get_position_ids_from_padding_mask(real)[:, start:]
    else:
        mask, pos = torch.tril(torch.ones(n + 2, slots, dtype=torch.bool, device="cuda")).unsqueeze(0)[:, :n], torch.arange(n, device="cuda")
    got = native(x, pos, mask)
    caches = [(l.attn.kv_cache.k_cache.clone(), l.attn.kv_cache.v_cache.clone(), l.attn.kv_cache.cache_pos.clone()) for l in model.layers]
    restart()
    want = hidden_states(model, x, input_pos=pos, mask=mask)
    assert torch.equal(got, want)
    for l, (k, v, at) in zip(model.layers, caches):
        assert torch.equal(l.attn.kv_cache.k_cache, k) and torch.equal(l.attn.kv_cache.v_cache, v) and torch.equal(l.attn.kv_cache.cache_pos, at)
    with pytest.raises(AssertionError, match="full"):
        more = slots - n - start + 1
        native(x[:, :1].repeat(1, more), torch.arange(more, device="cuda"), torch.ones(1, more, slots, dtype=torch.bool, device="cuda"))


@torch.no_grad()
def test_what_the_call_does_not_do_is_left_to_the_modules(monkeypatch):
    from torchtune_b200.generation._native_layers import NativeLayers

    for change in (lambda m: setattr(m.layers[1].mlp_norm, "eps", 1e-6), lambda m: setattr(m.layers[0].attn, "softcap", 50.0), lambda m: setattr(m.layers[1].mlp, "activation", nn.GELU()),
                   lambda m: setattr(m.layers[0].attn, "q_proj", nn.Linear(512, 512, bias=False, dtype=torch.bfloat16, device="cuda")), lambda m: setattr(m.layers[0].attn, "scale", -1.0),
                   lambda m: m.layers[1].attn.q_proj.register_forward_hook(lambda *a: None), lambda m: setattr(m.layers[0], "sa_scale", nn.Tanh()), lambda m: setattr(m.layers[0].mlp, "w3", None),
                   lambda m: setattr(m.layers[1].attn.kv_cache, "k_cache", m.layers[1].attn.kv_cache.k_cache.float()), lambda m: setattr(m.layers[1].attn.pos_embeddings, "interleaved", False)):
        model = _model(2, 512, 8, 2, 1024, 1024, 4, 60)
        assert NativeLayers.of(model, 4) is not None and NativeLayers.of(model, 5) is None
        model.layers[0].attn.pos_embeddings = type(model.layers[0].attn.pos_embeddings)(dim=64, max_seq_len=8192).to("cuda")  # layers share one module
        change(model)
        assert NativeLayers.of(model, 4) is None
    model = _model(2, 512, 8, 2, 1024, 1024, 4, 60)
    for name in ("TTB_FUSE_RESIDUAL", "TTB_FUSE_SWIGLU"):
        with monkeypatch.context() as m:
            m.setenv(name, "0")
            assert NativeLayers.of(model, 4) is None
    native = NativeLayers.of(model, 4)
    x, pos, mask = torch.ones(4, 2, dtype=torch.int64, device="cuda"), torch.arange(2, device="cuda"), torch.ones(1, 2, 60, dtype=torch.bool, device="cuda")
    assert native(x[:3], pos, mask) is None and native(x, pos, mask[:, :, :59]) is None and native(x, pos, mask.float()) is None
    assert int(model.layers[0].attn.kv_cache.cache_pos[0]) == 0 and native(x, pos, mask) is not None


@pytest.mark.parametrize("how", ["context", "default"])
def test_generation_where_tensors_are_made_on_the_device(how):
    """Inside a device context and with a default device: tokens and logits of a plain call, recorded steps included."""
    from torchtune_b200 import generation
    from torchtune_b200.generation._native_layers import NativeLayers

    model = _model(2, 512, 8, 2, 1024, 1024, 3, 60)
    prompt = torch.randint(1, 1024, (3, 9), device="cuda")
    prompt[0, :4] = 0

    def run():
        model.reset_caches()
        return generation.generate(model, prompt, max_generated_tokens=8, temperature=0.7, top_k=20, rng=torch.Generator(device="cuda").manual_seed(1))

    want = run()
    if how == "context":
        with torch.device("cuda"):
            assert NativeLayers.of(model, 3) is not None
            got = run()
    else:
        torch.set_default_device("cuda")
        try:
            got = run()
        finally:
            torch.set_default_device(None)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@torch.no_grad()
@pytest.mark.parametrize("first", [False, True])
def test_a_step_is_recorded_once_its_own_kernels_have_run(first):
    """Caches that were stepped by the modules, then by the native call, and the other way round: the first step of either way runs as it is."""
    from torchtune_b200.generation._native_layers import NativeLayers
    from torchtune_b200.generation._step_graph import StepGraph, _alone

    model = _model(1, 512, 8, 2, 1024, 1024, 2, 60)
    x, mask = torch.randint(1, 1024, (2, 1), device="cuda"), torch.tril(torch.ones(60, 60, dtype=torch.bool, device="cuda")).unsqueeze(0)
    at = 0
    for native in (first, not first):
        step = StepGraph(model, 2, NativeLayers.of(model, 2) if native else None)
        for recorded in (False, _alone()):
            step(x, torch.full((2,), at, device="cuda"), mask[:, at : at + 1].contiguous())
            at += 1
            assert (step.graph is not None) == recorded


@pytest.mark.parametrize("M,N,Ks", [(40, 64, (64, 24)), (300, 520, (512, 128, 128)), (8200, 1032, (1024, 136, 264)), (4100, 2048, (2048, 512, 512)), (700, 2048, (8192, 4096)), (9000, 520, (200, 8192))])
def test_linear_layers_of_one_input(M, N, Ks):
    """Values of joined layers are those of single ones; the input gradient, summed by its products, against 64 bits; outputs that nobody uses, frozen weights, biases."""
    from torchtune_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    x, ws, bs = rand(2, M // 2, N).requires_grad_(), [(rand(K, N) * N**-0.5).requires_grad_() for K in Ks], [rand(K).requires_grad_() if i != 1 else None for i, K in enumerate(Ks)]
    ws[-1].requires_grad_(False)
    assert ops.joins_gradients(x)
    ys = ops.linear_group(x, ws, bs)
    dys = [rand(*y.shape) for y in ys]
    single = [ops.linear(x, w, b) for w, b in zip(ws, bs)]
    assert all(torch.equal(a, b) for a, b in zip(ys, single))
    leaves = [x, *ws[:-1], *(b for b in bs if b is not None)]
    got = torch.autograd.grad(ys, leaves, dys)
    want = torch.autograd.grad(single, leaves, dys)
    assert all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
    terms = [d.view(-1, d.shape[-1]).double() @ w.double() for d, w in zip(dys, ws)]
    exact = sum(terms).view_as(x)
    # a rounding to bf16 errs by at most 2^-8 of what it rounds: the result, and for each further product the sum so far or the product
    bound = 2.0**-8 * (exact.abs() + sum(t.abs() for t in terms).view_as(x) * (len(Ks) - 1)) + 1e-4
    assert ((got[0].double() - exact).abs() <= bound).all()
    assert float((got[0].double() - exact).norm()) <= 1.02 * float((want[0].double() - exact).norm())
    first = torch.autograd.grad(ops.linear_group(x, ws, bs)[0], x, dys[0])[0]
    assert torch.equal(first, torch.autograd.grad(ops.linear(x, ws[0], bs[0]), x, dys[0])[0])
    with torch.no_grad():
        assert all(torch.equal(a, b) for a, b in zip(ops.linear_group(x, ws, bs), [ops.linear(x, w, b) for w, b in zip(ws, bs)]))


@pytest.mark.parametrize("rows,D", [(1, 8), (9, 264), (592, 1024), (3001, 4096), (31, 2056)])
def test_gain_gradient(rows, D):
    from torchtune_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows)
    x, dy = (torch.randn(rows, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    gain = torch.ones(D, device="cuda", dtype=torch.bfloat16).requires_grad_()
    got, = torch.autograd.grad(ops.rms_norm(x, gain, 1e-5), gain, dy)
    terms = dy.double() * x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5)
    assert ((got.double() - terms.sum(0)).abs() <= 2.0**-8 * terms.sum(0).abs() + 2.0**-18 * terms.abs().sum(0)).all()  # one rounding, fp32 sums


@pytest.mark.parametrize("n,dim,run", [(1, 8, 1), (7, 64, 7), (8, 264, 8), (9, 2056, 9), (666, 2048, 300), (5000, 128, 4097)])
def test_embedding_gradient_of_long_runs(n, dim, run):
    """One id for `run` tokens, the end of a run inside and on a group of eight: sums in the order of the tokens."""
    from torchtune_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(n)
    ids = torch.randint(0, 50, (n,), generator=g, device="cuda")
    ids[torch.randperm(n, generator=g, device="cuda")[:run]] = 3
    table = torch.zeros(64, dim, device="cuda", dtype=torch.bfloat16).requires_grad_()
    dy = torch.randn(n, dim, generator=g, device="cuda").to(torch.bfloat16)
    got, = torch.autograd.grad(ops.embedding(ids, table), table, dy)
    want, size = (torch.zeros(64, dim, device="cuda", dtype=torch.float64).index_add_(0, ids, t) for t in (dy.double(), dy.double().abs()))
    assert ((got.double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-23 * run * size).all()  # one rounding, fp32 sums one after the other


@pytest.mark.parametrize("b,s,hq,hkv,D", [(1, 1, 1, 1, 64), (3, 7, 3, 1, 128), (2, 333, 32, 8, 64), (1, 129, 20, 4, 128), (1, 9, 1600, 1600, 64), (1, 333, 3, 1, 128), (2, 601, 4, 2, 64), (1, 3, 12400, 12400, 64)])
def test_attention_gradient_of_ragged_tokens(b, s, hq, hkv, D):
    """The products of outputs and their gradients, one to eight tokens at a time, where tokens and heads fill no group, and for more heads than are staged."""
    from torchtune_b200 import ops
    from torchtune_b200.ops import AttentionMask

    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(b, s, h, D, generator=g, device="cuda").to(torch.bfloat16).requires_grad_() for h in (hq, hkv, hkv))
    dy = torch.randn(b, s, hq, D, generator=g, device="cuda").to(torch.bfloat16)
    got = torch.autograd.grad(ops.attention(q, k, v, AttentionMask(causal=True)), (q, k, v), dy)
    leaves = [t.detach().double().requires_grad_() for t in (q, k, v)]
    kk, vv = (t.repeat_interleave(hq // hkv, 2) for t in leaves[1:])
    scores = torch.einsum("bqhd,bkhd->bhqk", leaves[0], kk) * D**-0.5
    p = torch.softmax(scores.masked_fill(~torch.ones(s, s, dtype=torch.bool, device="cuda").tril(), float("-inf")), -1)
    want = torch.autograd.grad(torch.einsum("bhqk,bkhd->bqhd", p, vv), leaves, dy.double())
    for a, e in zip(got, want):
        assert float((a.double() - e).norm()) <= 0.01 * float(e.norm()) + 1e-3  # probabilities and their gradients are rounded to bf16 once each


def test_attention_gradient_of_a_saved_output_at_an_odd_address():
    """A hook on saved tensors hands the output back where 16-byte loads can't read it: the same gradients."""
    from torchtune_b200 import ops
    from torchtune_b200.ops import AttentionMask

    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, dy = (torch.randn(2, 77, h, 64, generator=g, device="cuda").to(torch.bfloat16) for h in (8, 2, 2, 8))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    want = torch.autograd.grad(ops.attention(q, k, v, AttentionMask(causal=True)), leaves, dy)
    moved = []

    def unpack(t):
        if t.dtype != torch.bfloat16 or t.shape != q.shape or torch.equal(t, q):
            return t
        moved.append(torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t))
        return moved[-1]

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        y = ops.attention(q, k, v, AttentionMask(causal=True))
    got = torch.autograd.grad(y, leaves, dy)
    assert len(moved) == 1 and moved[0].data_ptr() % 16 and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("b,hq,hkv,D,slots", [(1, 4, 1, 64, 40), (3, 8, 2, 128, 700)])
@pytest.mark.parametrize("interleaved", [0, 1])
def test_decode_step_with_indices_out_of_range(b, hq, hkv, D, slots, interleaved):
    """Positions outside the table count as position 0 and are noted; a slot outside the cache is not written.  Caches lie between guards."""
    from torchtune_b200.ops._lib import check, index_violations, lib, stream_ptr

    g = torch.Generator(device="cuda").manual_seed(slots)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    q, k, v, size, table_len = rand(b, hq, D), rand(b, hkv, D), rand(b, hkv, D), b * slots * hkv * D, 50
    angles = torch.rand(table_len, D // 2, generator=g, device="cuda")
    table, mask = torch.stack([angles.cos(), angles.sin()], -1).contiguous(), torch.ones(slots, dtype=torch.bool, device="cuda")
    guarded = [rand(size + 2 * 4096) for _ in range(2)]

    def step(pos, slot):
        buffers, o = [t.clone() for t in guarded], torch.empty_like(q)
        at, to = torch.tensor(pos[:b], dtype=torch.int32, device="cuda"), torch.tensor([slot], device="cuda")
        caches = [t[4096 : 4096 + size] for t in buffers]
        check(lib().ttb_attn_decode_append(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), caches[0].data_ptr(), caches[1].data_ptr(), table.data_ptr(), at.data_ptr(),
                                           to.data_ptr(), mask.data_ptr(), 0, b, slots, hq, hkv, D, interleaved, table_len, D**-0.5, stream_ptr()), "step")
        return o, buffers

    index_violations()
    want, kept = step([0, 0, 0], slots - 1)
    assert index_violations() == 0 and not torch.equal(kept[0], guarded[0]) and not torch.equal(kept[1], guarded[1])
    got, buffers = step([-1, table_len, 2**31 - 1], slots - 1)
    assert index_violations() == b and torch.equal(got, want) and all(torch.equal(x, y) for x, y in zip(buffers, kept))
    for slot in (slots, -1, 2**40):
        got, buffers = step([3, 1, 2], slot)
        assert index_violations() == 0 and got.isfinite().all() and all(torch.equal(x, y) for x, y in zip(buffers, guarded))
