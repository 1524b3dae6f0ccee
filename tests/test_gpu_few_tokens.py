"""Linear layers of a few tokens, and sampling, against plain statements in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from torchtune_b200 import ops


def _rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(torch.bfloat16)


def _check(got, want, x, w, extra=0.0):
    # one rounding to bf16 (2^-9 of the value, twice that for ties and the bias), and fp32 sums of K terms in any order
    bound = 2.0**-8 * (want.abs() + extra) + 2.0**-19 * (x.double().abs() @ w.double().abs().t())
    assert got.shape == want.shape and ((got.double() - want).abs() <= bound).all(), float(((got.double() - want).abs() - bound).max())


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(8, 8), (40, 136), (512, 2048), (1000, 1032), (4096, 1024), (20000, 264)])
def test_products(M, N, K):
    """Edges of the token tiles, rows and contractions that end inside a tile, one to eight CTAs per tile; pitched operands and outputs."""
    from torchtune_b200.ops._cuda import _gemm_rows, gemm

    x = _rand(M, K + 16, seed=M)[:, 8 : K + 8]
    w = _rand(N, K + 8, seed=N)[:, :K]
    bias = _rand(N, seed=3)
    want = x.double() @ w.double().t()
    _check(gemm(x, w), want, x, w)
    _check(gemm(x, w, bias=bias, alpha=0.5), 0.5 * want + bias.double(), x, w, 1.0)
    out = torch.full((M, N + 24), float("nan"), dtype=torch.float32, device="cuda")
    _gemm_rows(x, [w], [out[:, :N]])
    assert ((out[:, :N].double() - want).abs() <= 2.0**-19 * (x.double().abs() @ w.double().abs().t())).all() and out[:, N:].isnan().all()


@pytest.mark.parametrize("M", [1, 16, 40, 64])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 264), (8192, 2048), (1032, 14336)])
def test_residual_gate_and_groups(M, N, K):
    from torchtune_b200.ops._cuda import _gemm_rows, gate_up_swiglu

    x, w, w3 = _rand(M, K, seed=1), _rand(N, K, seed=2), _rand(N, K, seed=3)
    r = _rand(M, N, seed=4)
    a, b = x.double() @ w.double().t(), x.double() @ w3.double().t()
    with torch.no_grad():
        y = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        _gemm_rows(x, [w], [y], residual=r)
        _check(y, a + r.double(), x, w)
        _check(ops.linear_residual(x, w, None, r), a + r.double(), x, w, a.abs())  # other kernels round the product first
        x, scale = x / K**0.5, K**-0.5
        a, b = (x.double() @ t.double().t() for t in (w, w3))
        for clamp in (None, (0.7, 1.702)):
            got = gate_up_swiglu(x, w, w3, clamp)
            if got is None:  # left to the separate operators
                assert M > 32 and N > 4096
                continue
            got = got.double()
            ca, cb = (a, b) if clamp is None else (a.clamp(max=clamp[0]), b.clamp(-clamp[0], clamp[0]) + 1)
            want = ca * torch.sigmoid(ca * (1.0 if clamp is None else clamp[1])) * cb
            # both pre-activations are rounded to bf16 first: 2^-8 of each, with |gate'| <= 1.1, then the result once more
            bound = 2.0**-8 * (want.abs() + 1.2 * a.abs() * cb.abs() + ca.abs() * b.abs()) + 1e-4
            assert ((got - want).abs() <= bound).all()
        ws = [w, w3[: max(8, N // 4)], w3]
        bias = _rand(N, seed=5)
        for got, wi, bi in zip(ops.linear_group(x, ws, [None, None, bias]), ws, (None, None, bias)):
            _check(got, x.double() @ wi.double().t() + (0 if bi is None else bi.double()), x, wi, 0 if bi is None else bi.double().abs())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V,top_k", [(1, 1), (7, 3), (4099, 50), (128256, 300), (128256, 128255), (128256, 0), (400000, 20)])
def test_sampling(V, top_k, dtype):
    """Rows shorter than their eight parts, parts that don't fit shared memory, ties at the threshold, infinities."""
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = (torch.randn(3, V, generator=g, device="cuda") * 3).to(dtype)
    if V > 8:
        logits[1] = logits[1].round()  # many ties
        logits[2, : V // 2] = float("-inf")
    q = -torch.log(torch.rand(3, V, generator=g, device="cuda").clamp_min(1e-7)) + 1e-7
    got = ops.sample_tokens(logits, q, 0.6, top_k or None)
    t = (logits / 0.6).float()
    if 0 < top_k < V:
        t = torch.where(t < torch.topk(t, top_k).values[:, -1:], float("-inf"), t)
    race = t.double() - q.double().log()
    picked = race.gather(1, got.long())
    # logarithms and one subtraction in fp32: a few units of 2^-21 at logits below 32
    assert (picked >= race.amax(1, keepdim=True) - 1e-5).all()


@pytest.mark.parametrize("interleaved", [True, False])
@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 1, 4, 4, 64), (3, 5, 8, 2, 128), (2, 70, 32, 8, 64), (2, 3, 3, 1, 16)])
def test_rotation_into_a_cache(b, s, hq, hkv, d, interleaved):
    """The same bits as two rotations and two copies, and not a byte of the cache beside the named slots."""
    q, k, v = _rand(b, s, hq, d, seed=1), _rand(b, s, hkv, d, seed=2), _rand(b, s, hkv, d, seed=3)
    ang = torch.rand(97, d // 2, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda") * 6
    table = torch.stack([ang.cos(), ang.sin()], -1)
    kc, vc = _rand(b, s + 9, hkv, d, seed=5), _rand(b, s + 9, hkv, d, seed=6)
    want_k, want_v = kc.clone(), vc.clone()
    slots = torch.arange(4, 4 + s, device="cuda")
    for pos in (None, torch.arange(s, device="cuda") + 20, torch.randint(0, 97, (b, s), device="cuda")):
        want_k[:, 4 : 4 + s], want_v[:, 4 : 4 + s] = ops.rope(k, table, pos, interleaved), v
        with torch.no_grad():
            got = ops.rope_append(q, k, v, table, pos, interleaved, kc, vc, slots)
        assert torch.equal(got, ops.rope(q, table, pos, interleaved)) and torch.equal(kc, want_k) and torch.equal(vc, want_v)


def test_recorded_steps_are_the_plain_ones():
    """Generation with recorded steps, on used and on fresh caches, against a loop of plain calls; full caches are still refused."""
    import copy

    from torchtune_b200 import generation, training
    from torchtune_b200.generation._step_graph import StepGraph
    from torchtune_b200.models.llama3_1 import llama3_1

    torch.manual_seed(0)
    with training.set_default_dtype(torch.bfloat16), torch.device("cuda"):
        model = llama3_1(vocab_size=1024, num_layers=3, num_heads=8, num_kv_heads=2, embed_dim=512, max_seq_len=512, intermediate_dim=1024).eval()
        model.setup_caches(batch_size=3, dtype=torch.bfloat16, decoder_max_seq_len=60)

    def run(prompt, n, **kw):
        model.reset_caches()
        rng = torch.Generator(device="cuda").manual_seed(1)
        return generation.generate(model, prompt, max_generated_tokens=n, temperature=0.8, top_k=50, rng=rng, **kw)

    for b, s, n in ((3, 20, 12), (1, 7, 40), (3, 48, 12), (2, 30, 4)):
        prompt = torch.randint(1, 1024, (b, s), device="cuda")
        assert StepGraph.suits(model, prompt)
        tokens, logits = run(prompt, n)
        plain_tokens, plain_logits = run(prompt, n, custom_generate_next_token=generation.generate_next_token)
        assert torch.equal(tokens, plain_tokens) and torch.equal(logits, plain_logits)
        assert model.layers[1].attn.kv_cache.size == s + n - 1 and int(model.layers[1].attn.kv_cache.cache_pos[0]) == s + n - 1
        again, _ = run(prompt, n)
        assert torch.equal(again, tokens)
    copy.deepcopy(model)
    with pytest.raises(AssertionError, match="full"):
        run(torch.randint(1, 1024, (2, 55), device="cuda"), 8)
    model.layers[0].register_forward_hook(lambda *a: None)
    assert not StepGraph.suits(model, prompt)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K,splits", [(8, 8, 16, 2), (72, 264, 1000, 3), (136, 520, 4104, 8), (8, 4096, 2048, 9), (304, 2048, 8192, 4), (128, 64, 200, 64)])
def test_split_contraction(M, N, K, splits, a_mn, b_mn):
    """More ranges than blocks of the contraction, ragged tiles and ends, every epilogue; the same bits every time."""
    from torchtune_b200.ops._cuda import _gemm_split

    a, b = _rand(M, K, seed=1), _rand(N, K, seed=2)
    want = a.double() @ b.double().t()
    x = a.t().contiguous() if a_mn else a
    w = b.t().contiguous() if b_mn else b
    new = lambda: torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    bias, r = _rand(N, seed=3), _rand(M, N, seed=4)
    got = _gemm_split(x, w, new(), splits, a_mn=a_mn, b_mn=b_mn)
    _check(got, want, a, b)
    assert torch.equal(got, _gemm_split(x, w, new(), splits, a_mn=a_mn, b_mn=b_mn))
    _check(_gemm_split(x, w, new(), splits, a_mn=a_mn, b_mn=b_mn, bias=bias, residual=r, alpha=0.5), 0.5 * want + bias.double() + r.double(), a, b)
    _check(_gemm_split(x, w, r.clone(), splits, a_mn=a_mn, b_mn=b_mn, accumulate=True), want + r.double(), a, b)
    wide = torch.ones(M, N + 8, dtype=torch.float32, device="cuda")
    _gemm_split(x, w, wide[:, :N], splits, a_mn=a_mn, b_mn=b_mn, accumulate=True)
    assert ((wide[:, :N].double() - want - 1).abs() <= 2.0**-19 * (a.double().abs() @ b.double().abs().t() + 1)).all() and (wide[:, N:] == 1).all()


def test_observed_modules_are_called():
    """Hooks on every module are seen by each call of each layer: projections are not joined and steps are not recorded."""
    from torchtune_b200 import generation, training
    from torchtune_b200.models.llama3_1 import llama3_1

    with training.set_default_dtype(torch.bfloat16), torch.device("cuda"):
        model = llama3_1(vocab_size=256, num_layers=1, num_heads=4, num_kv_heads=2, embed_dim=256, max_seq_len=128, intermediate_dim=256).eval()
        model.setup_caches(batch_size=1, dtype=torch.bfloat16, decoder_max_seq_len=32)
    seen = []
    handle = torch.nn.modules.module.register_module_forward_hook(lambda m, args, out: seen.append(m))
    try:
        generation.generate(model, torch.randint(1, 256, (1, 9), device="cuda"), max_generated_tokens=8)
    finally:
        handle.remove()
    mlp = model.layers[0].mlp
    for m in (model.layers[0].attn.k_proj, model.layers[0].attn.output_proj, mlp.w1, mlp.w2, mlp.w3, mlp.activation, model.norm):
        assert sum(x is m for x in seen) == 8


@pytest.mark.parametrize("name", ["w1", "w3", "activation"])
def test_a_hook_on_a_gate_changes_the_result(name):
    from torchtune_b200.modules import FeedForward
    from torchtune_b200.modules.linear import Linear

    with torch.device("cuda"), torch.no_grad():
        mlp = FeedForward(gate_proj=Linear(64, 128, bias=False), down_proj=Linear(128, 64, bias=False), up_proj=Linear(64, 128, bias=False)).bfloat16()
        x = _rand(5, 64)
        assert mlp(x).any()
        getattr(mlp, name).register_forward_hook(lambda m, args, out: torch.zeros_like(out))
        assert not mlp(x).any()


@pytest.mark.parametrize("fresh", [True, False])
@pytest.mark.parametrize("n", [2, 8])
def test_padded_rows(n, fresh):
    """Generation of left-padded prompts, with plain and with recorded steps, on fresh caches and on used ones, against one pass over each row without its padding."""
    import copy

    from torchtune_b200 import generation, training
    from torchtune_b200.models.llama3_1 import llama3_1

    torch.manual_seed(0)
    with training.set_default_dtype(torch.bfloat16), torch.device("cuda"):
        model = llama3_1(vocab_size=1024, num_layers=2, num_heads=8, num_kv_heads=2, embed_dim=512, max_seq_len=512, intermediate_dim=1024).eval()
        plain = copy.deepcopy(model)
        model.setup_caches(batch_size=3, dtype=torch.bfloat16, decoder_max_seq_len=40)
    prompt = torch.randint(1, 1024, (3, 20), device="cuda")
    if not fresh:
        generation.generate(model, prompt, max_generated_tokens=8)
        model.reset_caches()
    prompt[0, :7], prompt[2, :1] = 0, 0
    tokens, logits = generation.generate(model, prompt, max_generated_tokens=n, pad_id=0)
    for row, got, pad in zip(tokens, logits, (7, 0, 1)):
        with torch.no_grad():
            want = plain(row[None, pad:])[0, 19 - pad : -1]
        # bf16 activations through two layers
        assert got.shape == want.shape and (got - want).norm() <= 0.03 * want.norm()


def test_generation_beside_other_threads():
    """Another thread waits for the device and draws random numbers all the while, and generates itself: nothing fails, and the results are those of a single thread."""
    import threading

    from torchtune_b200 import generation, training
    from torchtune_b200.models.llama3_1 import llama3_1

    def model(seed):
        torch.manual_seed(seed)
        with training.set_default_dtype(torch.bfloat16), torch.device("cuda"):
            m = llama3_1(vocab_size=512, num_layers=2, num_heads=4, num_kv_heads=2, embed_dim=256, max_seq_len=128, intermediate_dim=512).eval()
            m.setup_caches(batch_size=2, dtype=torch.bfloat16, decoder_max_seq_len=40)
        return m

    def run(m):
        m.reset_caches()
        rng = torch.Generator(device="cuda").manual_seed(1)
        return generation.generate(m, torch.arange(1, 19, device="cuda").view(2, 9), max_generated_tokens=10, rng=rng)

    models = model(1), model(2)
    want = [run(m) for m in models]
    errors, done = [], threading.Event()

    def check(i):
        for got, ref in zip(run(models[i]), want[i]):
            assert torch.equal(got, ref)

    def beside():
        try:
            for _ in range(2000):
                if done.is_set():
                    break
                torch.rand(1000, device="cuda")
                torch.cuda.synchronize()
            check(1)
        except BaseException as e:
            errors.append(e)

    other = threading.Thread(target=beside)
    other.start()
    try:
        for _ in range(4):
            check(0)
    finally:
        done.set()
        other.join()
    assert not errors, errors
    check(0)


@pytest.mark.parametrize("how", ["inference mode", "checkpointed layers", "compiled projection", "three tokens"])
def test_generation_of_models_that_are_not_recorded(how):
    """The plain loop, with caches that live for one call as rollouts have them: the same tokens and logits as with recorded steps."""
    import copy

    from torchtune_b200 import generation, training
    from torchtune_b200.models.llama3_1 import llama3_1
    from torchtune_b200.modules import TransformerSelfAttentionLayer
    from torchtune_b200.modules.common_utils import delete_kv_caches

    torch.manual_seed(0)
    with training.set_default_dtype(torch.bfloat16), torch.device("cuda"):
        model = llama3_1(vocab_size=1024, num_layers=2, num_heads=8, num_kv_heads=2, embed_dim=512, max_seq_len=512, intermediate_dim=1024).eval()
    other = copy.deepcopy(model)
    if how == "checkpointed layers":
        training.set_activation_checkpointing(other, auto_wrap_policy={TransformerSelfAttentionLayer})
    elif how == "compiled projection":
        attn = other.layers[0].attn
        plain, attn.q_proj = attn.q_proj, torch.nn.Linear(512, 512, bias=False, device="cuda", dtype=torch.bfloat16)
        attn.q_proj.weight = plain.weight
        attn.q_proj.compile(backend="eager")
    n = 3 if how == "three tokens" else 9
    prompt = torch.randint(1, 1024, (3, 20), device="cuda")

    def run(m):
        with torch.device("cuda"):
            m.setup_caches(batch_size=3, dtype=torch.bfloat16, decoder_max_seq_len=40)
        out = generation.generate(m, prompt, max_generated_tokens=n, rng=torch.Generator(device="cuda").manual_seed(1))
        assert [layer.attn.kv_cache.size for layer in m.layers] == [20 + n - 1] * 2
        delete_kv_caches(m)
        return out

    want = run(model)
    with torch.inference_mode(how == "inference mode"):
        for _ in range(2):
            got = run(other)
            if how == "compiled projection":  # another product in another order: bf16 through two layers, before any draw
                assert (got[1][:, 0] - want[1][:, 0]).norm() <= 0.03 * want[1][:, 0].norm()
            else:
                assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("K", [1024, 1032, 2048, 4096])
@pytest.mark.parametrize("M", [1, 2, 3, 7, 8])
def test_products_of_normalised_tokens(M, K):
    """Norms on the way into the products for few tokens: the values of the norm's kernel followed by the products', through every split of the contraction."""
    import ctypes

    from torchtune_b200 import ops
    from torchtune_b200.ops import _cuda
    from torchtune_b200.ops._lib import check, lib, stream_ptr

    x, gain = _rand(M, K, seed=M) * 3, 1 + _rand(1, K, seed=4)[0] * 0.1
    n = ops.rms_norm(x, gain, 1e-5)
    for rows in ((16, 24), (520, 72), (4096, 1024), (20000, 8)):
        ws = [_rand(r, K, seed=r) for r in rows]
        want, got = [torch.empty(M, r, dtype=torch.bfloat16, device="cuda") for r in rows], [torch.empty(M, r, dtype=torch.bfloat16, device="cuda") for r in rows]
        _cuda._gemm_rows(n, ws, want)
        vps, lls = ctypes.c_void_p * 2, ctypes.c_longlong * 2
        check(lib().ttb_gemm_rows_normed(x.data_ptr(), K, gain.data_ptr(), 1e-5, M, K, 2, vps(*[w.data_ptr() for w in ws]), lls(K, K), (ctypes.c_int * 2)(*rows), vps(*[o.data_ptr() for o in got]),
                                         lls(*rows), None, stream_ptr()), "normed rows")
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        w1, w3 = _rand(rows[0], K, seed=5), _rand(rows[0], K, seed=6)
        check(lib().ttb_gemm_rows_gated(n.data_ptr(), K, w1.data_ptr(), w3.data_ptr(), K, want[0].data_ptr(), rows[0], M, rows[0], K, 0.0, 0.0, stream_ptr()), "gated")
        check(lib().ttb_gemm_rows_gated_normed(x.data_ptr(), K, gain.data_ptr(), 1e-5, w1.data_ptr(), w3.data_ptr(), K, got[0].data_ptr(), rows[0], M, rows[0], K, stream_ptr()), "gated, normed")
        assert torch.equal(got[0], want[0])
    assert not lib().ttb_gemm_rows_norms(9, 2048) and not lib().ttb_gemm_rows_norms(1, 1016) and not lib().ttb_gemm_rows_norms(1, 4104)
