"""Log-probabilities from fp32 logits and scaled gradients against plain statements in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from torchtune_b200 import rlhf


def _logits(rows, V, dtype, seed=0):
    x = torch.randn(rows, V, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * 4
    return x.to(dtype)


@pytest.mark.parametrize("temperature", [1.0, 0.7])
@pytest.mark.parametrize("b,s,V", [(1, 1, 4), (2, 3, 2048), (3, 5, 8188), (2, 4, 128256), (2, 3, 1001)])
def test_log_probabilities(b, s, V, temperature):
    """Slices of a batch, widths that end inside a load, one that the kernel does not take; infinities."""
    x = _logits(b * (s + 2), V, torch.float32, V).view(b, s + 2, V)
    x[0, 1, 1:] = float("-inf")
    tokens = torch.randint(0, V, (b, s), device="cuda")
    tokens[0, 0] = 0
    with torch.no_grad():
        got = rlhf.logits_to_logprobs(x[:, 1:-1], tokens, temperature)
    want = torch.log_softmax((x[:, 1:-1] / temperature).double(), -1).gather(2, tokens[..., None])[..., 0]
    assert got.dtype == torch.float32 and ((got.double() - want).abs() <= 2.0**-20 * (1 + want.abs())).all()
    x[0, 1] = float("-inf")
    with torch.no_grad():
        assert rlhf.logits_to_logprobs(x[:, 1:-1], tokens, temperature)[0, 0].isnan()
    x[0, 1], x[0, 1, 1] = 0.0, float("nan")
    with torch.no_grad():
        assert rlhf.logits_to_logprobs(x[:, 1:-1], tokens, temperature)[0, 0].isnan()
    x.requires_grad_()
    rlhf.logits_to_logprobs(x, torch.zeros(b, s + 2, dtype=torch.int64, device="cuda")).nansum().backward()
    assert x.grad is not None


@pytest.mark.parametrize("n", [8, 8 * 255, 8 * 1025, 8 * 1_000_003])
def test_scaled_gradients(n):
    from torchtune_b200.ops._cuda import _scaled

    x = _logits(1, n, torch.bfloat16)[0]
    f = torch.tensor(1 / 3, device="cuda")
    assert torch.equal(_scaled(x, f), (x.float() * f).to(torch.bfloat16))


@pytest.mark.parametrize("n", [2**20, 2**20 + 8, 8 * 1_000_003])
def test_widened_logits(n):
    from torchtune_b200 import ops

    x = _logits(1, n, torch.bfloat16, n)
    x[0, :3] = torch.tensor([float("nan"), float("inf"), -0.0])
    with torch.no_grad():
        got = ops.widen(x)
    assert got.dtype == torch.float32 and torch.equal(got.view(torch.int32)[:, 1:], x.float().view(torch.int32)[:, 1:]) and got[0, 0].isnan()


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 2048, 64), (16, 9992, 4096), (17, 128256, 2048), (300, 19208, 136), (1031, 4136, 1024), (333, 520, 4096), (100, 24, 64), (0, 64, 64)])
def test_widened_projection(M, N, K, bias):
    """Kernel for few tokens, CTA pairs with ragged last tiles, sizes that are widened afterwards: the values of the bf16 projection in every case."""
    from torchtune_b200 import ops

    x, w = _logits(M, K, torch.bfloat16, 1) * 0.1, _logits(N, K, torch.bfloat16, 2)
    b = _logits(1, N, torch.bfloat16, 3)[0] if bias else None
    with torch.no_grad():
        got, want = ops.linear_widened(x, w, b), ops.linear(x, w, b).float()
    assert got.dtype == torch.float32 and torch.equal(got, want)
    w.requires_grad_()
    assert ops.linear_widened(x, w, b).requires_grad


def test_loss_gradients_of_batched_and_differentiated_factors():
    from torchtune_b200 import ops

    h, w = (_logits(n, 64, torch.bfloat16, n).requires_grad_() for n in (16, 128))
    loss, _ = ops.linear_cross_entropy(h, w, torch.randint(0, 128, (16,), device="cuda"))
    once = torch.autograd.grad(loss, (h, w), retain_graph=True)
    many = torch.autograd.grad(loss, (h, w), torch.tensor([1.0, 2.0, -4.0], device="cuda"), is_grads_batched=True, retain_graph=True)
    for a, b in zip(once, many):
        assert torch.equal(b, torch.stack([a, 2 * a, -4 * a]))
    factor = torch.tensor(2.0, device="cuda", requires_grad=True)
    g, = torch.autograd.grad(loss, h, factor, create_graph=True)
    assert torch.equal(g, 2 * once[0])
    d, = torch.autograd.grad(g.float().sum(), factor)
    assert (d - once[0].float().sum()).abs() <= 2.0**-8 * once[0].float().abs().sum()


@pytest.mark.parametrize("T,D,V", [(1, 128, 128256), (257, 192, 9608), (700, 2048, 20000), (300, 1024, 128256), (4097, 64 * 3, 8448)])
def test_softmax_statistics_of_the_logits_product(T, D, V, monkeypatch):
    """Losses and gradients where the product that makes the logits leaves the statistics of their softmax, against 64 bits on the same bf16 logits: ragged tiles, labels at both ends, ignored
    rows and ids out of range, rows with one dominant logit."""
    from torchtune_b200 import ops
    from torchtune_b200.ops._cuda import _ce_stats
    from torchtune_b200.ops._lib import index_violations

    monkeypatch.setattr("torchtune_b200.ops._cuda._stats_pay", lambda *sizes: True)
    h, w = (_logits(T, D, torch.bfloat16, 1) * 0.25).requires_grad_(), (_logits(V, D, torch.bfloat16, 2) * 0.25 * D**-0.5).requires_grad_()
    with torch.no_grad():
        h[T // 2] *= 40
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[-1], labels[0] = V - 1, 0
    if T > 1:
        labels[::5], labels[3::50] = -100, V + 3
    with torch.no_grad():
        logits = ops.linear(h, w)
        assert _ce_stats(h, w, logits, 0.0) == (T > 16) and not _ce_stats(h, w, logits, 30.0)
    index_violations()
    total, count = ops.linear_cross_entropy(h, w, labels)
    total.backward()
    seen = (labels >= 0) & (labels < V)
    assert int(count) == int((labels != -100).sum()) and index_violations() == int((labels >= V).sum())
    z = logits.double()
    lse = torch.logsumexp(z, -1)
    want = torch.where(seen, lse - z.gather(1, labels.clamp(0, V - 1)[:, None])[:, 0], 0.0)
    # fp32 sums of V terms (partials of 256 added pairwise) and one logarithm of a sum
    assert abs(float(total) - float(want.sum())) <= 2.0**-19 * float((lse.abs() * seen).sum() + want.abs().sum()) + 1e-6
    p = torch.softmax(z, -1)
    p[torch.arange(T, device="cuda"), labels.clamp(0, V - 1)] -= 1
    p *= seen[:, None]
    for got, exact in ((h.grad, p @ w.double()), (w.grad, p.t() @ h.double())):
        assert float((got.double() - exact).norm()) <= 2.0**-7 * float(exact.norm())  # p and the result are rounded to bf16


@pytest.mark.parametrize("V", [19208, 18944])
def test_softmax_statistics_of_shifted_and_extreme_logits(V, monkeypatch):
    """Maximum and sum of exponentials of every tile against 64 bits: rows with a common offset, all or every other tile at either end of bf16's range; and the losses from them."""
    from torchtune_b200 import ops
    from torchtune_b200.ops._cuda import _ce_stats
    from torchtune_b200.ops._lib import check, err_word, lib, stream_ptr

    monkeypatch.setattr("torchtune_b200.ops._cuda._stats_pay", lambda *sizes: True)
    T, D, big = 300, 192, torch.finfo(torch.bfloat16).max
    w, h = torch.zeros(V, D, device="cuda"), torch.zeros(T, D, device="cuda")
    w[:, 0], w[:, 1], w[:, 2] = 1, _logits(1, V, torch.float32)[0], (torch.arange(V, device="cuda") // 256 + 1) % 2  # ones, noise, every other tile
    offsets = torch.tensor([0.0, 100.0, -1000.0, 1000.0, 3e4, -1e6, 1e6, big, -big], device="cuda")
    h[:, 0], h[:, 1] = offsets.repeat(T // 9 + 1)[:T], 1
    h[-2:, 0] = 0
    h[-2, 2], h[-1, 2] = big, -big  # every other tile masked, the first one with them
    h, w = h.to(torch.bfloat16), w.to(torch.bfloat16)
    logits = torch.empty(T, V, dtype=torch.bfloat16, device="cuda")
    assert _ce_stats(h, w, logits, 0.0)
    stats = torch.empty(-(-V // 256), T, 2, device="cuda")
    check(lib().ttb_gemm_bf16_2sm_stats(h.data_ptr(), w.data_ptr(), logits.data_ptr(), stats.data_ptr(), T, V, D, D, D, V, err_word(h.device).data_ptr(), stream_ptr()), "statistics")
    with torch.no_grad():
        assert torch.equal(logits, ops.linear(h, w))
    z = logits.double()
    for tile in range(stats.shape[0]):
        part = z[:, tile * 256 : (tile + 1) * 256]
        top = part.amax(1)
        assert torch.equal(stats[tile, :, 0].double(), top)
        # differences and products of fp32, exponentials good to 2^-22 and eight rescaled partial sums: 2^-18 of a sum that is at least 1
        assert ((stats[tile, :, 1].double() / (part - top[:, None]).exp().sum(1) - 1).abs() <= 2.0**-18).all(), tile
    lse, labels = torch.logsumexp(z, -1), torch.randint(0, V, (T,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    want = lse - z.gather(1, labels[:, None])[:, 0]
    half_ulp = (torch.nextafter(lse.float().abs(), torch.full_like(lse, float("inf"), dtype=torch.float32)).double() - lse.float().abs().double()) / 2
    for i in (*range(9), T - 2, T - 1):
        alone = torch.full_like(labels, -100)
        alone[i] = labels[i]
        got = float(ops.linear_cross_entropy(h, w, alone)[0])
        # the logarithm's 2^-19, one rounding of its sum with the maximum, and one of the difference with the label's logit
        assert abs(got - float(want[i])) <= 2.0**-19 * 20 + float(half_ulp[i]) + 2.0**-24 * abs(float(want[i])), (i, got, float(want[i]))


@pytest.mark.parametrize("T,V", [(16, 128), (700, 20000)])
def test_mean_loss(T, V):
    """The mean's gradients with and without statistics of the softmax, for factors of one and others, kept graphs, hooks on saved tensors, batched factors, and no valid token."""
    from torchtune_b200 import ops
    from torchtune_b200.modules.loss import LinearCrossEntropyLoss

    h, w = _logits(T, 64, torch.bfloat16, T).requires_grad_(), (_logits(V, 64, torch.bfloat16, V) * 0.1).requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[::3] = -100
    total, count = ops.linear_cross_entropy(h, w, labels)
    sums = torch.autograd.grad(total, (h, w))
    mean = lambda: ops.linear_cross_entropy_mean(h, w, labels)
    exact = [g.double() / int(count) for g in sums]
    assert abs(float(mean().detach()) - float(total.detach()) / int(count)) <= 2.0**-20 * abs(float(total.detach()))

    def near(got, factor=1.0):
        for a, e in zip(got, exact):
            assert float((a.double() - factor * e).norm()) <= 2.0**-7 * abs(factor) * float(e.norm())  # a rounding to bf16 on each side, and one more of a rescaled result

    near(torch.autograd.grad(mean(), (h, w)))
    near(torch.autograd.grad(mean() * -2.5, (h, w)), -2.5)
    loss = mean()
    kept = torch.autograd.grad(loss, (h, w), retain_graph=True)
    again = torch.autograd.grad(loss, (h, w), torch.tensor(4.0, device="cuda"), retain_graph=True)
    once_more = torch.autograd.grad(loss, (h, w))
    assert all(torch.equal(a, c) and torch.equal(4 * a, b) for a, b, c in zip(kept, again, once_more))
    many = torch.autograd.grad(mean(), (h, w), torch.tensor([1.0, -2.0], device="cuda"), is_grads_batched=True)
    assert all(torch.equal(m, torch.stack([a, -2 * a])) for m, a in zip(many, kept))
    held = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: held.append(t) or t, lambda t: t):
        loss = mean()
    before = [t.clone() for t in held]
    near(torch.autograd.grad(loss * 3, (h, w)), 3.0)
    assert all(torch.equal(a, b) for a, b in zip(held, before))
    for keep in (lambda t: t, lambda t: t.detach(), torch.clone):  # hooks on the node's own saved tensors, which come later
        loss, held = mean(), []
        for saved in loss.grad_fn._raw_saved_tensors[:2]:
            saved.register_hooks(lambda t: held.append(keep(t)) or len(held) - 1, lambda i: held[i])
        before = [t.clone() for t in held]
        near(torch.autograd.grad(loss * 3, (h, w)), 3.0)
        assert len(held) == 2 and all(torch.equal(a, b) for a, b in zip(held, before))
    loss = mean()
    places = [t.data_ptr() for t in loss.grad_fn.saved_tensors[:2]]
    assert [g.data_ptr() for g in torch.autograd.grad(loss, (h, w))] == places  # nobody else has them: no copies
    labels.fill_(-100)
    loss = mean()
    assert float(loss.detach()) == 0.0 and all(not g.any() for g in torch.autograd.grad(loss, (h, w)))
    module = LinearCrossEntropyLoss()
    module.linear_projection = torch.nn.Linear(64, V, bias=False, device="cuda", dtype=torch.bfloat16)
    labels[1::3] = 5
    got, want = module(h, labels), torch.nn.functional.cross_entropy((h.double() @ module.linear_projection.weight.double().t()), labels)
    assert abs(float(got.detach()) - float(want.detach())) <= 0.02 * abs(float(want.detach()))


@pytest.mark.parametrize("written", [False, True])
@pytest.mark.parametrize("T,V", [(16, 128), (700, 20000)])
def test_mean_loss_of_a_weight_with_a_gradient_window(T, V, written):
    """A weight whose gradients are delivered straight to a flat buffer: the mean's arrives as that of the mean, whatever multiplies it and whatever was there before; the sum's
    goes straight to the buffer, and that of a loss without autograd nowhere."""
    from types import SimpleNamespace

    from torchtune_b200 import ops
    from torchtune_b200.ops import _cuda
    from torchtune_b200.parallel.dp import FlatLayout

    h, w = _logits(T, 64, torch.bfloat16, T).requires_grad_(), torch.nn.Parameter(_logits(V, 64, torch.bfloat16, V) * 0.1)
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[::3] = -100
    total, count = ops.linear_cross_entropy(h, w, labels)
    want_h, want_w = (g.double() / int(count) for g in torch.autograd.grad(total, (h, w)))
    w._grad_buffer, w._grad_written = torch.full_like(w, 0.25 if written else float("nan")), written
    _cuda.enable_direct_wgrad(True, use_side_stream=False)
    _cuda.register_grad_window(w)
    try:
        (ops.linear_cross_entropy_mean(h, w, labels) * 0.5).backward()
        FlatLayout.collect_autograd_grads(SimpleNamespace(params=[w]))
        for got, want in ((h.grad.double(), want_h), (w._grad_buffer.double() - 0.25 * written, want_w)):
            # roundings to bf16 of the gradient on both sides and of a sum with 0.25
            assert float((got - 0.5 * want).norm()) <= 2.0**-7 * 0.5 * float(want.norm()) + written * 2.0**-9 * want.numel() ** 0.5
        w._grad_written = False
        ops.linear_cross_entropy(h, w, labels)[0].backward()
        assert w.grad is None and w._grad_written and float((w._grad_buffer.double() - int(count) * want_w).norm()) <= 2.0**-7 * int(count) * float(want_w.norm())
        before = w._grad_buffer.clone()
        with torch.no_grad():  # a validation loss between two steps
            for w._grad_written in (True, False):
                again, mean = ops.linear_cross_entropy(h, w, labels)[0], ops.linear_cross_entropy_mean(h, w, labels)
                assert torch.equal(w._grad_buffer, before) and not again.requires_grad and not mean.requires_grad
                assert abs(float(again) - float(total)) <= 2.0**-20 * float(total) and abs(float(mean) * int(count) - float(total)) <= 2.0**-19 * float(total)
            assert w._grad_written is False
    finally:
        _cuda.enable_direct_wgrad(False)
        _cuda.unregister_grad_window(w.data_ptr())
