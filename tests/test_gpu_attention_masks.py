"""Attention of few queries and attention under boolean masks against the plain statement in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from torchtune_b200 import ops
from torchtune_b200.ops.mask import AttentionMask


@pytest.fixture(autouse=True)
def _check_device_errors():
    yield
    from torchtune_b200.ops._lib import check_device_errors

    torch.cuda.synchronize()
    check_device_errors()


def _qkv(b, s, sk, hq, hkv, d, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(b, n, h, d, generator=g, device="cuda").to(torch.bfloat16) for n, h in ((s, hq), (sk, hkv), (sk, hkv))]


def _check(q, k, v, mask, dense):
    with torch.no_grad():
        got = ops.attention(q, k, v, mask)
    b, s, hq, d = q.shape
    group = q.double().view(b, s, k.shape[2], -1, d)
    score = torch.einsum("bqgnd,bkgd->bgnqk", group, k.double()) * d**-0.5
    p = torch.softmax(score.masked_fill(~dense[:, None, None], float("-inf")), -1).nan_to_num()  # a query without keys: 0
    want, square = (torch.einsum("bgnqk,bkgd->bqgnd", w, t).reshape(b, s, hq, d) for w, t in ((p, v.double()), (p.square(), v.double().square())))
    # The result is rounded to 8 bits (at most 2^-9 of it; twice that here), and so is every weight before it meets its value: errors of at most 2^-9 of
    # the terms, without a common sign, so eight times 2^-9 of the terms' root of squares (14 standard deviations) bounds their sum.
    bound = 2.0**-8 * want.abs() + 2.0**-6 * square.sqrt()
    assert ((got.double() - want).abs() <= bound).all(), float(((got.double() - want).abs() - bound).max())


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("sk", [1, 17, 64, 65, 333])
def test_every_key_counts_for_few_queries(sk, d):
    """One key holds all of the weight, another one in each batch row: the result is its value."""
    u = _qkv(1, 1, 1, 1, 1, d, seed=1)[0].sign()
    v = _qkv(sk, 1, sk, 1, 1, d, seed=2)[2]
    k = torch.zeros_like(v)
    at = torch.arange(sk, device="cuda")
    k[at, at] = u[0, 0] * (40.0 / d**0.5)  # its score is 40, the others' 0
    with torch.no_grad():
        got = ops.attention(u.expand(sk, 1, 1, d).contiguous(), k, v, AttentionMask(causal=False))
    assert ((got[:, 0].double() - v[at, at].double()).abs() <= 2.0**-8 * v[at, at].double().abs() + 1e-9).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("at", [0, 15, 16, 63, 64, 4095, 8191, 8192, 40000, 65535])
def test_any_key_of_a_long_range_counts(at, d):
    u = _qkv(1, 1, 1, 1, 1, d, seed=1)[0].sign()
    v = _qkv(1, 1, 65536, 1, 1, d, seed=2)[2]
    k = torch.zeros_like(v)
    k[0, at] = u[0, 0] * (40.0 / d**0.5)
    with torch.no_grad():
        got = ops.attention(u, k, v, AttentionMask(causal=False, bool_mask=torch.ones(1, 1, 65536, dtype=torch.bool, device="cuda")))
    assert ((got[0, 0].double() - v[0, at].double()).abs() <= 2.0**-8 * v[0, at].double().abs() + 1e-9).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("sk", [130, 300, 513])
def test_every_key_counts_on_the_tiles(sk, d):
    """Every query looks for one key, which a mask with gaps leaves visible; codes of random signs keep the other scores at least 20 below."""
    code = _qkv(1, 1, sk, 1, 1, d, seed=3)[1].sign()
    v = _qkv(1, 1, sk, 1, 1, d, seed=4)[2]
    order = torch.randperm(sk, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    q = code[:, order] * 8
    m = torch.rand(1, sk, sk, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)) < 0.5
    m[0, torch.arange(sk, device="cuda"), order] = True
    score = torch.einsum("qd,kd->qk", q[0, :, 0].double(), code[0, :, 0].double()) * d**-0.5
    own = score.gather(1, order[:, None])
    assert (score.scatter(1, order[:, None], float("-inf")).amax(1) <= own[:, 0] - 20).all()
    with torch.no_grad():
        got = ops.attention(q, code, v, AttentionMask(causal=False, bool_mask=m))
    want = v[0, order].double()
    assert ((got[0].double() - want).abs() <= 2.0**-8 * want.abs() + 1e-5).all()  # 513 others of weight e^-20


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,s,sk,hq,hkv", [(1, 1, 1, 4, 4), (1, 1, 61, 32, 8), (3, 1, 64, 8, 8), (2, 1, 65, 16, 1), (1, 4, 129, 8, 2), (40, 1, 200, 32, 8), (1, 1, 4097, 8, 1), (2, 16, 333, 2, 2),
                                           (1, 1, 65536, 1, 1)])
def test_few_queries(b, s, sk, hq, hkv, d):
    """Tile edges, cluster sizes, one to sixteen rows per key head; boolean masks (also views of wider ones), causal ends and row starts."""
    q, k, v = _qkv(b, s, sk, hq, hkv, d, seed=sk)
    at = torch.arange(sk, device="cuda")
    used = max(s, sk - 3)
    own = torch.arange(used - s, used, device="cuda")
    wide = torch.zeros(1, s, sk + 5, dtype=torch.bool, device="cuda")
    wide[..., :sk] = at[None, None, :] <= own[None, :, None]
    k[:, used:], v[:, used:] = float("nan"), float("nan")  # slots that no query sees don't enter the result
    kk, vv = k.nan_to_num(), v.nan_to_num()
    with torch.no_grad():
        torch.testing.assert_close(ops.attention(q, k, v, AttentionMask(causal=False, bool_mask=wide[..., :sk])), ops.attention(q, kk, vv, AttentionMask(causal=False, bool_mask=wide[..., :sk])), rtol=0, atol=0)
    _check(q, kk, vv, AttentionMask(causal=False, bool_mask=wide[..., :sk]), wide[..., :sk].expand(b, s, sk))
    _check(q, kk, vv, AttentionMask(causal=True), (at[None, None, :] <= (sk - s + torch.arange(s, device="cuda"))[None, :, None]).expand(b, s, sk))
    g = torch.Generator(device="cuda").manual_seed(1)
    m = torch.rand(b, s, sk, generator=g, device="cuda") < 0.4
    m[0, 0] = False  # a query that sees nothing gives zeros
    _check(q, kk, vv, AttentionMask(causal=False, bool_mask=m), m)
    start = torch.randint(0, max(1, sk - s), (b,), generator=g, device="cuda", dtype=torch.int32)
    slots = AttentionMask(causal=True, key_start=start, query_start=sk - s)
    _check(q, kk, vv, slots, slots.dense(b, s, sk, "cuda"))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,s,sk", [(2, 300, 300), (1, 513, 700), (3, 130, 257)])
def test_boolean_masks(b, s, sk, d):
    """Causal masks over a wider cache (shared by all rows), left padding, masks with gaps, ranges that jump and rows that see nothing."""
    q, k, v = _qkv(b, s, sk, 8, 2, d, seed=s)
    at, own = torch.arange(sk, device="cuda"), torch.arange(s, device="cuda")
    causal = (at[None, :] <= own[:, None])[None]
    _check(q, k, v, AttentionMask(causal=False, bool_mask=causal), causal.expand(b, s, sk))
    pad = torch.randint(0, s // 2, (b,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    left = (causal & (at >= pad[:, None, None])) | (at[None, :] == own[:, None])
    _check(q, k, v, AttentionMask(causal=False, bool_mask=left.unsqueeze(1)), left)
    g = torch.Generator(device="cuda").manual_seed(2)
    gaps = torch.rand(b, s, sk, generator=g, device="cuda") < 0.2
    gaps[:, 5] = False
    _check(q, k, v, AttentionMask(causal=False, bool_mask=gaps), gaps)
    jump = torch.zeros(b, s, sk, dtype=torch.bool, device="cuda")  # the two query tiles of a CTA see far ranges, in either order
    jump[:, :128, sk - 20 :], jump[:, 128:, :9] = True, True
    _check(q, k, v, AttentionMask(causal=False, bool_mask=jump), jump)
    jump = jump.flip(2).contiguous()
    _check(q, k, v, AttentionMask(causal=False, bool_mask=jump), jump)


def test_mask_bounds_on_the_device_are_the_plain_ones():
    from torchtune_b200.ops._cuda_attention import dense_mask_bounds, mask_row_bounds

    g = torch.Generator().manual_seed(0)
    for sk in (1, 15, 16, 17, 47, 400):
        m = torch.rand(3, 7, sk + 3, generator=g) < 0.5
        m[1, 2] = False
        m[2, 3] = True
        for view in (m[..., :sk], m[..., 3:], m[:1, :, 1 : sk + 1].expand(3, 7, sk)):
            _, lo, hi = dense_mask_bounds(view, 3, 7, sk)
            count = view.sum(-1)
            lo2, hi2, solid = mask_row_bounds(view.cuda() if view.stride(0) else view[:1].cuda().expand(3, 7, sk))
            assert (lo2.cpu() == lo).all() and (hi2.cpu() == hi).all()
            assert (solid.cpu().bool() == ((count == 0) | (count == hi - lo + 1))).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,s,sk,hq,hkv,kind", [(1, 1, 1, 1, 1, "full"), (2, 130, 70, 4, 2, "full"), (3, 257, 257, 6, 2, "causal"), (1, 640, 640, 8, 1, "causal"), (2, 100, 333, 4, 4, "causal"),
                                                (2, 500, 500, 4, 2, "documents"), (1, 700, 700, 4, 1, "window"), (2, 150, 500, 4, 2, "slots"), (2, 129, 300, 2, 1, "slots")])
def test_gradients(b, s, sk, hq, hkv, kind, d):
    """One to many query blocks per key block, ragged ends beside another batch row, keys and queries that nothing reaches."""
    q, k, v = _qkv(b, s, sk, hq, hkv, d, seed=s + d)
    do = _qkv(b, s, sk, hq, hkv, d, seed=5)[0]
    at, own = torch.arange(sk, device="cuda"), torch.arange(sk - s, sk, device="cuda")
    dense = (at[None, :] <= own[:, None])[None].expand(b, s, sk)
    mask = AttentionMask(causal=True)
    if kind == "full":
        mask, dense = AttentionMask(causal=False), torch.ones(b, s, sk, dtype=torch.bool, device="cuda")
    elif kind == "documents":
        mask = AttentionMask.from_seq_lens([[3, 250, 1, 246], [128, 372]]).to("cuda")
        ids = mask.doc_ids
        dense = dense & (ids[:, :, None] == ids[:, None, :])
    elif kind == "window":
        mask = AttentionMask(causal=True, window=90)
        dense = dense & (own[:, None] - at[None, :] < 90)
    elif kind == "slots":
        start = torch.randint(0, 60, (b,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1), dtype=torch.int32)
        mask = AttentionMask(causal=True, key_start=start, query_start=40)  # the first queries of a row see nothing, nor does anything see the last keys
        dense = mask.dense(b, s, sk, "cuda")
    leaves = [t.requires_grad_() for t in (q, k, v)]
    ops.attention(*leaves, mask).backward(do)
    want = [t.detach().double().requires_grad_() for t in (q, k, v)]
    with torch.no_grad():
        seen = dense.any(-1)
    group = hq // hkv
    kk, vv = (t.repeat_interleave(group, 2) for t in want[1:])
    score = torch.einsum("bqhd,bkhd->bhqk", want[0], kk) * d**-0.5
    prob = torch.softmax(score.masked_fill(~dense[:, None], float("-inf")).masked_fill(~seen[:, None, :, None], 0.0), -1) * dense[:, None]
    torch.einsum("bhqk,bkhd->bqhd", prob, vv).backward(do.double())
    for got, ref64, name in zip(leaves, want, "qkv"):
        # probabilities, their gradients and the results are rounded to 8 bits; so are the output and dO that delta is the sum of
        err = (got.grad.double() - ref64.grad).norm() / ref64.grad.norm().clamp_min(1e-3)
        assert err < 0.01 and (got.grad.double() - ref64.grad).abs().max() < 0.03 * max(1.0, ref64.grad.abs().max().item()), (name, float(err))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("scale", [-0.2, 0.0, 0.05])
@pytest.mark.parametrize("s,sk", [(1, 77), (200, 200), (140, 300)])
def test_scales_of_any_sign(s, sk, scale, d):
    """Scores times a negative scale or 0, without a mask, causal and under a boolean mask with gaps: results and gradients of all kernels."""
    q, k, v = _qkv(2, s, sk, 4, 2, d, seed=sk)
    do = _qkv(2, s, sk, 4, 2, d, seed=5)[0]
    at, own = torch.arange(sk, device="cuda"), torch.arange(sk - s, sk, device="cuda")
    causal = (at[None, :] <= own[:, None])[None].expand(2, s, sk)
    gaps = (torch.rand(2, s, sk, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) < 0.3) | (at[None, None, :] == own[None, :, None])
    for mask, dense in ((AttentionMask(causal=False), torch.ones_like(causal)), (AttentionMask(causal=True), causal), (AttentionMask(causal=False, bool_mask=gaps), gaps)):
        leaves = [t.detach().clone().requires_grad_() for t in (q, k, v)]
        got = ops.attention(*leaves, mask, scale=scale)
        got.backward(do)
        with torch.no_grad():
            alone = ops.attention(q, k, v, mask, scale=scale)
        want = [t.detach().double().requires_grad_() for t in (q, k, v)]
        kk, vv = (t.repeat_interleave(2, 2) for t in want[1:])
        prob = torch.softmax((torch.einsum("bqhd,bkhd->bhqk", want[0], kk) * scale).masked_fill(~dense[:, None], float("-inf")), -1)
        out = torch.einsum("bhqk,bkhd->bqhd", prob, vv)
        out.backward(do.double())
        # probabilities and results are rounded to 8 bits, as in the tests above
        bound = 2.0**-8 * (out.abs() + torch.einsum("bhqk,bkhd->bqhd", prob, vv.abs()))
        assert ((got.double() - out).abs() <= bound).all() and ((alone.double() - out).abs() <= bound).all()
        for leaf, ref64 in zip(leaves, want):
            assert (leaf.grad.double() - ref64.grad).norm() <= 0.01 * ref64.grad.norm().clamp_min(1e-3)


@pytest.mark.parametrize("d", [64, 128])
def test_a_cap_below_zero_is_none(d):
    q, k, v = (t.requires_grad_() for t in _qkv(2, 130, 130, 4, 2, d))
    m = torch.rand(2, 130, 130, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) < 0.5
    for mask in (AttentionMask(causal=True), AttentionMask(causal=False, bool_mask=m)):
        got, want = (ops.attention(q, k, v, mask, softcap=cap) for cap in (-5.0, 0.0))
        assert torch.equal(got, want)
        for a, b in zip(torch.autograd.grad(got, (k, v), torch.ones_like(got)), torch.autograd.grad(want, (k, v), torch.ones_like(want))):
            assert torch.equal(a, b)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("s", [3, 100, 129, 200, 255])
def test_values_keep_clear_of_the_next_row(s, d):
    """The last query tile of a batch row ends in the next one's queries: infinite scores there don't reach this row's values."""
    q, k, v = _qkv(2, s, s, 4, 2, d, seed=s)
    q[1] = float("inf")
    k = k.abs() + 0.1
    leaves = [t.requires_grad_() for t in (q, k, v)]
    ops.attention(*leaves, AttentionMask(causal=True)).backward(torch.ones_like(q))
    assert leaves[0].grad[0].isfinite().all() and leaves[2].grad[0].isfinite().all()
    one = [t.detach()[:1].clone().requires_grad_() for t in leaves]
    ops.attention(*one, AttentionMask(causal=True)).backward(torch.ones_like(one[0]))
    assert torch.equal(one[2].grad, leaves[2].grad[:1])
