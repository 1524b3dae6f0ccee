"""Weight gradients of grouped products whose contraction, the rows of an expert, is the ragged dimension."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from torchtune_b200 import ops


@pytest.mark.parametrize("K,N", [(64, 8), (136, 264), (1024, 512)])
@pytest.mark.parametrize("counts", [[1, 15, 16, 17], [0, 63, 64, 65, 0], [200, 1, 0, 47, 128, 31], [5] * 130])
def test_ragged_contraction(counts, K, N):
    """Ends inside and on a step of 16 rows and a block of 64, experts without rows, more experts than the staged epilogue takes; a neighbour's
    infinities stay its own; accumulation into a flat buffer is covered by the data-parallel tests."""
    g = torch.Generator(device="cuda").manual_seed(K + len(counts))
    rows = sum(counts)
    x = torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(rows, N, generator=g, device="cuda").to(torch.bfloat16)
    bad = next(e for e, c in enumerate(counts) if e > 0 and c)
    first = sum(counts[:bad])
    x[first], dy[first] = float("inf"), float("nan")
    w = torch.zeros(len(counts), K, N, dtype=torch.bfloat16, device="cuda").requires_grad_()
    ops.grouped_matmul(x, w, torch.tensor(counts, device="cuda")).backward(dy)
    at = 0
    for e, c in enumerate(counts):
        a, b = x[at : at + c].double(), dy[at : at + c].double()
        at += c
        if e == bad:
            assert w.grad[e].isnan().all()
            continue
        bound = 2.0**-8 * (a.t() @ b).abs() + 2.0**-19 * (a.abs().t() @ b.abs())  # one rounding to bf16, fp32 sums in any order
        assert ((w.grad[e].double() - a.t() @ b).abs() <= bound).all(), e


@pytest.mark.parametrize("K,N", [(64, 256), (136, 264), (1024, 2056), (5120, 520)])
@pytest.mark.parametrize("counts", [[1], [31, 32, 33], [0, 255, 256, 257, 0], [700, 1, 0, 513, 128, 64], [3] * 300, [2049, 5]])
def test_grouped_products_on_cta_pairs(counts, K, N, monkeypatch):
    """Pieces of all sizes, ends inside a TMA box, experts without rows, ragged blocks of weight rows and contractions; a neighbour's infinities stay its own."""
    monkeypatch.setattr("torchtune_b200.ops._cuda._groups_on_pairs", lambda rows, E, N, K: N >= 256)
    g = torch.Generator(device="cuda").manual_seed(K + len(counts))
    rows = sum(counts)
    x = torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(len(counts), K, N, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(rows, N, generator=g, device="cuda").to(torch.bfloat16)
    bad = next((e for e, c in enumerate(counts) if e > 0 and c), None)
    if bad is not None:
        x[sum(counts[:bad])] = float("inf")
    x.requires_grad_()
    y = ops.grouped_matmul(x, w, torch.tensor(counts, device="cuda"))
    y.backward(dy)
    at = 0
    for e, c in enumerate(counts):
        a, d, we = x[at : at + c].detach().double(), dy[at : at + c].double(), w[e].double()
        if e == bad:
            assert not y[at].isfinite().all()
            a, y_e = a[1:], y[at + 1 : at + c]
        else:
            y_e = y[at : at + c]
        for got, want, bound in ((y_e, a @ we, a.abs() @ we.abs()), (x.grad[at : at + c], d @ we.t(), d.abs() @ we.abs().t())):
            assert ((got.double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-19 * bound).all(), e  # one rounding to bf16, fp32 sums in any order
        at += c


@pytest.mark.parametrize("w_mn", [0, 1])
@pytest.mark.parametrize("counts", [[0, 0], [100, 0, 33], [300, -5, 257, 1], [700, 1], [600, 90, 400], [2**40, 3]])
def test_rows_of_no_expert_on_cta_pairs(counts, w_mn):
    """Counts that add up to fewer rows than there are leave the rest of the result alone, and no counts reach past it."""
    from torchtune_b200.ops._lib import check, check_device_errors, err_word, lib, stream_ptr

    rows, K, N, E = 700, 136, 264, len(counts)
    g = torch.Generator(device="cuda").manual_seed(E)
    x, w = torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16), torch.randn(E, *((K, N) if w_mn else (N, K)), generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((rows + 300, N), 7.0, dtype=torch.bfloat16, device="cuda")
    table, held = torch.empty(5 * (-(-rows // 256) + E) + 1, dtype=torch.int32, device="cuda"), torch.tensor(counts, device="cuda")
    check(lib().ttb_gemm_grouped_bf16_2sm(x.data_ptr(), w.data_ptr(), out.data_ptr(), held.data_ptr(), table.data_ptr(), rows, E, N, K, w_mn, K, w.stride(1),
                                          w.stride(0), N, err_word(x.device).data_ptr(), stream_ptr()), "grouped product")
    check_device_errors()
    at = 0
    for e, c in enumerate(counts):
        c = min(max(c, 0), rows - at)
        a, b = x[at : at + c].double(), w[e].double() if w_mn else w[e].double().t()
        assert ((out[at : at + c].double() - a @ b).abs() <= 2.0**-8 * (a @ b).abs() + 2.0**-19 * (a.abs() @ b.abs())).all(), e  # one rounding to bf16, fp32 sums in any order
        at += c
    assert (out[at:] == 7).all()
