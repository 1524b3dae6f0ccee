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
