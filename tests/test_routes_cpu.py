"""Which calls the CUDA wrappers take, pass on or refuse, with the kernel library replaced by a recorder (no GPU)."""
import pytest
import torch

from torchtune_b200 import ops
from torchtune_b200.ops import _cuda


class _Recorder:
    """Stands for the kernel library: notes the entry points that are called and does nothing."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append(name)
            return 0

        return entry


@pytest.fixture
def library(monkeypatch):
    rec = _Recorder()
    monkeypatch.setattr(_cuda, "lib", lambda: rec)
    monkeypatch.setattr(_cuda, "stream_ptr", lambda: 0)
    monkeypatch.setattr(_cuda, "err_word", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(_cuda, "_SM_PAIRS", 74)
    return rec


def _zeros(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


@pytest.mark.parametrize("tokens", [4, 300, 20000])
@pytest.mark.parametrize("width,weight_width", [(4096, 2048), (8192, 4096), (2048, 4096)])
def test_contraction_widths_have_to_agree(library, tokens, width, weight_width):
    """An input of another width than the weight is refused, whichever kernel the sizes would choose."""
    x, w, r = _zeros(1, width).expand(tokens, width), _zeros(4096, weight_width), _zeros(1, 4096).expand(tokens, 4096)
    with pytest.raises(ValueError, match="contraction mismatch"):
        _cuda.gemm_residual(x, w, r)
    with torch.no_grad():
        assert _cuda.linear_group(x, [_zeros(4096, width), w], [None, None]) is None
        assert _cuda.gate_up_swiglu(x, w, w) is None
    assert library.calls == []


def test_agreeing_widths_are_taken(library):
    x, w = _zeros(4, 2048), _zeros(512, 2048)
    with torch.no_grad():
        assert _cuda.gemm_residual(x, w, _zeros(4, 512)).shape == (4, 512)
        assert [y.shape for y in _cuda.linear_group(x, [w, w], [None, None])] == [(4, 512)] * 2
        assert _cuda.gate_up_swiglu(x, w, w).shape == (4, 512)
    assert library.calls == ["ttb_gemm_rows", "ttb_gemm_rows", "ttb_gemm_rows_gated"]


def test_a_bias_of_another_length_is_left_to_the_general_path(library):
    x, w = _zeros(4, 2048), _zeros(512, 2048)
    with torch.no_grad():
        assert _cuda.linear_group(x, [w, w], [None, _zeros(256)]) is None
    assert library.calls == []


@pytest.mark.parametrize("width", [2048, 4096, 8192])
def test_residual_product_of_no_tokens(library, width):
    """Nothing to multiply: an empty result, and gradients of zeros, at widths that would be cut into ranges too."""
    x, w, r = (_zeros(*s).requires_grad_() for s in ((0, width), (512, width), (0, 512)))
    y = _cuda.linear_residual(x, w, None, r)
    assert y.shape == (0, 512)
    y.sum().backward()
    assert x.grad.shape == (0, width) and r.grad.shape == (0, 512) and w.grad.shape == (512, width) and not w.grad.any()
    assert _cuda.gemm_residual(_zeros(5, width), _zeros(0, width), _zeros(5, 0)).shape == (5, 0)
    assert library.calls == []


def test_positions_of_single_tokens():
    """Padded rows are stepped with one position each, as a vector: the rows', not the sequence's."""
    assert torch.equal(_cuda._positions(torch.tensor([4, 7, 2]), 3, 1, "cpu"), torch.tensor([[4], [7], [2]], dtype=torch.int32))
    assert torch.equal(_cuda._positions(torch.tensor([4, 7]), 3, 2, "cpu"), torch.tensor([[4, 7]] * 3, dtype=torch.int32))
    assert torch.equal(_cuda._positions(torch.tensor([5]), 3, 1, "cpu"), torch.tensor([[5]] * 3, dtype=torch.int32))
    assert torch.equal(_cuda._positions(torch.tensor([[4], [7], [2]]), 3, 1, "cpu"), torch.tensor([[4], [7], [2]], dtype=torch.int32))
    with pytest.raises(RuntimeError):
        _cuda._positions(torch.tensor([4, 7, 2]), 2, 1, "cpu")


@pytest.mark.parametrize("bad", [-100, -1, 64, 2**40])
def test_token_ids_out_of_range_are_refused(library, bad):
    """Log-probabilities of ids that no column belongs to: refused by the same operation as in the plain statement."""
    logits, tokens = torch.zeros(2, 3, 64), torch.zeros(2, 3, dtype=torch.int64)
    assert _cuda.logits_logprobs_f32(logits, tokens, 1.0) is not None
    tokens[1, 2] = bad
    with pytest.raises(RuntimeError, match="out of bounds"):
        _cuda.logits_logprobs_f32(logits, tokens, 1.0)
    assert library.calls == ["ttb_token_logprobs_f32"]


def test_log_probabilities_want_a_batch():
    """As the plain statement does: rows of a batch, not a single sequence."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    with FakeTensorMode(), torch.no_grad():
        assert ops.logits_logprobs(torch.zeros(3, 64, device="cuda"), torch.zeros(3, dtype=torch.int64, device="cuda")) is None


def test_tensors_without_memory_take_the_plain_statements():
    """Fake tensors of a trace and batched ones of vmap have no address to give to a kernel."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    from torchtune_b200 import rlhf

    with FakeTensorMode(), torch.no_grad():
        logits, tokens = torch.zeros(2, 3, 64, device="cuda"), torch.zeros(2, 3, dtype=torch.int64, device="cuda")
        assert rlhf.logits_to_logprobs(logits, tokens).shape == (2, 3)
        assert ops.widen(torch.zeros(2**20, dtype=torch.bfloat16, device="cuda")).dtype == torch.float32
        many = torch.vmap(rlhf.logits_to_logprobs)(torch.zeros(5, 2, 3, 64, device="cuda"), torch.zeros(5, 2, 3, dtype=torch.int64, device="cuda"))
        assert many.shape == (5, 2, 3)


def test_scaled_gradients_of_batched_and_differentiated_factors(library):
    """The loss's stored gradients times an upstream factor: the kernel for a plain number, tensor operations where the factor is batched or its own gradient is wanted."""
    t, many = torch.arange(16, dtype=torch.bfloat16), torch.tensor([1.0, 2.0, -4.0])
    batched = torch.vmap(lambda f: _cuda._scaled(t, f))(many)
    assert torch.equal(batched, t * many[:, None].bfloat16())

    class Stored(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.float().sum()

        @staticmethod
        def backward(ctx, g):
            return _cuda._scaled(t, g)

    x = torch.zeros(16, dtype=torch.bfloat16, requires_grad=True)
    assert torch.equal(torch.autograd.grad(Stored.apply(x), x, many, is_grads_batched=True)[0], batched)
    factor = torch.tensor(3.0, requires_grad=True)
    g, = torch.autograd.grad(_cuda._scaled(t, factor).float().sum(), factor)
    assert g == t.float().sum()
    assert library.calls == []
    with torch.no_grad():
        _cuda._scaled(t, factor)
    _cuda._scaled(t, factor.detach())
    assert library.calls == ["ttb_scale_bf16"] * 2


@pytest.mark.parametrize("M,N,K,pays", [(64, 32000, 2048, False), (300, 32000, 2048, False), (1000, 32000, 2048, True), (20, 128256, 2048, True), (300, 128256, 1024, False), (4096, 128256, 512, False), (8192, 128256, 4096, True)])
def test_softmax_statistics_are_taken_where_they_were_measured_to_pay(library, M, N, K, pays):
    assert _cuda._stats_pay(M, N, K, None) is pays


@pytest.mark.parametrize("rows,E,K,N,pairs", [
    (4096, 8, 2048, 2048, False), (6144, 8, 2048, 2048, False), (8192, 32, 2048, 768, False), (16384, 32, 1024, 1024, False), (16384, 64, 768, 1024, False), (4096, 8, 4096, 2048, False), (4096, 8, 2048, 4096, True), (10000, 16, 2048, 1280, False), (10000, 16, 1280, 2048, True),
    (8192, 16, 2048, 2048, True), (32768, 64, 768, 2048, True), (5000, 8, 8192, 8192, True), (600, 4, 8192, 8192, True), (2048, 16, 4096, 4096, True), (256, 4, 8192, 14336, False),
    (512, 8, 8192, 4096, False), (1024, 16, 4096, 4096, False), (4096, 64, 2048, 2048, False), (2048, 32, 4096, 4096, False), (300, 16, 5120, 8192, True), (8192, 128, 2048, 1024, True), (40000, 16, 8192, 200, False)])
def test_grouped_products_run_where_they_were_measured_to_be_faster(rows, E, K, N, pairs):
    assert _cuda._groups_on_pairs(rows, E, N, K) is pairs
