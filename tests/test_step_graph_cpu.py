"""When a decode step is recorded (the recording itself needs a GPU)."""
import os
import threading
from types import SimpleNamespace

import pytest
import torch
from tqdm import tqdm

from torchtune_b200.generation._step_graph import StepGraph
from torchtune_b200.models.llama3_1 import llama3_1


@pytest.fixture
def steps(monkeypatch):
    """Runs decode steps and tells how many of them ran as they are and which masks were recorded."""
    torch.manual_seed(0)
    model = llama3_1(vocab_size=64, num_layers=1, num_heads=4, num_kv_heads=2, embed_dim=32, max_seq_len=32, intermediate_dim=64).eval()
    model.setup_caches(batch_size=4, dtype=torch.float32, decoder_max_seq_len=16)
    plain, recorded = [], []
    forward = model.forward
    monkeypatch.setattr(model, "forward", lambda *a, **kw: plain.append(a) or forward(*a, **kw))

    def record(self, x, input_pos, mask):
        recorded.append(tuple(mask.shape))
        self.x, self.pos, self.mask, self.logits = x.clone(), input_pos.view(-1, 1).clone(), mask.clone(), torch.zeros(x.shape[0], 64)
        self.graph = self.home.graph = SimpleNamespace(replay=lambda: None)

    monkeypatch.setattr(StepGraph, "_record", record)

    def run(batch, mask_rows, n=3):
        plain.clear(), recorded.clear()
        model.reset_caches()
        step = StepGraph(model, batch)
        with torch.no_grad():
            for i in range(n):
                step(torch.ones(batch, 1, dtype=torch.int64), torch.tensor([i]), torch.ones(mask_rows, 1, 16, dtype=torch.bool))
        return len(plain), recorded[:]

    return run


def test_a_step_of_a_new_batch_runs_before_it_is_recorded(steps):
    """Which kernels a step launches hangs on its batch and mask: what a recording from before has set up need not be what this one needs."""
    assert steps(2, 1) == (1, [(1, 1, 16)])
    assert steps(2, 1) == (0, [(1, 1, 16)])  # known
    assert steps(4, 1) == (1, [(1, 1, 16)])
    assert steps(4, 4) == (1, [(4, 1, 16)])
    assert steps(4, 4) == (0, [(4, 1, 16)]) and steps(2, 1) == (0, [(1, 1, 16)])


def test_nothing_is_recorded_beside_other_threads(steps):
    stop = threading.Event()
    other = threading.Thread(target=stop.wait)
    other.start()
    try:
        assert steps(2, 1) == (3, [])
    finally:
        stop.set()
        other.join()
    bars = tqdm(range(2), disable=False, file=open(os.devnull, "w"))  # with a thread of its own, which only draws
    assert steps(2, 1) == (0, [(1, 1, 16)])
    bars.close()
    inside = []
    other = threading.Thread(target=lambda: inside.append(steps(2, 1)))  # the main thread is the other one here
    other.start()
    other.join()
    assert inside == [(3, [])]
