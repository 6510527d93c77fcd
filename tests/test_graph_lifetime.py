"""What a captured training step reads by address lives as long as its graph (CPU: the CUDA
stream and graph calls are replaced by stand-ins, so only the lifetimes are exercised)."""
import contextlib
import gc
import types
import weakref

import pytest
import torch

from matpl_gb300 import nep_ops, ops, splitk
from matpl_gb300.nep_train import GraphedNepTrainer
from matpl_gb300.train import GraphedTrainer

SIDE = 77


class _Stream:
    cuda_stream = SIDE

    def wait_stream(self, other):
        pass


@pytest.fixture
def fake_cuda(monkeypatch):
    nothing = lambda *a, **k: contextlib.nullcontext()  # noqa: E731
    monkeypatch.setattr(torch.cuda, "Stream", _Stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: _Stream())
    monkeypatch.setattr(torch.cuda, "stream", nothing)
    monkeypatch.setattr(torch.cuda, "graph", nothing)
    monkeypatch.setattr(torch.cuda, "CUDAGraph",
                        lambda: types.SimpleNamespace(replay=lambda: None))
    monkeypatch.setattr(nep_ops, "_check_each_call", True)


def test_nep_graph_keeps_its_type_index_and_cached_tensors(fake_cuda):
    seen = []

    class Model:
        q_scaler = torch.ones(3)

        def type_index(self, tm):
            t = torch.zeros(tm.numel(), 2)
            seen.append(weakref.ref(t))
            return t

    w = torch.nn.Parameter(torch.ones(()))
    tr = GraphedNepTrainer(Model(), torch.optim.SGD([w], lr=0.1))

    def loss(batch, tindex):
        ones = splitk._ones_row(12345, torch.device("cpu"), torch.float32)
        img = nep_ops._image_index((2, 3), torch.device("cpu"))
        seen.extend([weakref.ref(ones), weakref.ref(img)])
        return (w * tindex.sum()).sum()

    tr.loss = loss
    batch = {k: torch.zeros(5) for k in GraphedNepTrainer.KEYS}
    batch["num_atom"] = torch.tensor([2, 3])
    tr.step(batch)
    splitk._ones_rows.clear()
    nep_ops._img_cache.clear()
    gc.collect()
    assert len(seen) >= 3 and all(r() is not None for r in seen)


def test_dp_graph_keeps_its_rows_and_workspaces(fake_cuda, monkeypatch):
    monkeypatch.setattr(ops, "_ws_cache", {})
    w = torch.nn.Parameter(torch.ones(()))

    class Trainer:
        _rows = None

        def _loss_and_backward(self, batch, w_f, w_e):
            self._rows = torch.arange(batch["type_map"].numel())
            ops._ws_cache[("cuda:0", SIDE, "dp")] = torch.empty(64)
            w.grad = torch.zeros(())
            return torch.zeros(()), None, None

    t = Trainer()
    tr = GraphedTrainer(t, torch.optim.SGD([w], lr=0.1))

    def batch(n):
        return {**{k: torch.zeros(n) for k in GraphedTrainer.KEYS}, "atom_type": [3]}

    tr.step(batch(4))
    first = [weakref.ref(t._rows), weakref.ref(ops._ws_cache[("cuda:0", SIDE, "dp")])]
    tr.step(batch(6))            # another shape: the trainer's rows and the workspace change
    gc.collect()
    assert all(r() is not None for r in first)
