"""The fused training step groups atoms by the values of the batch's type map: a map refilled in place
(another order of the same elements, other counts) trains like a fresh trainer on that map."""
import numpy as np
import pytest
import torch

from matpl_gb300 import params as P, structures, train
from oracle import neigh

pytestmark = pytest.mark.gpu
DEV = "cuda"


def batches(n=40):
    """Three batches of one shape: types, the types reversed (equal counts), other counts."""
    st = structures.random_packed(n, 0.07, [72, 8], [1 / 3, 2 / 3], seed=3, strain=0.03)
    cfg = P.DPConfig(atom_type=[72, 8], maxNeighborNum=100)
    prm = P.init_params(cfg, 5)
    types = np.random.default_rng(4).permutation(st.types).astype(np.int32)
    other = np.random.default_rng(5).permutation((np.arange(n) < n // 2).astype(np.int32))
    out, stats = [], None
    g = torch.Generator().manual_seed(6)
    E = torch.randn(1, 1, generator=g, dtype=torch.float64)
    F = 0.1 * torch.randn(1, n, 3, generator=g, dtype=torch.float64)
    for t in (types, types[::-1].copy(), other):
        ln, idr = neigh.find_neighbore(t, st.frac, st.lattice, 2, 100, 6.0, [6.0, 6.0])
        stats = stats or P.calc_stat(cfg, ln, idr, t)
        d = lambda a: torch.tensor(a, device=DEV)  # noqa: E731
        out.append({"list_neigh": d(ln), "type_map": d(t), "atom_type": cfg.atom_type, "ImageDR": d(idr),
                    "Etot": E.to(DEV), "Force": F.to(DEV)})
    return lambda: train.DPTrainModel(cfg, prm, *stats, dtype=torch.float64, device=DEV), out


@pytest.mark.parametrize("fit_kernel", [True, False])
def test_refilled_type_map(fit_kernel):
    make, data = batches()
    model = make()
    tr = train.FusedTrainer(model, fit_kernel=fit_kernel)
    held = torch.empty_like(data[0]["type_map"])
    for b in data + data[:1]:
        fresh = make()
        want = train.FusedTrainer(fresh, fit_kernel=fit_kernel).loss_and_backward(b)
        for p in model.parameters():
            p.grad = None
        held.copy_(b["type_map"])
        got = tr.loss_and_backward({**b, "type_map": held})
        assert got == pytest.approx(want, rel=1e-12)
        for k in model.names:
            x, y = model.param(k).grad, fresh.param(k).grad
            assert (x is None) == (y is None), k
            if x is not None:      # the weight gradients are summed by FP64 atomics
                assert float((x - y).abs().max()) <= 1e-10 * max(1e-3, float(y.abs().max())), k


def test_graphed_step_follows_the_type_map():
    """Captured steps on batches of one shape with other orders and counts of the elements: every
    update from the first weights (SGD, rate 1) is minus an eager step's gradient of that batch."""
    make, data = batches()
    model = make()
    tr = train.GraphedTrainer(train.FusedTrainer(model), torch.optim.SGD(model.parameters(), lr=1.0))
    first = {k: model.param(k).detach().clone() for k in model.names}
    for k in (0, 1, 2, 0, 2, 1, 1, 0):
        tr.step(data[k])                       # a capture makes warm-up updates too
        with torch.no_grad():
            for name in model.names:
                model.param(name).copy_(first[name])
        fresh = make()
        want = train.FusedTrainer(fresh).loss_and_backward(data[k])[0]
        assert float(tr.step(data[k])) == pytest.approx(want, rel=1e-12), k
        with torch.no_grad():
            for name in model.names:
                y = fresh.param(name).grad
                y = torch.zeros_like(first[name]) if y is None else y
                x = first[name] - model.param(name)
                assert float((x - y).abs().max()) <= 1e-10 * max(1e-3, float(y.abs().max())), (k, name)
                model.param(name).copy_(first[name])
