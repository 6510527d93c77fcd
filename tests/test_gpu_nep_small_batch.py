"""The fused NEP evaluation of a small batch: every block stages the model's parameters, so blocks with
few atoms must not leave that to few threads (100 atoms take no longer than 1,000, with 30 % allowed),
and its results are those of a batch with all blocks full (FP64, 1e-11 of the largest value)."""
import numpy as np
import pytest
import torch

from matpl_gb300 import _lib, nep as NP, ops, structures

pytestmark = pytest.mark.gpu
DEV = "cuda"


def t(a, dt=torch.float64):
    return torch.tensor(np.ascontiguousarray(a), dtype=dt, device=DEV)


def build(frames, n, prec):
    els = [3, 8, 14, 72]
    cfg = NP.NepConfig(atom_type=els, cutoff=[6.0, 6.0], basis_size=[12, 12], neuron=100)
    one = structures.random_packed(n, 0.06, els, [0.25] * 4, seed=n)
    fr = NP.frames_from_structures([one] * frames, 6.0)
    tm = t(fr.type_map, torch.int64)
    na = t(fr.num_atom.reshape(-1, 1), torch.int64)
    prm = NP.init_params(cfg, 3, energy_shift=-3.0)
    prm["q_scaler"] = torch.full((cfg.feature_nums,), 0.1, dtype=torch.float64)
    a, b, la, lb, ra, rb = ops.calculate_neighbor(na, tm, torch.arange(4, device=DEV), t(fr.box),
                                                  t(fr.box_orig), t(fr.num_cell, torch.int64),
                                                  t(fr.position), 6.0, 6.0, 96, 96, True)
    m = NP.NEP(cfg, prm, prec, device=DEV)
    return lambda: m.evaluate(a, la, ra, b, lb, rb, na, tm)


def eval_us(call, reps=7):
    call()
    best = float("inf")
    for _ in range(reps):
        _lib.profile_begin(64)
        call()
        torch.cuda.synchronize()
        best = min(best, _lib.profile_collect()["nep_eval"][0])
    return 1e3 * best


@pytest.mark.parametrize("prec", ["float32", "float64"])
def test_small_batch_takes_no_longer(prec):
    small, large = eval_us(build(1, 100, prec)), eval_us(build(10, 100, prec))
    assert small <= 1.3 * large, (small, large)


def test_small_batch_equals_large():
    one, many = build(1, 100, "float64")(), build(20, 100, "float64")()
    for k in ("Ei", "Force"):
        x, y = one[k], many[k].reshape(20, *one[k].shape)
        assert float((y - x).abs().max()) <= 1e-11 * max(1.0, float(x.abs().max())), k
