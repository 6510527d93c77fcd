"""The captured NEP training step reads the type map of each batch: batches of one shape with the elements
in other orders and counts, each update from the first weights (SGD, rate 1) against minus the
gradient of an eager step (FP64, 1e-10 of each array's largest value or of 1)."""
import numpy as np
import torch
import pytest

from tests.test_gpu_nep_train import close, dev, nep_train_model

pytestmark = pytest.mark.gpu


def test_graphed_step_follows_the_type_map(nep_case):
    from matpl_gb300 import nep_ops
    from matpl_gb300.nep_train import GraphedNepTrainer
    c = nep_case("nep_q4_tri2")
    N, B = c.NL_r.shape[0], len(c.g["num_atom"])
    rng = np.random.default_rng(3)
    b = {"NN_r": dev(c.NN_r), "NL_r": dev(c.NL_r), "Ri_r": dev(c.Ri_r), "NN_a": dev(c.NN_a),
         "NL_a": dev(c.NL_a), "Ri_a": dev(c.Ri_a), "num_atom": torch.tensor(c.g["num_atom"]),
         "per_atom": dev(np.asarray(c.g["num_atom"], dtype=np.float64)),
         "Etot": dev(rng.standard_normal(B)), "Force": dev(rng.standard_normal((N, 3))),
         "Virial": dev(rng.standard_normal((B, 9)))}
    types = np.asarray(c.g["type_map"])
    data = [{**b, "type_map": dev(t)} for t in
            (types, types[::-1].copy(), rng.integers(0, c.cfg.ntypes, N).astype(types.dtype))]
    m1, m2 = nep_train_model(c), nep_train_model(c)
    first = {k: p.detach().clone() for k, p in m1.named_parameters()}
    t1 = GraphedNepTrainer(m1, torch.optim.SGD(m1.parameters(), lr=1.0), w_v=0.1, warmup=1)
    t2 = GraphedNepTrainer(m2, torch.optim.SGD(m2.parameters(), lr=0.0), w_v=0.1)
    try:
        t1.step(data[0])
        for k in (0, 1, 2, 0):
            with torch.no_grad():
                for name, p in m1.named_parameters():
                    p.copy_(first[name])
            loss = float(t1.step(data[k]).detach())
            m2.zero_grad(set_to_none=True)
            want = t2.loss(data[k])
            want.backward()
            close(torch.tensor([loss], dtype=torch.float64), np.array([float(want.detach())]), 1e-10)
            for name, p in m2.named_parameters():
                g = torch.zeros_like(p) if p.grad is None else p.grad
                close(first[name] - dict(m1.named_parameters())[name].detach(), g.cpu().numpy(), 1e-10)
        t1.check_errors()
    finally:
        nep_ops.set_check_errors(True)
