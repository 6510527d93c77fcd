"""The dual backward of the force-loss training step, where two warps share 32 slots: one, two and three
elements (a type's slots starting anywhere in the 32), atoms with few, none and more than 32
neighbors, batches that leave warps without an atom.  Parameter gradients of E + F losses against
second-order autograd of the FP64 oracle: FP64 1e-8 and FP32 2e-3 of each array's largest value (of a
thousandth of the largest of all where that is more), the bounds of the training step elsewhere."""
import numpy as np
import pytest
import torch

from matpl_gb300 import params as P, structures, train
from oracle import dp_oracle, neigh

pytestmark = pytest.mark.gpu
DEV = "cuda"


CASES = [([14], 3, 0.0008), ([14], 41, 0.06), ([72, 8], 37, 0.02), ([72, 8], 50, 0.08),
         ([3, 8, 14], 45, 0.06)]
F64, F32 = (torch.float64, 1e-8), (torch.float32, 2e-3)


# three elements' nets in FP64 do not fit in shared memory (refused)
@pytest.mark.parametrize("dtype,tol,elements,n,density",
                         [F64 + c for c in CASES[:4]] + [F32 + c for c in CASES])
def test_parameter_gradients(dtype, tol, elements, n, density):
    nt, m = len(elements), 100
    st = structures.random_packed(n, density, elements, [1.0 / nt] * nt, seed=n, strain=0.02)
    types = np.random.default_rng(n).permutation(st.types).astype(np.int32)
    cfg = P.DPConfig(atom_type=elements, maxNeighborNum=m)
    ln, idr = neigh.find_neighbore(types, st.frac, st.lattice, nt, m, 6.0, [6.0] * nt)
    davg, dstd = P.calc_stat(cfg, ln, idr, types)
    prm = P.init_params(cfg, 5)
    g = torch.Generator().manual_seed(n)
    E_lab = torch.randn(1, generator=g, dtype=torch.float64)
    p = {k: v.clone().requires_grad_() for k, v in prm.items()}
    out = dp_oracle.dp_eval(cfg, p, torch.tensor(davg), torch.tensor(dstd), torch.tensor(ln),
                            torch.tensor(types), torch.tensor(cfg.atom_type), torch.tensor(idr), 0,
                            create_graph=True)
    F_lab = 0.1 * torch.randn(out["Force"].shape, generator=g, dtype=torch.float64)
    mse = torch.nn.functional.mse_loss
    loss = mse(out["Etot"], E_lab.reshape(out["Etot"].shape)) + mse(out["Force"], F_lab)
    names = sorted(p)
    want = dict(zip(names, torch.autograd.grad(loss, [p[k] for k in names], allow_unused=True)))

    model = train.DPTrainModel(cfg, prm, davg, dstd, dtype=dtype, device=DEV)
    batch = {"list_neigh": torch.tensor(ln, device=DEV), "type_map": torch.tensor(types, device=DEV),
             "atom_type": cfg.atom_type, "ImageDR": torch.tensor(idr, device=DEV),
             "Etot": E_lab.reshape(out["Etot"].shape).to(DEV), "Force": F_lab.to(DEV)}
    train.FusedTrainer(model).loss_and_backward(batch)
    ref = {k: torch.zeros_like(prm[k]) if want[k] is None else want[k] for k in names}
    largest = max(float(w.abs().max()) for w in ref.values())
    for k, w in ref.items():
        got = model.param(k).grad
        got = torch.zeros_like(w) if got is None else got.detach().cpu().double()
        assert float((got - w).abs().max()) <= tol * max(float(w.abs().max()), 1e-3 * largest), k
