"""A type map that is a view (a column of a wider array, an expanded element) is evaluated and trained
like its contiguous copy."""
import pytest
import torch

from matpl_gb300 import dp, ops, params as P, structures, train

pytestmark = pytest.mark.gpu
DEV = "cuda"
N = 60


@pytest.mark.parametrize("expanded", [False, True])
def test_views(expanded):
    els = [29] if expanded else [3, 14]
    nt = len(els)
    st = structures.random_packed(N, 0.05, els, [1 / nt] * nt, seed=1)
    cfg = P.DPConfig(atom_type=els, maxNeighborNum=60, Rmax=5.0)
    tm = torch.tensor(st.types, dtype=torch.int32, device=DEV)
    if expanded:
        view = tm[:1].expand(N)
    else:
        wide = torch.full((N, 3), 1, dtype=torch.int32, device=DEV)
        wide[:, 1] = tm
        view = wide[:, 1]
    ln, idr = ops.find_neighbore(tm, torch.tensor(st.frac, device=DEV), torch.tensor(st.lattice, device=DEV),
                                 nt, 60, 5.0, 5.0)
    davg, dstd = P.calc_stat(cfg, ln.cpu().numpy(), idr.cpu().numpy(), st.types)
    prm = P.init_params(cfg, 5)
    model = dp.DP(cfg, prm, davg, dstd, precision="float64", device=DEV)
    present = list(range(nt))
    assert torch.equal(model.evaluate(ln, view, present, idr)["Ei_atom"], model.evaluate(ln, tm, present, idr)["Ei_atom"])
    assert torch.equal(model(ln, view, els, idr)[1], model(ln, tm, els, idr)[1])
    grads = []
    for m in (tm, view):
        net = train.DPTrainModel(cfg, prm, davg, dstd, dtype=torch.float64, device=DEV)
        batch = {"list_neigh": ln, "type_map": m, "atom_type": els, "ImageDR": idr,
                 "Etot": torch.zeros(1, 1, dtype=torch.float64, device=DEV),
                 "Force": torch.ones(1, N, 3, dtype=torch.float64, device=DEV)}
        train.FusedTrainer(net).loss_and_backward(batch)
        grads.append({k: net.param(k).grad for k in net.names})
    for k, g in grads[0].items():       # weight gradients are summed by FP64 atomics
        assert (grads[1][k] - g).abs().max() <= 1e-10 * max(1e-3, float(g.abs().max())), k
