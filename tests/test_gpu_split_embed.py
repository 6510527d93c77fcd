"""Small FP64 batches of the plain DP form, where four warps share an atom: fewer and more occupied runs
of 32 slots than warps, atoms without neighbors, elements absent from the model, and nets that
stay in global memory (four elements), against the oracle to 1e-10 of the largest value (the form's
bar everywhere)."""
import numpy as np
import pytest
import torch

from matpl_gb300 import dp, ops, params as P, structures
from oracle import dp_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("elements,n,density,m", [([29], 5, 0.001, 40), ([29], 450, 0.06, 200),
                                                  ([3, 14], 64, 0.06, 60), ([3, 8, 14, 29], 90, 0.08, 50),
                                                  ([3, 8, 14, 29], 700, 0.05, 33)])
def test_atoms_shared_by_warps(elements, n, density, m):
    nt = len(elements)
    st = structures.random_packed(n, density, elements, [1.0 / nt] * nt, seed=n)
    types = np.random.default_rng(n).permutation(st.types).astype(np.int32)
    cfg = P.DPConfig(atom_type=elements, maxNeighborNum=m, Rmax=5.0 if nt > 1 else 8.5)
    prm = P.init_params(cfg, 5)
    tm = torch.tensor(types, device=DEV)
    ln, idr = ops.find_neighbore(tm, torch.tensor(st.frac, device=DEV),
                                 torch.tensor(st.lattice, device=DEV), nt, m, cfg.Rmax, cfg.Rmax)
    davg, dstd = P.calc_stat(cfg, ln.cpu().numpy(), idr.cpu().numpy(), types)
    for present in ({tuple(elements), tuple(elements[:max(1, nt - 1)])}):
        ref = dp_oracle.dp_eval_chunked(cfg, prm, torch.tensor(davg), torch.tensor(dstd), ln.cpu(),
                                        torch.tensor(types), list(present), idr.cpu())
        model = dp.DP(cfg, prm, davg, dstd, precision="float64", device=DEV)
        r = model.evaluate(ln, tm, model.present_types(list(present)), idr, 0)
        for key in ("Ei_atom", "Force", "Virial"):
            got, want = r[key].cpu(), ref[key]
            assert float((got - want).abs().max()) <= 1e-10 * max(1.0, float(want.abs().max())), key
