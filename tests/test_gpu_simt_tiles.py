"""DP evaluation of the plain FP64 / FP32 forms at batch sizes around the lines where the fitting
kernel changes its tile (16, 8, 4 or 1 atoms) and the embedding kernels their block (one or four
warps), with interleaved elements, against the oracle.  FP64: 1e-10 of the largest value (the
form's bar everywhere); FP32: 2e-4 of it."""
import numpy as np
import pytest
import torch

from matpl_gb300 import dp, ops, params as P, structures
from oracle import dp_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


def sizes():
    sms = 152
    return sorted({3, 4 * sms - 1, 4 * sms + 1, 8 * sms + 3, 16 * sms - 1, 16 * sms + 5})


@pytest.mark.parametrize("n", sizes())
def test_plain_forms_match_the_oracle_at_tile_edges(n):
    st = structures.random_packed(n, 0.05, [3, 14], [0.4, 0.6], seed=n)
    types = np.random.default_rng(n).permutation(st.types).astype(np.int32)
    cfg = P.DPConfig(atom_type=[3, 14], maxNeighborNum=60, Rmax=5.0)
    prm = P.init_params(cfg, 5)
    tm = torch.tensor(types, device=DEV)
    ln, idr = ops.find_neighbore(tm, torch.tensor(st.frac, device=DEV),
                                 torch.tensor(st.lattice, device=DEV), 2, 60, 5.0, 5.0)
    davg, dstd = P.calc_stat(cfg, ln.cpu().numpy(), idr.cpu().numpy(), types)
    ref = dp_oracle.dp_eval_chunked(cfg, prm, torch.tensor(davg), torch.tensor(dstd), ln.cpu(),
                                    torch.tensor(types), [3, 14], idr.cpu())
    for prec, tol in (("float64", 1e-10), ("float32", 2e-4)):
        model = dp.DP(cfg, prm, davg, dstd, precision=prec, device=DEV)
        r = model.evaluate(ln, tm, [0, 1], idr.to(model.dtype), 0)
        for key, want in (("Ei_atom", ref["Ei_atom"]), ("Force", ref["Force"])):
            got = r[key].double().cpu()
            assert float((got - want).abs().max()) <= tol * max(1.0, float(want.abs().max())), key
        V = r["Virial"].double().cpu()
        assert float((V - ref["Virial"]).abs().max()) <= tol * max(1.0, float(ref["Virial"].abs().max()))
