"""The element-grouped atom energies of DP.forward belong to the type map of the call: another map of
the same length, a map changed in place, and maps of other dtypes and on the host."""
import pytest
import torch

from matpl_gb300 import dp, ops, params as P, structures

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("where,dtype", [(DEV, torch.int32), (DEV, torch.int64), ("cpu", torch.int32)])
def test_order_follows_the_map(where, dtype):
    st = structures.random_packed(40, 0.05, [3, 14], [0.5, 0.5], seed=1)
    cfg = P.DPConfig(atom_type=[3, 14], maxNeighborNum=60, Rmax=5.0)
    prm = P.init_params(cfg, 5)
    lat, frac = torch.tensor(st.lattice, device=DEV), torch.tensor(st.frac, device=DEV)
    model = None
    for seed in range(4):
        tm = torch.randint(0, 2, (40,), generator=torch.Generator().manual_seed(seed))
        ln, idr = ops.find_neighbore(tm.to(DEV, torch.int32), frac, lat, 2, 60, 5.0, 5.0)
        if model is None:
            davg, dstd = P.calc_stat(cfg, ln.cpu().numpy(), idr.cpu().numpy(), tm.numpy())
            model = dp.DP(cfg, prm, davg, dstd, precision="float64", device=DEV)
            held = torch.empty(40, dtype=dtype, device=where)
        Ei = model.evaluate(ln, tm.to(DEV, torch.int32), [0, 1], idr)["Ei_atom"].cpu()
        want = Ei[:, torch.cat([torch.nonzero(tm == t).flatten() for t in (0, 1)])]
        fresh = model(ln, tm.to(where, dtype), [3, 14], idr)[1].cpu()        # a freed map's address
        held.copy_(tm)
        kept = model(ln, held, [3, 14], idr)[1].cpu()                        # changed in place
        assert torch.equal(fresh, want) and torch.equal(kept, want)
