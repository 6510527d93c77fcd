"""The element-grouped atom energies of DP.forward follow the values of the type map wherever its
address and version do not tell that they changed: an inference tensor refilled in place, a
write through ``.data``, the replay of a captured call, another stream."""
import pytest
import torch

from matpl_gb300 import dp, ops, params as P, structures

pytestmark = pytest.mark.gpu
DEV = "cuda"
N = 40


def setup():
    st = structures.random_packed(N, 0.05, [3, 14], [0.5, 0.5], seed=1)
    cfg = P.DPConfig(atom_type=[3, 14], maxNeighborNum=60, Rmax=5.0)
    lat, frac = torch.tensor(st.lattice, device=DEV), torch.tensor(st.frac, device=DEV)
    maps = [torch.randint(0, 2, (N,), generator=torch.Generator().manual_seed(s)) for s in range(2)]
    maps.append(maps[0].flip(0))                               # the counts of the first
    lists = [ops.find_neighbore(m.to(DEV, torch.int32), frac, lat, 2, 60, 5.0, 5.0) for m in maps]
    davg, dstd = P.calc_stat(cfg, lists[0][0].cpu().numpy(), lists[0][1].cpu().numpy(), maps[0].numpy())
    model = dp.DP(cfg, P.init_params(cfg, 5), davg, dstd, precision="float64", device=DEV, check_errors=False)

    def want(k):
        Ei = model.evaluate(lists[k][0], maps[k].to(DEV, torch.int32), [0, 1], lists[k][1])["Ei_atom"]
        return Ei[:, torch.cat([torch.nonzero(maps[k] == t).flatten() for t in (0, 1)]).to(DEV)]
    return model, maps, lists, [want(k) for k in range(3)]


@pytest.mark.parametrize("how", ["inference", "data", "stream"])
def test_refilled_map(how):
    model, maps, lists, want = setup()
    with torch.inference_mode(how == "inference"):
        held = torch.empty(N, dtype=torch.int32, device=DEV)
        for k in (0, 1, 2, 0):
            (held.data if how == "data" else held).copy_(maps[k])
            s = torch.cuda.Stream() if how == "stream" else torch.cuda.current_stream()
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                got = model(lists[k][0], held, [3, 14], lists[k][1])[1]
            torch.cuda.current_stream().wait_stream(s)
            assert torch.equal(got, want[k]), (how, k)
            torch.cuda.synchronize()
    # an entry made under inference mode serves a call outside
    assert torch.equal(model(lists[0][0], maps[0].to(DEV, torch.int32), [3, 14], lists[0][1])[1], want[0])


def test_captured_call_reads_the_map():
    model, maps, lists, want = setup()
    held = maps[0].to(DEV, torch.int32)
    ln, idr = lists[0][0].clone(), lists[0][1].clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        model(ln, held, [3, 14], idr)
    torch.cuda.current_stream().wait_stream(side)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        got = model(ln, held, [3, 14], idr)[1]
    for k in (0, 2, 0):                                        # maps of the same element counts
        held.copy_(maps[k])
        ln.copy_(lists[k][0])
        idr.copy_(lists[k][1])
        model(lists[1][0], maps[1].to(DEV, torch.int32), [3, 14], lists[1][1])    # another map in between
        g.replay()
        assert torch.equal(got, want[k]), k
