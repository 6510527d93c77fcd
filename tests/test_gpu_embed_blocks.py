"""The block shape of the plain DP form's embedding kernels below 16 atoms per SM: models of three and four
elements, whose nets every block stages, cost no more per atom than in a larger batch of four-atom
blocks (half as much again allowed), and FP32 agrees with FP64 there (2e-4 of the largest value)."""
import pytest
import torch

from matpl_gb300 import _lib, dp, ops, params as P, structures

pytestmark = pytest.mark.gpu
DEV = "cuda"


def build(elements, n, prec):
    nt = len(elements)
    st = structures.random_packed(n, 0.05, elements, [1.0 / nt] * nt, seed=n)
    cfg = P.DPConfig(atom_type=elements, maxNeighborNum=60, Rmax=6.0)
    tm = torch.tensor(st.types, device=DEV)
    ln, idr = ops.find_neighbore(tm, torch.tensor(st.frac, device=DEV), torch.tensor(st.lattice, device=DEV),
                                 nt, 60, 6.0, 6.0)
    davg, dstd = P.calc_stat(cfg, ln.cpu().numpy(), idr.cpu().numpy(), st.types)
    return lambda p=prec: (lambda m: m.evaluate(ln, tm, list(range(nt)), idr.to(m.dtype), 0))(
        dp.DP(cfg, P.init_params(cfg, 5), davg, dstd, precision=p, device=DEV))


def embed_us(call, reps=5):
    call()
    best = float("inf")
    for _ in range(reps):
        _lib.profile_begin(64)
        call()
        torch.cuda.synchronize()
        t = _lib.profile_collect()
        best = min(best, sum(v[0] for k, v in t.items() if k.startswith("dp_embed")))
    return 1e3 * best


@pytest.mark.parametrize("prec,elements,small", [("float32", [3, 8, 14, 29], 14), ("float32", [3, 8, 14], 14),
                                                 ("float64", [3, 8, 14], 8)])
def test_small_batches_cost_no_more_per_atom(prec, elements, small):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    a, b = (embed_us(build(elements, k * sms, prec)) / (k * sms) for k in (small, 20))
    assert a <= 1.5 * b, (a, b)


@pytest.mark.parametrize("elements", [[3, 8, 14], [3, 8, 14, 29]])
@pytest.mark.parametrize("n", [90, 607, 1300])
def test_fp32_agrees_with_fp64(elements, n):
    run = build(elements, n, "float32")
    got, want = run(), run("float64")
    for k in ("Ei_atom", "Force", "Virial"):
        x, y = got[k].double(), want[k].double()
        assert float((x - y).abs().max()) <= 2e-4 * max(1.0, float(y.abs().max())), k
