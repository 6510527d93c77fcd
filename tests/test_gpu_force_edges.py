"""calculateForce / calculateVirial and their backward where a warp stages 32 slots: widths around it,
empty lists and atoms, holes, ghosts, several configurations, against sums by index in FP64.
FP64: 1e-12 of the largest value; FP32: 60 terms of 4 products, each rounded to 6e-8: 2e-5 of it."""
import pytest
import torch

from matpl_gb300 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dt,tol", [(torch.float64, 1e-12), (torch.float32, 2e-5)])
@pytest.mark.parametrize("B,N,S,nghost,fill", [(1, 1, 1, 0, 1.0), (1, 7, 31, 0, 0.5), (2, 33, 32, 5, 0.9),
                                               (3, 20, 33, 0, 0.0), (2, 301, 64, 17, 0.7),
                                               (1, 1000, 150, 0, 0.4)])
def test_force_and_virial(dt, tol, B, N, S, nghost, fill):
    g = torch.Generator().manual_seed(B * N + S)
    nall = N + nghost
    nl = torch.randint(0, nall, (B, N, S), generator=g)
    nl[torch.rand(B, N, S, generator=g) >= fill] = -1
    if N > 2:
        nl[:, 1] = -1
    rn = lambda *s: torch.randn(*s, generator=g, dtype=dt)  # noqa: E731
    dE, rij, rid, Fc = rn(B, N, 1, 4 * S), rn(B, N, S, 3), rn(B, N, 4 * S, 3), rn(B, N, 3)
    gF, gV = rn(B, nall, 3), rn(B, 9)
    d = lambda t: t.to(DEV)  # noqa: E731
    dEg = d(dE).requires_grad_()
    li = d(nl.to(torch.int32)).unsqueeze(2)
    F = ops.calculateForce(li, dEg, d(rid), d(Fc), nghost)[0]
    V, av = ops.calculateVirial(li, dEg, d(rij), d(rid), nghost)
    got = torch.autograd.grad([F, V], [dEg], [d(gF), d(gV)])[0]

    has = (nl >= 0).unsqueeze(-1)
    f = (dE.double().reshape(B, N, S, 4, 1) * rid.double().reshape(B, N, S, 4, 3)).sum(3) * has
    vv = (f.unsqueeze(-1) * rij.double().unsqueeze(-2)).reshape(B, N * S, 9)
    j = nl.clamp(min=0).reshape(B, N * S)
    base = torch.cat([Fc.double(), torch.zeros(B, nghost, 3, dtype=torch.float64)], 1)
    Fw = base.scatter_add(1, j.unsqueeze(-1).expand(-1, -1, 3), f.reshape(B, N * S, 3))
    avw = torch.zeros(B, nall, 9, dtype=torch.float64).scatter_add(1, j.unsqueeze(-1).expand(-1, -1, 9), vv)
    Vw = vv.sum(1)
    # the operators' backward (calculateForceGrad.cu:10-60, calculateVirialGrad.cu:16-66): the centre's
    # gradient reaches every slot, a neighbor's is that of atom j % N
    gj = torch.gather(gF.double(), 1, (j % N).unsqueeze(-1).expand(-1, -1, 3)).reshape(B, N, S, 3) * has
    u = gj - gF.double()[:, :N].unsqueeze(2) + \
        (torch.einsum("bac,bnsc->bnsa", gV.double().reshape(B, 3, 3), rij.double()) * has)
    gw = torch.einsum("bnswa,bnsa->bnsw", rid.double().reshape(B, N, S, 4, 3), u).reshape(dE.shape)
    for x, y in ((F, Fw), (V, Vw), (av, avw), (got, gw)):
        x, y = x.detach().cpu().double(), y.detach()
        assert x.shape == y.shape
        assert float((x - y).abs().max()) <= tol * max(1.0, float(y.abs().max())) * (1 + fill * S) ** 0.5
