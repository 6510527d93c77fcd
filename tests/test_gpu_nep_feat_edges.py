"""The NEP descriptor operators with first and second backward at the edges of their forms: list
widths around a warp's 32 slots, empty lists and atoms, one type and many (c-gradient tables in shared
memory and by workspace), both compiled sizes and odd ones inside them, G as a slice of a wider
array.  Against the oracle's features under autograd in FP64."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from matpl_gb300 import nep_ops, ops
from oracle import nep_oracle as NO

pytestmark = pytest.mark.gpu
DEV = "cuda"
RC = 4.5
# FP64: as the fixtures' tests.  FP32: about 100 roundings of 6e-8 (64 pairs, Chebyshev recursion, up to
# the fourth power of their sums) with a threefold cancellation, of the largest value
TOL = {torch.float64: 1e-11, torch.float32: 2e-5}


def inputs(N, W, T, n, K, seed):
    g = np.random.default_rng(seed)
    count = g.integers(0, W + 1, N)
    count[:2] = (W, 0)
    slot = np.arange(W)[None] < count[:, None]
    nl = np.where(slot, g.integers(0, N, (N, W)), -1)
    xyz = g.normal(size=(N, W, 3))
    r = g.uniform(0.8, 1.05 * RC, (N, W, 1))
    xyz *= r / np.linalg.norm(xyz, axis=2, keepdims=True)
    d = np.where(slot[..., None], np.concatenate([r, xyz], 2), 0.0)
    H = g.normal(size=(N, W, 4)) * slot[..., None]
    return (torch.tensor(nl), torch.tensor(d), torch.tensor(g.integers(0, T, N)),
            torch.tensor(0.3 * g.normal(size=(T, T, n, K))), torch.tensor(H), g)


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("angular", [False, True])
@pytest.mark.parametrize("N,W,T,n,K,l", [(37, 1, 1, 1, 1, (1, 0, 0)), (131, 31, 3, 5, 9, (4, 2, 1)),
                                         (64, 33, 4, 5, 9, (4, 2, 0)), (66, 64, 9, 5, 9, (4, 2, 1)),
                                         (50, 40, 3, 8, 16, (3, 0, 1)), (45, 32, 6, 6, 12, (4, 2, 1)),
                                         (7000, 5, 2, 2, 3, (2, 2, 0))])
def test_first_and_second_backward(dt, angular, N, W, T, n, K, l):
    nl, d, tm, c, H, g = inputs(N, W, T, n, K, 100 * N + W)
    cfg = SimpleNamespace(kr=K, ka=K, cutoff=[RC, RC], l_max=list(l))
    feat = NO.features_mb if angular else NO.features_2b
    cast = lambda t: t.to(dt).double()  # noqa: E731   (the oracle takes the rounded inputs)
    F = n * (l[0] + (l[1] > 0) + (l[2] > 0)) if angular else n
    wide = torch.tensor(g.normal(size=(N, F + 3)))
    G, U = wide[:, 2:2 + F], torch.tensor(g.normal(size=(N, F)))

    def grads(q, c_, d_, G_, H_, U_):
        gc, gd = torch.autograd.grad(q, [c_, d_], G_, create_graph=True)
        return [q, gc, gd] + list(torch.autograd.grad([q, gd], [c_, G_], [U_, H_]))
    oc, od, oG = cast(c).requires_grad_(), cast(d).requires_grad_(), cast(G).requires_grad_()
    want = grads(feat(cfg, oc, tm, nl, od), oc, od, oG, cast(H), cast(U))
    dev = lambda t, k=dt: t.to(DEV, k)  # noqa: E731
    gc_, gd_ = dev(c).requires_grad_(), dev(d).requires_grad_()
    gG = dev(wide)[:, 2:2 + F].requires_grad_()
    a = (dev(nl, torch.int64), dev(tm, torch.int64), torch.empty(0, dtype=dt, device=DEV), RC)
    if angular:
        q = ops.calculateNepMbFeat(gc_, gd_, a[0], a[1], a[2], 0, *l, RC)[0]
    else:
        q = ops.calculateNepFeat(gc_, gd_, a[0], a[1], a[2], RC, 0)[0]
    got = grads(q, gc_, gd_, gG, dev(H), dev(U))
    for name, x, y in zip(("q", "dc", "dd12", "second dc", "second dG"), got, want):
        y = y.detach()
        occ = slice(None)
        if name == "dd12":
            occ = nl >= 0
            assert bool((x.detach().cpu()[~occ] == 0).all()), "empty slots"
        err = (x.detach().cpu().double() - y)[occ].abs().max().item() if y[occ].numel() else 0.0
        assert err <= TOL[dt] * max(1.0, y[occ].abs().max().item() if y[occ].numel() else 0.0), (name, err)
    only, = torch.autograd.grad(nep_ops.nep_feat_d12(gc_, gG, gd_, a[0], a[1], angular, RC, *l), [gG],
                                dev(H))
    assert (only - got[4]).abs().max().item() <= TOL[dt] * max(1.0, got[4].abs().max().item())
