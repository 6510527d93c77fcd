"""Host threads that run one kernel with different needs of shared memory: neither call may lower the
kernel's limit between the other's request and launch (the descriptor backward of a one-element and an
eight-element model, 23 and 69 KB a block)."""
import threading

import pytest
import torch

from matpl_gb300 import _lib
from matpl_gb300._lib import ptr

pytestmark = pytest.mark.gpu
DEV = "cuda"
N, NN, NMAX, K = 24, 16, 5, 9


def caller(T, calls, failed):
    g = torch.Generator().manual_seed(T)
    nl = torch.randint(0, N, (N, NN), generator=g).to(DEV)
    xyz = torch.randn(N, NN, 3, generator=g)
    d12 = torch.cat([xyz.norm(dim=2, keepdim=True), xyz], 2).float().to(DEV)
    tm = torch.randint(0, T, (N,), generator=g).to(DEV)
    coeff = torch.randn(T, T, NMAX, K, generator=g).to(DEV)
    G = torch.randn(N, 6 * NMAX, generator=g).to(DEV)
    gd, dc = torch.empty_like(d12), torch.empty_like(coeff)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    lib = _lib.load()
    need = lib.matpl_nep_feat_grad_workspace_bytes(_lib.MATPL_F32, 1, N, T, NMAX, K)
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()

    def run():
        for q in range(calls):
            if q % 64 == 0:
                stream.synchronize()
            st = lib.matpl_nep_feat_grad(_lib.MATPL_F32, 1, 1, N, NN, T, NMAX, K, 4, 2, 1, 4.0,
                                         ptr(coeff), ptr(d12), ptr(nl), ptr(tm), ptr(G), 6 * NMAX, 0, 0, 6 * NMAX,
                                         ptr(gd), ptr(dc), ptr(ws), need, ptr(err), stream.cuda_stream)
            if st:
                failed.append(lib.matpl_last_error().decode())
                return
    return run, (stream, dc, gd, err)


def test_threads_share_a_kernel():
    failed = []
    runs = [caller(T, 20000, failed) for T in (1, 8)]
    threads = [threading.Thread(target=r) for r, _ in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    for _, (_, dc, gd, err) in runs:
        assert int(err.item()) == 0 and bool(torch.isfinite(dc).all()) and bool(torch.isfinite(gd).all())
