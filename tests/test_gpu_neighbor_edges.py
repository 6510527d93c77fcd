"""Neighbor search and skin filter at the edges of their index paths: slot counts that leave the
per-warp scratch rows unaligned without padding, image walks whose radices differ per direction
(and atom counts below and above a warp), and unwrapped positions several cells away (images
outside the filter's table).  Lists bit-exact against the oracle; forces to 1e-10 of the largest
(FP64, the same pairs)."""
import numpy as np
import pytest
import torch

from matpl_gb300 import md, params as P, structures
from tests.test_gpu_md import _setup
from tests.test_gpu_neighbor import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntypes,m", [(1, 75), (1, 101), (3, 37), (5, 33)])
def test_odd_slot_counts(ntypes, m):
    rng = np.random.default_rng(ntypes)
    st = structures.random_packed(700, 0.03, list(range(1, ntypes + 1)), [1 / ntypes] * ntypes, seed=m)
    types = rng.permutation(st.types).astype(np.int32)
    assert_same(structures.Structure(st.lattice, st.frac, types, st.elements), ntypes, m)


@pytest.mark.parametrize("edges", [(4.0, 7.0, 30.0), (30.0, 4.0, 7.0), (11.9, 11.9, 11.9), (5.0, 26.0, 5.0),
                                   (2.5, 2.5, 90.0)])
@pytest.mark.parametrize("shear", [0.0, 0.4])
def test_image_walk_radices(edges, shear):
    n = max(1, int(round(0.02 * np.prod(edges))))
    rng = np.random.default_rng(n)
    lat = np.diag(edges)
    lat[1] += shear * lat[0]
    types = (np.arange(n) % 2).astype(np.int32)
    st = structures.Structure(lat, rng.random((n, 3)), types, [3, 14])
    assert_same(st, 2, 200)


def test_filter_images_outside_the_table():
    cfg, prm, davg, dstd, reps = _setup()
    a = md.ReplicaMD(cfg, prm, davg, dstd, reps, [63.546], precision="float64")
    b = md.ReplicaMD(cfg, prm, davg, dstd, reps, [63.546], precision="float64")
    g = torch.Generator().manual_seed(3)
    n = torch.randint(-5, 6, (a.natoms_total, 3), generator=g).double().to(b.x.device)
    b.x += torch.einsum("na,nac->nc", n, b.lat[b.atom_rep.long()])
    for sim in (a, b):
        sim.gate.fill_(1)
        sim._forces()
        sim.check_errors()
    assert torch.equal(a.nn, b.nn)
    assert float((a.out["Force"] - b.out["Force"]).abs().max()) <= \
        1e-10 * float(a.out["Force"].abs().max())
